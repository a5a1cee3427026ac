"""The kernels' shared-memory limits, on the CPU with a recording stand-in for
the CUDA runtime's calls.  A limit belongs to a kernel on one device and is
shared by all host threads, so a launch must find it high enough whatever other
launches were made before it: on every device, and with one value per kernel
(a second thread that set a lower one between a call's own and its launch would
make that launch fail)."""

import json
import os
import subprocess
import sys

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

STAND_IN = r"""
#include <cuda_runtime_api.h>
#include <string.h>
static struct { int dev; const void* f; int limit; } known[4096];
static int nknown, device, changed, refused, launches;
static cudaError_t last = cudaSuccess;
static int* limit_of(const void* f) {
  for (int i = 0; i < nknown; ++i)
    if (known[i].dev == device && known[i].f == f) return &known[i].limit;
  known[nknown].dev = device;
  known[nknown].f = f;
  return &known[nknown++].limit;
}
void stand_in_device(int d) { device = d; }
void stand_in_counts(int* out) { out[0] = launches; out[1] = refused; out[2] = changed; }
cudaError_t cudaFuncSetAttribute(const void* f, enum cudaFuncAttribute a, int value) {
  if (a != cudaFuncAttributeMaxDynamicSharedMemorySize) return cudaSuccess;
  if (value > 227 * 1024) return last = cudaErrorInvalidValue;
  int* l = limit_of(f);
  if (*l && *l != value) ++changed;
  *l = value;
  return cudaSuccess;
}
cudaError_t cudaFuncGetAttributes(struct cudaFuncAttributes* a, const void* f) {
  memset(a, 0, sizeof(*a));
  a->numRegs = 80;
  a->maxThreadsPerBlock = 1024;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3 g, dim3 b, void** args, size_t smem,
                             cudaStream_t s) {
  ++launches;
  if (smem > 48 * 1024 && smem > (size_t)*limit_of(f)) {
    ++refused;
    return last = cudaErrorInvalidValue;
  }
  return cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void** args) {
  return cudaLaunchKernel(f, c->gridDim, c->blockDim, args, c->dynamicSmemBytes, c->stream);
}
cudaError_t cudaGetLastError(void) {
  const cudaError_t e = last;
  last = cudaSuccess;
  return e;
}
"""

CALLS = r"""
import ctypes, json, sys
import numpy as np
from pulsesuite_b200 import _lib, abi

lib = _lib.load()
me = ctypes.CDLL(sys.argv[1])
any_ptr = ctypes.c_void_p(1 << 20)   # never read by the host
model, prm = abi.model_array(1.0), np.zeros(1, dtype=abi.FULL_PARAMS_DTYPE)
prm["hbar"], prm["lf"] = 1.0, 1
mb = np.zeros(1, dtype=abi.FULL_MB_DTYPE)
for f in abi.FULL_MB_DTYPE.names:
    mb[f] = 1 << 20 if abi.FULL_MB_DTYPE[f] == np.uint64 else 1
mb["n_hw"] = 8
m, p, q = abi.as_ptr(model), any_ptr, None
tail = (4, 1e-15, p, 1 << 40, 1, 4, m, q)
errors = []

def call(name, *a):
    try:
        _lib.call(name, *a)
    except _lib.PsbError as e:
        errors.append(str(e))

for device in (0, 1, 0):
    me.stand_in_device(device)
    for nk in (1024, 600, 512, 300, 256, 200, 128, 64, 20):
        for flags in (0, 4, 8, 12, 2, 6, 10, 14):
            common = (p, 1, p, 1 << 40, p, 7)
            call("psb_rhs_f64", *common, p, p, 1 << 30, nk, flags, m, q)
            call("psb_calch_f64", *common, p, p, 1 << 30, nk, flags, m, q)
            call("psb_rk4_f64", *common, q, 0, p, 1 << 30, nk, flags, *tail)
            call("psb_leapfrog_f64", *common, q, 0, p, p, 1 << 30, nk, flags, p, 8, 1 << 40, *tail)
            if not flags & 8:
                for w in range(1, lib.psb_split_wire_max_group(nk, flags) + 1, 5):
                    call("psb_rk4_split_wire", *common, p, 3, w, nk, flags | 1, p, 1000, p,
                         1 << 40, *tail)
        for w in (4, 8, 16):
            if nk <= lib.psb_split_max_nk(w):
                call("psb_rk4_split", *common, p, 3, w, nk, p, 1000, p, 1 << 40, *tail)
        nr = 2 * (nk + 1)
        for nw in (64, 9, 1):
            call("psb_full_step_batch_f64", nw, nk, nr, nr // 2, p, 1.0, 1.0, 1, p,
                 abi.as_ptr(prm), p, abi.as_ptr(mb), p, p, p, p, 1 << 60, q)
            call("psb_full_sources_batch_f64", nw, nk, nr, p, p, p, 1.0, 1.0, p, p, p, q)
c = (ctypes.c_int * 3)()
me.stand_in_counts(c)
print(json.dumps({"launches": c[0], "refused": c[1], "changed": c[2], "errors": errors[:5]}))
"""


def test_limits_of_every_launch(tmp_path):
    inc = "/usr/local/cuda/include"
    if not os.path.exists(os.path.join(inc, "cuda_runtime_api.h")):
        pytest.skip("no CUDA headers")
    src, lib = tmp_path / "stand_in.c", str(tmp_path / "stand_in.so")
    src.write_text(STAND_IN)
    r = subprocess.run(["gcc", "-shared", "-fPIC", "-w", "-I", inc, "-o", lib, str(src)],
                       capture_output=True, text=True)
    if r.returncode:
        pytest.skip("no host C compiler: " + r.stderr)
    r = subprocess.run([sys.executable, "-c", CALLS, lib], capture_output=True, text=True,
                       cwd=REPO, env={**os.environ, "LD_PRELOAD": lib, "PYTHONPATH": REPO})
    assert r.returncode == 0, r.stderr
    got = json.loads(r.stdout)
    assert got["launches"] > 500 and got["errors"] == [], got
    assert got["refused"] == 0 and got["changed"] == 0, got
