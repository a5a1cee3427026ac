// sbe_f64.cuh -- what the FP64 step's entry points (sbe_f64.cu) and its
// fast-convolution kernel (sbe_conv.cu) share.
#pragma once

#include "psb_common.cuh"

namespace psb {

enum Mode { kRhs = 0, kRk4 = 1, kLeapfrog = 2, kCalcH = 3 };

// Largest grid whose single right-hand side the direct kernel takes (one point
// of k per thread).  Measured on B200, one call of WireBatch.rhs, direct / by
// transforms (us): Nk 256, 16 wires 15 / 18, 2048 wires 69 / 40; Nk 512, 16
// wires 21 / 18, 2048 wires 215 / 72.  The line lies where few wires, whose
// call is launches and latency, break even.
constexpr int kDirectNk = 256;

struct Batch {
  const PsbTable* tables;
  int ntab;
  const double* tabdata;
  int64_t n_tabdata;
  PsbWire* wires;
  int nw;
  const int32_t* order;
  double* y;   // RK4 state, leapfrog X2, RHS input
  double* y1;  // leapfrog X1
  double* dy;  // RHS output
  int64_t n_state;
  const double* field;
  int64_t field_stride;
  int64_t n_field;
  int nsteps;
  double dt;
  double* P;
  int64_t n_P;
  int p_stride;
  int p_cap;
  double hbar;
  int nk_limit;  // largest nk the launch's shared memory was sized for
};

// `mode` over grid wires (bt.order, or wires 0 .. grid - 1): those of more
// than nkmin points; one_class: every wire is of nkmax's size class.
int launch_sbe_conv(const Batch& bt, int mode, int grid, int nkmax, int nkmin, bool screened,
                    bool shared, bool one_class, cudaStream_t st);
// Dynamic shared memory of that launch for one wire of nk points.
size_t conv_smem_bytes(int nk, bool shared);

}  // namespace psb
