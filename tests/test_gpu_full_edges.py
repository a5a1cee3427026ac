"""The full-matrix step and its sources where their kernels change: k grids
that fill no tile (34 .. 148 points), few and many wires (16- and 32-blocks of
the right-hand side, 4 and 8 positions a CTA in the density sums), and wire
grids whose k points are not equidistant; with the many-body terms, batches on
both sides of every grouping of wires.

Against 64-bit torch the bound is 1e-12 of each output's largest value: sums
of at most 150 products of values of one scale, 150 x 1.1e-16 x a factor of
ten for the terms that cancel, with a margin of five.
"""

import numpy as np
import pytest
import torch
from helpers import relerr
from test_gpu_manybody import MB
from test_gpu_pstd_batch import LEVELS, make_solver

from perf import cases
from pulsesuite_b200 import _lib, device

pytestmark = pytest.mark.gpu

TOL = 1e-12


@pytest.mark.parametrize("L,nw", [(30e-9, 1), (30e-9, 33), (47e-9, 3), (62e-9, 9), (100e-9, 1),
                                  (110e-9, 40), (130e-9, 5)])
@pytest.mark.parametrize("screened", [False, True])
def test_full_step_edges(cuda, L, nw, screened):
    case = {"kind": "full", "nw": nw, "L": L, "screened": screened}
    got = cases.run(cases.prepare(case, 3))
    want = cases.exact(case, 3)
    for key in ("L1", "L2", "L3", "out"):
        parts = 5 if key == "out" else 3
        for j in range(parts):
            g, w = got[key][:, j].cpu().numpy(), want[key][:, j].cpu().numpy()
            assert relerr(g, w) < TOL, (key, j)


@pytest.mark.parametrize("uneven", [0.0, 1e-3, 0.3])
def test_sources_of_any_k_grid(cuda, uneven):
    """Equidistant k points take the diagonal sums, all others the double
    sums; a spacing off by a part in a thousand already does."""
    case = {"kind": "full", "nw": 3, "L": 62e-9, "screened": False}
    s = cases.prepare(case, 4)
    n, nk, nr = 3, s["nk"], s["nr"]
    kr = s["kr"].clone()
    kr += uneven * (kr[1] - kr[0]) * torch.sin(torch.arange(nk, device="cuda") * 1.7)
    _lib.call("psb_full_sources_batch_f64", n, nk, nr, device.ptr(kr), device.ptr(s["r"]),
              device.ptr(s["window"]), s["grid"].L, s["grid"].dcv, device.ptr(s["wpar"]),
              device.ptr(s["L3"]), device.ptr(s["out"]), device.stream_ptr())
    g, W, x3 = s["grid"], s["window"], s["L3"]
    yw, sg = s["wpar"][:, 0, None], s["wpar"][:, 1, None]
    i = torch.arange(nk, device="cuda")
    xs = (1.0 - 2.0 * ((i + 1) % 2).double()).to(torch.complex128)
    E = torch.exp(1j * kr[None, :] * s["r"][:, None])

    def src(A, left):
        return torch.einsum("ra,wab,rb->wr", E.conj() * left, A, E)

    one = torch.ones_like(xs)
    px, py = src(x3[:, 0], xs).real, src(x3[:, 0], one).real
    want = [W * g.dcv * px, W * yw * g.dcv * py, -W * sg * g.dcv * py,
            W / (2 * g.L) * src(x3[:, 1], one), W / (2 * g.L) * src(x3[:, 2].conj(), one)]
    for j, w in enumerate(want):
        assert relerr(s["out"][:, j].cpu().numpy(), w.cpu().numpy()) < TOL, j


@pytest.mark.parametrize("L,nw", [(2.4e-8, 3), (3.1e-8, 4), (3.1e-8, 9), (2.85e-8, 17),
                                  (2.4e-8, 33)])
def test_many_body_batches_bitwise(cuda, tmp_path, L, nw):
    """Every wire of a batch has the bits of its own call, whatever the
    wires that share a CTA with it."""
    nrr, dt = 48, 1e-17
    text = MB.format(scr=1, lor=0, rc=1, dc=1, lf=1)
    a = make_solver(tmp_path / "a", L, 5e12, nw, text, edc=2e6, nrr=nrr)
    b = make_solver(tmp_path / "b", L, 5e12, nw, text, edc=2e6, nrr=nrr)
    rr = np.linspace(-5e-8, 5e-8, nrr)
    scale, shift = np.linspace(0.4, 1.3, nw), np.linspace(-1.5e-8, 1.5e-8, nw)
    for i in range(3):
        pr = 2e8 * np.exp(-(((rr[:, None] - shift) / 3e-8) ** 2)) * scale * np.cos(0.3 * i)
        F = [(0.3 * pr * rr[:, None] / 3e-8).astype(complex), pr.astype(complex),
             (0.2 * pr).astype(complex), np.zeros((nrr, nw), complex)]
        oa = [np.zeros((nrr, nw), complex) for _ in range(4)]
        ob = [np.zeros((nrr, nw), complex) for _ in range(4)]
        a.QWCalculatorAll(*F, rr, None, dt, *oa, [False], [False])
        for w in range(nw):
            o = [np.zeros(nrr, complex) for _ in range(4)]
            b.QWCalculator(*(f[:, w] for f in F), rr, None, dt, w + 1, *o, [False], [False])
            for x, y in zip(ob, o):
                x[:, w] = y
        for x, y in zip(oa, ob):
            assert np.array_equal(x, y), i
    la, lb = a._level_arrays(), b._level_arrays()
    for key in LEVELS:
        assert np.array_equal(la[key], lb[key]), key
