"""The screening logarithm of the FP64 step (log_ratio, sbe_conv.cu) where its
short form does not hold: momentum transfers near the ends of the range of
doubles, against the CPU oracle (tolerance of test_gpu_conv).  Wires without
carriers for one right-hand side only: a step gives them a density of rounding
errors, zero or not, and log |(q - pi n) / (q + n)| of a transfer below that
jumps between 0 and log pi."""

import numpy as np
import pytest
from helpers import HBAR
from test_gpu_conv import batch, case, compare, oracle_wires

from oracle import oracle as orc

pytestmark = pytest.mark.gpu

NKS = [30, 64, 128, 200, 256, 300, 512, 1024]


def far_case(q, which):
    grids, tables, tabdata, w, y0 = case(NKS, "distinct", True, seed=9)
    tabdata = np.array(tabdata)
    for t in tables:
        nk, off = int(t["nk"]), int(t["off"])
        d = np.array([1, nk // 3, nk - 1])  # transfers 1, some, the largest
        for blk in {"electrons": (7,), "holes": (8,), "both": (7, 8)}[which]:
            tabdata[off + blk * nk + d] = q
    return grids, tables, tabdata, w, y0


@pytest.mark.parametrize("q", [1e300, 1e-300, 5e-324])
@pytest.mark.parametrize("which", ["electrons", "holes", "both"])
def test_far_momenta_step(cuda, q, which):
    n, dt = 2, 1e-15
    grids, tables, tabdata, w, y0 = far_case(q, which)
    b = batch(grids, tables, tabdata, w, y0, True, n)
    b.rk4(n, dt)
    yo = y0.reshape(-1).copy()
    orc.rk4(tables, tabdata, oracle_wires(w, tables, n), yo, n, dt, HBAR, p_stride=1, p_cap=n)
    assert np.isfinite(yo).all() and (b.wires()["status"] == 0).all()
    compare(b, b.state(), yo.reshape(-1, 4), NKS)


@pytest.mark.parametrize("q", [1e300, 1e-300, 5e-324])
@pytest.mark.parametrize("empty", [False, True])
def test_far_momenta_right_hand_side(cuda, q, empty):
    grids, tables, tabdata, w, y0 = far_case(q, "both")
    if empty:
        y0[:, 2:] = 0.0
    b = batch(grids, tables, tabdata, w, y0, True, 1)
    f = orc.rhs(tables, tabdata, oracle_wires(w, tables, 1), y0.reshape(-1), HBAR).reshape(-1, 4)
    assert np.isfinite(f).all()
    o, g = 0, b.rhs().cpu().numpy()
    for nk in NKS:  # (without a pulse n's own derivative may vanish: p's scale for it)
        top = np.abs(f[o:o + nk]).max()
        assert np.abs(g[o:o + nk] - f[o:o + nk]).max() < 1e-12 * top, nk
        o += nk
