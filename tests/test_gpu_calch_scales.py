"""psb_calch_f64 on large grids, electrons and holes of very different
occupation: the self-energy of each keeps its own precision, although the two
occupations travel through one complex transform.

Tolerance 4e-14 of a column's own largest sum, derived: the transforms of M <=
2048 points carry 2^-53 * 3 log2 M ~ 4e-15 of the larger of the two signals,
which the kernel brings within a factor of two of one another; spectra and
products of three of them and the pass through distinct tables' mirrored
frequencies a factor of four; with a margin of two.
"""

import numpy as np
import pytest
import torch
from test_gpu_conv import any_grid, batch, oracle_wires

from pulsesuite_b200 import _lib, abi, device
from pulsesuite_b200 import grid as pgrid

pytestmark = pytest.mark.gpu

TOL = 4e-14


def sums(V, n):
    """sum_k' V(|k - k'|) n_k', k' != k, in long double."""
    nk = len(n)
    d = np.abs(np.arange(nk)[:, None] - np.arange(nk)[None, :])
    T = V.astype(np.longdouble)
    T[0] = 0.0
    return T[d] @ n.astype(np.longdouble)


@pytest.mark.parametrize("ratio", [1.0, 1e-3, 1e-8, 1e3, 1e-200, 1e-310, 0.0])
@pytest.mark.parametrize("kind", ["k0", "distinct"])
@pytest.mark.parametrize("nk", [258, 511, 1024])
def test_self_energies_keep_their_own_scale(cuda, nk, kind, ratio):
    g, blk = any_grid(nk, kind)
    blk = np.array(blk).reshape(9, nk)
    blk[3:5] = 0.0  # band energies: Hee, Hhh are the self-energies alone
    tables, tabdata = pgrid.pack_tables([g], [blk.reshape(-1)], screened=False)
    w = np.zeros(1, dtype=abi.WIRE_DTYPE)
    x = np.linspace(-2, 2, nk)
    ne = 0.4 * np.exp(-x * x)
    nh = ratio * (0.3 * np.exp(-(x - 0.3) ** 2) + 0.01)
    if ratio > 1.0:
        ne, nh = ne / ratio, nh / ratio
    y = np.stack([0.1 * ne, -0.2 * ne, ne, nh], 1)
    b = batch([g], tables, tabdata, w, y, False, 0)
    h = torch.empty_like(b.y)
    _lib.call("psb_calch_f64", *b._common(), device.ptr(b.y), device.ptr(h), b.n_state, b.nkmax,
              b.tab_flags, abi.as_ptr(b.model), device.stream_ptr())
    h = h.cpu().numpy()
    assert (oracle_wires(w, tables, 0)["off"] == 0).all()
    for col, t, n in ((0, 0, y[:, 0]), (1, 0, y[:, 1]), (2, 1, ne), (3, 2, nh)):
        want = sums(blk[t], n) * (1.0 if col < 2 else -1.0)
        top = np.abs(want).max()
        # (below 1e-308 the spacing of doubles itself is the error)
        assert np.abs(h[:, col] - want).max() <= max(TOL * top, 1e-323 * nk), col
