"""The batched split kernel where its arrangement changes: row tiles of 128,
slices of 64, the three ways the Coulomb tiles are fed (all resident, one by
one, row by row) and the state's move out of shared memory, at every group
width, with a group that is not full.

The digit products are exact, so every width gives the same bits.  Against the
FP64 form the bounds are those of the split form (2^-24.6 of the scale in V
and X, FP32 stage points): 1e-6 in P(t), 1e-5 in the state.
"""

import numpy as np
import pytest
from helpers import relerr
from test_gpu_parity import uneven_case

from pulsesuite_b200 import _lib
from pulsesuite_b200.batch import WireBatch

pytestmark = pytest.mark.gpu

EDGES = [62, 64, 66, 126, 128, 130, 190, 194, 254, 256, 258, 320, 322, 384, 510, 512, 514, 642,
         1022, 1024]


@pytest.mark.parametrize("nk", EDGES)
def test_split_edges(cuda, nk):
    steps, dt = 9, 1e-15
    grids, w = uneven_case([nk] * 5, seed=nk, nsteps=steps)
    w["t0"] = 3e-15  # the columns outgrow their scales within the run
    ref = WireBatch(grids, w, p_cap=steps)
    ref.rk4(4, dt)
    ref.rk4(steps - 4, dt)
    yr, Pr = ref.state(), ref.P.cpu().numpy()
    first = None
    for width in (4, 8, 16):
        if nk > _lib.load().psb_split_max_nk(width):
            continue
        b = WireBatch(grids, w, p_cap=steps, form="split", tune=False, split_w={nk: width})
        b.rk4(4, dt)
        b.rk4(steps - 4, dt)
        assert (b.wires()["status"] == 0).all() and (b.wires()["steps"] == steps).all()
        y, P = b.state(), b.P.cpu().numpy()
        if first is None:
            first = y, P
            assert relerr(P, Pr) < 1e-6
            for c in (slice(0, 2), slice(2, 3), slice(3, 4)):
                assert relerr(y[:, c], yr[:, c]) < 1e-5
        np.testing.assert_array_equal(y, first[0])
        np.testing.assert_array_equal(P, first[1])


@pytest.mark.parametrize("nk", [64, 66, 126, 130, 254, 258, 510, 512, 514, 1022, 1024])
def test_split_wire_edges(cuda, nk):
    """Screened wires (a matrix each): groups of 1, an odd and an even number
    of wires give the same bits, at the edges of the row tiles and on both
    sides of Nk 512, where an epilogue warp's tiles double."""
    steps, dt = 6, 1e-15
    grids, w = uneven_case([nk] * 4, seed=nk, screened=True, nsteps=steps)
    w["t0"] = 3e-15
    ref = WireBatch(grids, w, screened=True, p_cap=steps)
    ref.rk4(steps, dt)
    yr, Pr = ref.state(), ref.P.cpu().numpy()
    first = None
    for width in (4, 3, 1):
        b = WireBatch(grids, w, screened=True, p_cap=steps, form="split", split_w={nk: width})
        b.rk4(steps, dt)
        assert (b.wires()["status"] == 0).all() and (b.wires()["steps"] == steps).all()
        y, P = b.state(), b.P.cpu().numpy()
        if first is None:
            first = y, P
            assert relerr(P, Pr) < 1e-6
            for c in (slice(0, 2), slice(2, 3), slice(3, 4)):
                assert relerr(y[:, c], yr[:, c]) < 1e-5
        np.testing.assert_array_equal(y, first[0])
        np.testing.assert_array_equal(P, first[1])
