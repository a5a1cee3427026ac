"""Groups of the split form: every wire in one slot whatever the count, and the
per-wire kernel's widths where they were measured (148 SMs)."""

import numpy as np
import pytest

from pulsesuite_b200 import abi
from pulsesuite_b200.batch import groups_of, wire_group


@pytest.mark.parametrize("wg", [1, 3, 4, 8, 16])
@pytest.mark.parametrize("n", [1, 2, 15, 16, 17, 47, 48, 49, 1000])
def test_every_wire_has_one_slot(wg, n):
    wires = np.random.default_rng(n).permutation(3 * n)[:n]
    g = groups_of(5, wires, wg)
    assert g.dtype == abi.SPLIT_GROUP_DTYPE and len(g) == -(-n // wg)
    assert (g["table"] == 5).all() and (g["nw"] >= 1).all() and (g["nw"] <= wg).all()
    used = np.arange(abi.PSB_SPLIT_WMAX)[None, :] < g["nw"][:, None]
    np.testing.assert_array_equal(g["wire"][used], wires)  # in order, none twice
    assert (g["wire"][~used] == -1).all()


# Screened wires: 1600 of Nk 512 (at most ten a group) 2.12 ms in two waves of
# groups of 6 against 3.37 with groups of ten, 16384 19.2 with 8 against 20.1;
# an uneven batch of 1024 on fifteen grids has ten SMs a grid, 1.11 ms with 7 or
# so a group against 1.61 with one; up to a wire an SM none waits for another.
@pytest.mark.parametrize("n,wmax,sms,want", [(1600, 10, 148, 6), (16384, 10, 148, 8),
                                             (70, 16, 148 / 15, 7), (148, 10, 148, 1),
                                             (149, 10, 148, 2), (1, 16, 0.3, 1)])
def test_measured_widths(n, wmax, sms, want):
    assert wire_group(n, wmax, sms) == want
