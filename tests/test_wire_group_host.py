"""wire_group: the group size of the per-wire split kernel against every other
choice, by the time that its rule assigns (waves of CTAs times w + 1)."""

import pytest

from pulsesuite_b200.batch import wire_cost, wire_group


@pytest.mark.parametrize("wmax", [1, 2, 9, 16])
@pytest.mark.parametrize("sms", [0.2, 1.0, 9.7, 148.0])
def test_wire_group(wmax, sms):
    s = max(1, round(sms))
    for n in (1, 2, 3, 10, 147, 148, 149, 700, 1480, 1600, 16384):
        w = wire_group(n, wmax, sms)
        assert 1 <= w <= wmax
        times = [-(-(-(-n // v)) // s) * (v + 1) for v in range(1, wmax + 1)]
        assert times[w - 1] == min(times)


def test_wire_cost_grows():
    costs = [wire_cost(nk) for nk in range(2, 1025)]
    assert costs[0] > 0 and all(a < b for a, b in zip(costs, costs[1:]))
