"""The wire-space sources on k points that are not equidistant: a wire has the
same bits alone (4 positions a CTA) and in a batch (8), and the call takes
little more than on an equidistant grid, whose polarisation has a shorter form
(6 real sums of Nk^2 terms a position instead of 4: 1.5 times the work; below
2.5 asked, the best of several runs of one process each)."""

import pytest
import torch

from perf import cases
from pulsesuite_b200 import _lib, device

pytestmark = pytest.mark.gpu


def sources(s, kr, w=None, out=None):
    g, ptr = s["grid"], device.ptr
    common = (ptr(kr), ptr(s["r"]), ptr(s["window"]), g.L, g.dcv)
    if w is None:
        _lib.call("psb_full_sources_batch_f64", s["case"]["nw"], s["nk"], s["nr"], *common,
                  ptr(s["wpar"]), ptr(s["L3"]), ptr(s["out"]), device.stream_ptr())
        return s["out"]
    yw, sg = s["wpar"][w, :2].tolist()
    _lib.call("psb_full_sources_f64", s["nk"], s["nr"], *common, yw, sg, ptr(s["L3"][w]), ptr(out),
              device.stream_ptr())
    return out


def uneven(s):
    i = torch.arange(s["nk"], device="cuda")
    return s["kr"] + 1e-3 * (s["kr"][1] - s["kr"][0]) * torch.sin(i * 1.7)


@pytest.mark.parametrize("L,nw", [(30e-9, 80), (62e-9, 40), (130e-9, 17)])
def test_wire_alone_and_in_a_batch(cuda, L, nw):
    s = cases.prepare({"kind": "full", "nw": nw, "L": L, "screened": False}, 3)
    kr = uneven(s)
    assert (s["nr"] + 7) // 8 * nw >= 296  # the batch takes 8 positions a CTA
    all_ = sources(s, kr)
    for w in (0, nw // 2, nw - 1):
        out = torch.full_like(all_[w], float("nan"))
        assert torch.equal(sources(s, kr, w, out), all_[w]), w


@pytest.mark.parametrize("L,nw", [(100e-9, 1), (100e-9, 64), (250e-9, 1)])
def test_uneven_costs_little_more(cuda, L, nw):
    s = cases.prepare({"kind": "full", "nw": nw, "L": L, "screened": False}, 3)

    def best(kr):
        t = []
        for _ in range(8):
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            torch.cuda.synchronize()
            e[0].record()
            for _ in range(5):
                sources(s, kr)
            e[1].record()
            torch.cuda.synchronize()
            t.append(e[0].elapsed_time(e[1]) / 5)
        return min(t)

    even, other = best(s["kr"]), best(uneven(s))
    assert other < 2.5 * even, (even, other)
