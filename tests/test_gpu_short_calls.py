"""Short FP64 calls over several size classes: one library call whose launches
are chained on the caller's stream, without events or side streams.  The wires
get the bits of the side-stream form, what follows on the stream finds every
class done, and a captured call replays the same."""

import numpy as np
import pytest
import torch
from test_gpu_conv import batch, case

from pulsesuite_b200 import batch as batch_mod

pytestmark = pytest.mark.gpu

NKS = [1024, 64, 3, 128, 100, 256, 255, 512, 300]


def make(nks, kind, screened, p_cap):
    grids, tables, tabdata, w, y0 = case(nks, kind, screened, seed=7)
    return batch(grids, tables, tabdata, w, y0, screened, p_cap)


def step(b, how, n, f):
    if how == "rk4":
        b.rk4(n, 1e-16)
    else:
        b.leapfrog(f, n, 2e-17)


def outputs(b):
    w = b.wires()
    return [b.state(), b.y1.cpu().numpy(), b.P.cpu().numpy(), w["t"], w["steps"], w["status"]]


@pytest.mark.parametrize("how", ["rk4", "leap"])
@pytest.mark.parametrize("kind,screened", [("k0", False), ("distinct", True)])
def test_chained_and_forked(cuda, monkeypatch, how, kind, screened):
    n = 3
    f = torch.as_tensor(np.random.default_rng(2).uniform(-1e8, 1e8, (len(NKS), 8 * n)),
                        device="cuda")
    got = []
    for most in (0, batch_mod.CHAIN_STAGES):
        monkeypatch.setattr(batch_mod, "CHAIN_STAGES", most)
        b = make(NKS, kind, screened, n)
        with monkeypatch.context() as m:
            if most:  # no fork and join
                m.setattr(torch.cuda, "Event", None)
            for _ in range(4):
                step(b, how, n, f)
        got.append(outputs(b))
    for x, y in zip(*got):
        np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("how", ["rk4", "leap"])
def test_what_follows_finds_all_classes_done(cuda, how):
    """A long class first, short ones behind it: a copy queued after the call
    holds the finished long class."""
    nks, n = [1024, 64, 100, 200], 100
    b = make(nks, "k0", True, 0)
    f = torch.zeros((len(nks), 2 * n * 4), dtype=torch.float64, device="cuda")
    for _ in range(4):
        step(b, how, n, f)
        now, wires = b.y.clone(), b.d_wires.clone()
        torch.cuda.synchronize()
        assert torch.equal(now, b.y) and torch.equal(wires, b.d_wires)


def test_captured(cuda):
    n = 2
    a, b = make(NKS, "k0", False, n), make(NKS, "k0", False, n)
    g = a.capture(n, 1e-16)  # (advances the batch once)
    copies = []
    for _ in range(5):
        g.replay()
        copies.append(a.y.clone())
    b.rk4(n, 1e-16)
    for c in copies:
        b.rk4(n, 1e-16)
        assert torch.equal(c, b.y)
    assert torch.equal(a.P, b.P)
    np.testing.assert_array_equal(a.wires()["steps"], b.wires()["steps"])
