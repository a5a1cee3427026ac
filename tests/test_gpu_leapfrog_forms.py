"""``WireBatch.leapfrog`` on a split batch: the leapfrog runs in FP64 whatever
the form, one launch per size class, and a split batch may have more of these
classes than launches of its own step.  Every wire gets the bits of the plain
batch and takes its steps."""

import numpy as np
import pytest
import torch
from test_gpu_parity import uneven_case

from pulsesuite_b200 import _lib
from pulsesuite_b200.batch import WireBatch


@pytest.mark.gpu
@pytest.mark.parametrize("screened", [False, True])
@pytest.mark.parametrize("nks", [[64, 64, 128], [60, 128, 250, 256, 500], [64, 128, 600, 256],
                                 [100, 90]])
def test_leapfrog_of_a_split_batch(cuda, nks, screened):
    steps = 3
    grids, w = uneven_case(nks, seed=5, screened=screened, nsteps=steps)
    y = np.random.default_rng(1).uniform(0.0, 0.4, (sum(nks), 4))
    f = torch.as_tensor(np.random.default_rng(2).uniform(-1e8, 1e8, (len(nks), 2 * steps)),
                        device="cuda")
    kw = {} if screened else {"tune": False, "split_w": {n: 4 if n > 512 else 8 for n in nks}}
    got = []
    for form, more in (("plain", {}), ("split", kw)):
        b = WireBatch(grids, w, screened=screened, p_cap=steps, form=form, **more)
        b.set_state(y, y)
        b.leapfrog(f, steps, 2e-17)
        assert (b.wires()["steps"] == steps).all() and (b.wires()["status"] == 0).all(), form
        got.append((b.state(), b.y1.cpu().numpy(), b.P.cpu().numpy()))
    for x, z in zip(*got):
        np.testing.assert_array_equal(x, z)


class _Stream:
    def __init__(self):
        self.waits = []

    def wait_event(self, e):
        self.waits.append(e)


class _Event:
    def record(self, stream):
        self.on = stream


def test_no_launch_is_dropped(monkeypatch):
    """More launches than side streams: an error, not a shorter list."""
    monkeypatch.setattr(torch.cuda, "Event", _Event)
    b = object.__new__(WireBatch)
    b.side_streams = [_Stream(), _Stream()]
    main, ran = _Stream(), []
    calls = [lambda s, i=i: ran.append((i, s)) for i in range(3)]
    with pytest.raises(_lib.PsbError):
        b._concurrent(calls, main)
    assert not ran
    b._concurrent(calls[:2], main)
    assert ran == [(0, b.side_streams[0]), (1, b.side_streams[1])]
    assert [e.on for e in main.waits] == b.side_streams
    ran.clear()
    b._concurrent(calls[:1], main)
    assert ran == [(0, main)]
