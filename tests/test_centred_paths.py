"""Which arrays fftg / ifftg hand to the library's in-place passes: the rest
takes the same operations in numpy, with the same bits."""

import importlib.util

import numpy as np
import pytest
from test_centred_host import written_out

from pulsesuite_b200 import _lib
from pulsesuite_b200 import wirespace as ws


def signals(shape, seed=3):
    rng = np.random.default_rng(seed)
    return rng.standard_normal(shape) + 1j * rng.standard_normal(shape)


def test_numpy_whose_transforms_take_no_out(monkeypatch):
    """numpy 1.x: the transforms have no out= argument."""
    fft, ifft = np.fft.fft, np.fft.ifft
    monkeypatch.setattr(np.fft, "fft", lambda a, n=None, axis=-1, norm=None: fft(a, n, axis, norm))
    monkeypatch.setattr(np.fft, "ifft",
                        lambda a, n=None, axis=-1, norm=None: ifft(a, n, axis, norm))
    spec = importlib.util.spec_from_file_location("pulsesuite_b200.wirespace_again", ws.__file__)
    again = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(again)
    F = signals((8, 230))
    for f, inverse in ((again.fftg, False), (again.ifftg, True)):
        G = F.copy()
        f(G)
        np.testing.assert_array_equal(G, written_out(F, inverse))


def test_arrays_the_library_cannot_take(monkeypatch):
    """Signals whose doubles do not lie on 8-byte boundaries, in rows apart, or
    read-only: never handed over."""
    monkeypatch.setattr(_lib, "call", lambda *a: pytest.fail("handed to the library"))
    F = signals((8, 230))
    raw = np.empty(F.nbytes + 4, np.uint8)[4:].view(np.complex128).reshape(F.shape)
    assert not raw.flags.aligned
    strided = np.empty((8, 460), np.complex128)[:, ::2]
    for G in (raw, strided):
        for f, inverse in ((ws.fftg, False), (ws.ifftg, True)):
            G[...] = F
            f(G)
            np.testing.assert_array_equal(G, written_out(F, inverse))
    G = F.copy()
    G.flags.writeable = False
    with pytest.raises(ValueError):
        ws.fftg(G)


@pytest.mark.parametrize("shape,library", [((64,), False), ((3, 85), False), ((256,), True),
                                           ((8, 32), True), ((5, 230), True)])
def test_small_signals_stay_in_numpy(monkeypatch, shape, library):
    """Below 256 values the library's two calls cost more than they save."""
    real, calls = _lib.call, []
    monkeypatch.setattr(_lib, "call", lambda *a: calls.append(a[0]) or real(*a))
    F = signals(shape)
    for f, inverse in ((ws.fftg, False), (ws.ifftg, True)):
        G = F.copy()
        f(G)
        np.testing.assert_array_equal(G, written_out(F, inverse))
    assert calls == (["psb_centred_c128"] * 4 if library else [])
