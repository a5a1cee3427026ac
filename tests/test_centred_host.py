"""fftg / ifftg with the library's sign-and-scale passes (psb_centred_c128)
against the same operations written out in numpy: the same bits, for one
signal and many, odd and even lengths, and values that are not finite."""

import numpy as np
import pytest

from pulsesuite_b200 import wirespace as ws


def written_out(F, inverse):
    F = F.copy()
    F[..., 1::2] = -F[..., 1::2]
    F[...] = np.fft.ifft(F, axis=-1) if inverse else np.fft.fft(F, axis=-1)
    F[..., 1::2] = -F[..., 1::2]
    n = float(F.shape[-1])
    return -F * n if inverse else -F / n


@pytest.mark.parametrize("shape", [(1,), (2,), (7,), (230,), (5, 64), (3, 1), (2, 3, 46)])
@pytest.mark.parametrize("special", [False, True])
def test_centred_passes(shape, special):
    rng = np.random.default_rng(3)
    F = rng.standard_normal(shape) * 1e7 + 1j * rng.standard_normal(shape)
    if special:
        F.flat[0], F.flat[-1] = complex(np.inf, 1.0), complex(0.0, np.nan)
    for f, inverse in ((ws.fftg, False), (ws.ifftg, True)):
        G, H = F.copy(), np.stack([F, F], axis=-1)[..., 0]   # contiguous, strided
        with np.errstate(all="ignore"):
            f(G)
            f(H)
            want = written_out(F, inverse)
        np.testing.assert_array_equal(G, want)
        np.testing.assert_array_equal(H, want)
