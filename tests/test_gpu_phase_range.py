"""Carrier phases far beyond a recording's: the phase of a sample, as f32, may
be any float.  Two samples, one of phase 0 and one of phase v, correlate to
max |1 +- exp(i v)| over the lags, |cos(v / 2)| or |sin(v / 2)| of its value
at v = 0.  The reduction holds 2/pi to 2^-108 and its low term, below 2^48
quarter turns for v < 3e30, is rounded to 2^-6 of one twice: 0.035 quarter turns
in all, 0.055 radians, half of that in the ratio."""
import numpy as np
import pytest

import tga

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("v", [3.0, 1.0e6, 1.0e15, 9.9e29, 1.01e30, 1.3e30, 1.7e30, 2.2e30, 2.9e30])
def test_two_samples(v):
    n, fs, f = 64, 2.0e6, 1.0e6
    sig = np.zeros(n, np.float32)
    sig[5] = sig[40] = 1.0
    pp = np.zeros(n)
    got = []
    with tga.Context(0) as ctx:
        for p in (0.0, float(np.float32(v)) / f):
            pp[40] = p
            got.append(ctx.acquire_single(tga.GPS, sig, pp, fs, f, 0.0, 5, 32).signal_strength)
    ph = float(np.float32(pp[40] * f))
    want = max(abs(1 + np.exp(1j * ph)), abs(1 - np.exp(1j * ph))) / 2
    assert abs(got[1] / got[0] - want) <= (0.028 if v > 1e20 else 1e-5)
