"""Generic path on a signal with a NaN: every correlation is a NaN, which is
above nothing, so the first bin and [c, c] stand, as in a serial walk over the
bins that replaces its choice by a value not below it."""
import numpy as np
import pytest

import tga
from testutil import phasepoints

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [4000, 2 * 1009], ids=["direct", "bluestein"])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_first_bin_stands(n, bad):
    fs = 2.0e6
    sig = np.random.default_rng(n).standard_normal(n).astype(np.float32)
    with tga.Context(0) as ctx:
        a = ctx.acquire_single(tga.GPS, sig, phasepoints(fs, n), fs, 0.0, 3000.0, 5, 2000)
        sig[17] = bad
        r = ctx.acquire_single(tga.GPS, sig, phasepoints(fs, n), fs, 0.0, 3000.0, 5, 2000)
        assert r.path == 1 and r.best_freq_idx == 0 and r.hypothesis == 0
        assert np.isnan(r.signal_strength)
        sig[17] = 0.0
        b = ctx.acquire_single(tga.GPS, sig, phasepoints(fs, n), fs, 0.0, 3000.0, 5, 2000)
        assert np.isfinite(a.signal_strength) and np.isfinite(b.signal_strength)
