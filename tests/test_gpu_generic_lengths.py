"""Generic path at window lengths that take every radix of its FFT (32, 16, 8,
4, 2; 33, 25, 15, 31, 13, 11, 7, 5, 3; the R-term sum for 17 and 61) and
Bluestein's transform (a prime factor above 64), one and odd lengths, and the
BOC codes' replica, against the oracle under the suite's parity rule."""
import numpy as np
import pytest

import acq_oracle as O
import tga
from parity import assert_cell_parity
from testutil import phasepoints

pytestmark = pytest.mark.gpu
LENGTHS = [31, 64, 2 * 33, 2 * 31, 3 * 7 * 13, 11 * 17, 16 * 25, 1009, 2 * 15 * 61, 2 * 1009, 8 * 11 * 25, 5 * 7 * 67, 4000,
           4095, 4096]


@pytest.fixture(scope="module")
def ctx():
    c = tga.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("const,prn", [(O.GPS, 5), (O.L1C, 3)], ids=["gps", "l1c-boc"])
@pytest.mark.parametrize("n", LENGTHS)
def test_generic_lengths(ctx, const, prn, n):
    fs, period = 2.0e6, 2000
    rng = np.random.default_rng(n)
    code = O.resampled_code(const, prn, float(period), n)
    sig = (np.roll(code, 7) + 0.5 * rng.standard_normal(n)).astype(np.float32)
    pp = phasepoints(fs, n)
    g = ctx.acquire_single(const, sig, pp, fs, 0.0, 3000.0, prn, period)
    r = O.acquire_single(const, sig, pp, fs, 0.0, 3000.0, prn, period, grid=True)
    assert g.path == 1
    assert_cell_parity(dict(signal_strength=g.signal_strength, second_peak=g.second_peak,
                            best_codephase=g.best_codephase, best_freq_idx=g.best_freq_idx, frequency=g.frequency,
                            codephase_frac=g.codephase_frac), r, n)
