"""Front end with antennas that share carrier phasors, at many samples a chip:
S = 48 and 64 take the most shared memory (134 KB a CTA at 64, one CTA per SM).
Seven antennas, in groups that leave a shorter last one, each against a search
of that antenna alone, which computes its phasors for itself."""
import numpy as np
import pytest

import tga

pytestmark = pytest.mark.gpu
FIELDS = ("best_codephase", "best_freq_idx", "hypothesis", "signal_strength", "second_peak", "frequency")


@pytest.mark.parametrize("S", [47, 48, 64])
@pytest.mark.parametrize("const,chips,band", [(tga.GPS, 1023, 6000.0), (tga.GALILEO, 4092, 1800.0), (tga.L1C, 10230, 600.0)])
def test_groups_at_many_samples_a_chip(const, chips, band, S):
    fs = 1.023e6 * S
    bits = np.random.default_rng(S).integers(0, 256, size=(7, (2 * chips * S + 7) // 8 + 3), dtype=np.uint8)
    kw = dict(mask=1 << const, prn_filter=[4], center_freq=0.3e6, search_band=band)
    with tga.Context(0) as ctx:
        r = ctx.acquire_cells(bits, fs, **kw)
        for a in range(7):
            one = ctx.acquire_cells(bits[a:a + 1], fs, **kw)
            for f in FIELDS:
                assert one[f][0] == r[f][r["antenna"] == a][0], (a, f)
