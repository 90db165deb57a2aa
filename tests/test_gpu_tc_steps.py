"""Tensor-core correlator at the edges of its steps: residue counts that leave
part of a step empty, PRN counts below and off the number of chains, few rows
(an item's PRNs split over CTAs), one and odd numbers of coherent blocks.

Noise-only recordings, whose near-equal rows are the hardest for the row
choice: every cell must equal the FP32 search's, and the FP16 row keys must
lie within the bound that the candidate rule assumes (2^-8 of the largest row
of their (antenna, PRN)).
"""
import numpy as np
import pytest

import tga

pytestmark = pytest.mark.gpu
KEY_BOUND = 2.0 ** -8
FIELDS = ("best_codephase", "best_freq_idx", "hypothesis", "signal_strength", "second_peak", "frequency")
NC_FIELDS = ("best_codephase", "best_freq_idx", "power", "second_power", "frequency")


@pytest.fixture(scope="module")
def ctxs():
    a, b = tga.Context(0), tga.Context(0)
    b.set_precision(tga.PRECISION_FP16_TC)
    yield a, b
    a.close()
    b.close()


def _rows(n_ant, n, seed):
    return np.random.default_rng(seed).integers(0, 256, size=(n_ant, n // 8), dtype=np.uint8)


# (constellation, chips, samples per chip): one residue up to several steps
SHAPES = [(tga.GPS, 1023, 1), (tga.GPS, 1023, 3), (tga.GPS, 1023, 5), (tga.GPS, 1023, 9), (tga.GALILEO, 4092, 1),
          (tga.GALILEO, 4092, 3), (tga.GALILEO, 4092, 6), (tga.L1C, 10230, 2), (tga.L1C, 10230, 6)]


@pytest.mark.parametrize("n_prn", [1, 2, 3, 7])
@pytest.mark.parametrize("const,chips,S", SHAPES)
def test_ragged_steps_equal_fp32(ctxs, const, chips, S, n_prn):
    fs = 1.023e6 * S
    bits = _rows(2, 2 * chips * S // 8 * 8 + 64, 100 * S + n_prn)
    kw = dict(mask=1 << const, prn_filter=list(range(1, n_prn + 1)), center_freq=0.3e6, search_band=450.0)
    a, b = (c.acquire_cells(bits, fs, **kw) for c in ctxs)
    for f in FIELDS:
        assert np.array_equal(a[f], b[f]), f
    pa, pb = (c.row_peaks(chips)[0].reshape(2, -1, n_prn) for c in ctxs)  # 4 bins x 2 hypotheses per antenna
    assert np.max(np.abs(pa - pb) / pa.max(axis=1, keepdims=True)) < KEY_BOUND


@pytest.mark.parametrize("n_prn,blocks", [(1, 1), (2, 3), (3, 2), (5, 5)])
@pytest.mark.parametrize("const,chips,S", [(tga.GPS, 1023, 5), (tga.GALILEO, 4092, 3), (tga.L1C, 10230, 2)])
def test_ragged_blocks_equal_fp32(ctxs, const, chips, S, n_prn, blocks):
    fs = 1.023e6 * S
    bits = _rows(2, blocks * chips * S // 8 * 8 + 64, 7 * S + blocks)
    kw = dict(prns=list(range(1, n_prn + 1)), center_freq=0.3e6, bin_step_hz=50.0, n_bins=3, blocks=blocks)
    a, b = (c.search_noncoherent(bits, fs, const, **kw) for c in ctxs)
    for f in NC_FIELDS:
        assert np.array_equal(a[f], b[f]), f
