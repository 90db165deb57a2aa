"""Rows whose residue groups are shared between CTAs (few rows in a call): the
cells of one PRN, one antenna and few bins, searched alone, must equal the same
cells out of a call with enough rows that no row is shared; residue counts
below, at and off the groups of every code length.  Numbers of Doppler bins
around the width of the bin reduction, and recordings whose rows start at
every byte alignment (each antenna must give the cells of a recording that
holds it alone).  All equalities are exact: the same FP32 values are compared,
and ties have one winner.
"""
import numpy as np
import pytest

import tga

pytestmark = pytest.mark.gpu
FIELDS = ("best_codephase", "best_freq_idx", "hypothesis", "signal_strength", "second_peak", "frequency")
NC_FIELDS = ("best_codephase", "best_freq_idx", "power", "second_power", "frequency")
SHAPES = [(tga.GPS, 1023, 1), (tga.GPS, 1023, 8), (tga.GPS, 1023, 9), (tga.GPS, 1023, 17), (tga.GALILEO, 4092, 2),
          (tga.GALILEO, 4092, 5), (tga.GALILEO, 4092, 16), (tga.L1C, 10230, 1), (tga.L1C, 10230, 5),
          (tga.L1C, 10230, 16)]


@pytest.fixture(scope="module")
def ctx():
    with tga.Context(0) as c:
        yield c


def _rows(n_ant, n_bytes, seed):
    return np.random.default_rng(seed).integers(0, 256, size=(n_ant, n_bytes), dtype=np.uint8)


@pytest.mark.parametrize("precision", [tga.PRECISION_FP32, tga.PRECISION_FP16_TC])
@pytest.mark.parametrize("const,chips,S", SHAPES)
def test_few_rows_equal_many(ctx, const, chips, S, precision):
    fs = 1.023e6 * S
    bits = _rows(6, (2 * chips * S + 7) // 8 + 3, 10 * S)
    prns = list(range(1, 27))
    kw = dict(mask=1 << const, center_freq=0.3e6, search_band=400.0)
    ctx.set_precision(precision)
    try:
        many = ctx.acquire_cells(bits, fs, prn_filter=prns, **kw)
        few = ctx.acquire_cells(bits[:1], fs, prn_filter=[2], **kw)
        two = ctx.acquire_cells(bits[:2], fs, prn_filter=[2, 5], **kw)
    finally:
        ctx.set_precision(tga.PRECISION_FP32)
    sel = lambda r, a, p: [c for c in range(len(r)) if r["antenna"][c] == a and r["prn"][c] == p][0]
    for r, cells in ((few, [(0, 2)]), (two, [(0, 2), (0, 5), (1, 2), (1, 5)])):
        for a, p in cells:
            for f in FIELDS:
                assert r[f][sel(r, a, p)] == many[f][sel(many, a, p)], (f, a, p)


@pytest.mark.parametrize("precision", [tga.PRECISION_FP32, tga.PRECISION_FP16_TC])
@pytest.mark.parametrize("const,chips,S", SHAPES)
def test_few_nc_rows_equal_many(ctx, const, chips, S, precision):
    fs, blocks = 1.023e6 * S, 2
    bits = _rows(6, (blocks * chips * S + 7) // 8 + 3, 11 * S)
    kw = dict(center_freq=0.3e6, bin_step_hz=120.0, n_bins=3, blocks=blocks)
    ctx.set_precision(precision)
    try:
        many = ctx.search_noncoherent(bits, fs, const, prns=list(range(1, 27)), **kw)
        few = ctx.search_noncoherent(bits[:1], fs, const, prns=[2], **kw)
    finally:
        ctx.set_precision(tga.PRECISION_FP32)
    at = [c for c in range(len(many)) if many["antenna"][c] == 0 and many["prn"][c] == 2][0]
    for f in NC_FIELDS:
        assert few[f][0] == many[f][at], f


@pytest.mark.parametrize("n_bins", [1, 2, 15, 16, 17, 33])
def test_bin_reduction_widths(ctx, n_bins):
    """The reduction's choice against one search per bin."""
    S, fs, step = 4, 4.092e6, 300.0
    bits = _rows(3, 3 * 4092 // 8, n_bins)
    kw = dict(prns=[1, 7, 32], bin_step_hz=step, blocks=2)
    r = ctx.search_noncoherent(bits, fs, tga.GPS, center_freq=0.4e6, n_bins=n_bins, **kw)
    each = [ctx.search_noncoherent(bits, fs, tga.GPS, center_freq=0.4e6 + (b - (n_bins - 1) // 2) * step, n_bins=1,
                                   **kw) for b in range(n_bins)]
    power = np.stack([e["power"] for e in each])
    assert np.array_equal(r["power"], power.max(axis=0))
    pick = n_bins - 1 - power[::-1].argmax(axis=0)  # the last of equal maxima
    assert np.array_equal(r["best_freq_idx"], pick)
    for f in ("best_codephase", "second_power"):
        assert np.array_equal(r[f], np.stack([e[f] for e in each])[pick, np.arange(len(r))]), f


@pytest.mark.parametrize("extra", [1, 3, 8, 15, 16, 1021])
def test_rows_at_every_alignment(ctx, extra):
    """17 rows of an odd (or even) number of bytes: starts at all offsets of a
    16-byte word; the mean enters every sample."""
    rng = np.random.default_rng(extra)
    n = 2 * 1023 * 2 // 8 + 1 + extra
    bits = rng.integers(0, 256, size=(17, n), dtype=np.uint8) | rng.integers(0, 256, size=(17, 1), dtype=np.uint8)
    kw = dict(mask=1 << tga.GPS, prn_filter=[3], center_freq=0.3e6, search_band=400.0)
    r = ctx.acquire_cells(bits, 2.046e6, **kw)
    for a in range(17):
        one = ctx.acquire_cells(bits[a:a + 1], 2.046e6, **kw)
        for f in FIELDS:
            assert one[f][0] == r[f][r["antenna"] == a][0], (a, f)


@pytest.mark.parametrize("const,chips,S,band", [(tga.L1C, 10230, 1, 600.0), (tga.L1C, 10230, 3, 900.0),
                                                (tga.GALILEO, 4092, 4, 2000.0)])
def test_antenna_groups_share_phasors(ctx, const, chips, S, band):
    """Seven antennas in groups that leave a shorter last one, each against a
    search of that antenna alone."""
    fs = 1.023e6 * S
    bits = _rows(7, (2 * chips * S + 7) // 8 + 3, 12 * S)
    kw = dict(mask=1 << const, prn_filter=[4], center_freq=0.3e6, search_band=band)
    r = ctx.acquire_cells(bits, fs, **kw)
    for a in range(7):
        one = ctx.acquire_cells(bits[a:a + 1], fs, **kw)
        for f in FIELDS:
            assert one[f][0] == r[f][r["antenna"] == a][0], (a, f)


@pytest.mark.parametrize("n_ant,n_prn", [(1, 1), (6, 26)])
@pytest.mark.parametrize("const,chips,S", [(tga.GPS, 1023, 9), (tga.GALILEO, 4092, 5), (tga.L1C, 10230, 3)])
def test_all_equal_takes_the_last(ctx, const, chips, S, n_ant, n_prn):
    """A constant recording has no signal left after its mean: every value is
    0, and of equal values the last lag and the last bin are taken."""
    P, fs = chips * S, 1.023e6 * S
    bits = np.full((n_ant, (2 * P + 7) // 8), 255, dtype=np.uint8)
    r = ctx.acquire_cells(bits, fs, mask=1 << const, prn_filter=list(range(1, n_prn + 1)), center_freq=0.3e6,
                          search_band=600.0)
    assert len(r) == n_ant * n_prn
    assert np.all(r["best_codephase"] == P - 1)
    assert np.all(r["best_freq_idx"] == 4) and np.all(r["hypothesis"] == 0)


@pytest.mark.parametrize("precision", [tga.PRECISION_FP32, tga.PRECISION_FP16_TC])
@pytest.mark.parametrize("const,chips,S", [(tga.GPS, 1023, 1), (tga.GPS, 1023, 9), (tga.GALILEO, 4092, 3),
                                           (tga.L1C, 10230, 1), (tga.L1C, 10230, 3)])
def test_odd_numbers_of_sequences(ctx, const, chips, S, precision):
    """One antenna, bin and block: S sequences, the last of them alone in its
    forward transform; against the same cell among three antennas."""
    fs = 1.023e6 * S
    bits = _rows(3, (chips * S + 7) // 8 + 2, 13 * S)
    kw = dict(bin_step_hz=200.0, blocks=1)
    ctx.set_precision(precision)
    try:
        one = ctx.search_noncoherent(bits[1:2], fs, const, prns=[3], center_freq=0.3e6, n_bins=1, **kw)
        many = ctx.search_noncoherent(bits, fs, const, prns=[3], center_freq=0.3e6, n_bins=1, **kw)
    finally:
        ctx.set_precision(tga.PRECISION_FP32)
    at = [c for c in range(len(many)) if many["antenna"][c] == 1][0]
    for f in NC_FIELDS:
        assert one[f][0] == many[f][at], f


@pytest.mark.parametrize("const,chips,S,n_prn,n_bins", [(tga.GPS, 1023, 9, 32, 33), (tga.GALILEO, 4092, 3, 50, 33),
                                                        (tga.GALILEO, 4092, 6, 7, 51), (tga.L1C, 10230, 2, 63, 33)])
def test_tensor_core_shares(ctx, const, chips, S, n_prn, n_bins):
    """Numbers of items between one and three times the SMs, whose rounds are
    divided: the FP32 cells, drop-in and non-coherent."""
    fs = 1.023e6 * S
    bits = _rows(1, (3 * chips * S + 7) // 8 + 2, 14 * S)
    prns = list(range(1, n_prn + 1))
    a, b = [], []
    for out, precision in ((a, tga.PRECISION_FP32), (b, tga.PRECISION_FP16_TC)):
        ctx.set_precision(precision)
        try:
            out.append(ctx.acquire_cells(bits, fs, mask=1 << const, prn_filter=prns, center_freq=0.3e6,
                                         search_band=150.0 * (n_bins - 1)))
            out.append(ctx.search_noncoherent(bits, fs, const, prns=prns, center_freq=0.3e6, bin_step_hz=150.0,
                                              n_bins=n_bins, blocks=3))
        finally:
            ctx.set_precision(tga.PRECISION_FP32)
    for f in FIELDS:
        assert np.array_equal(a[0][f], b[0][f]), f
    for f in NC_FIELDS:
        assert np.array_equal(a[1][f], b[1][f]), f
