"""RFI scan at record lengths that take every pass radix of the f64 FFT (32,
16, 8, 4, 2; 33, 25, 15, 31, 13, 11, 7, 5, 3; the R-term sum), its smallest
records, and a row whose powers are all but equal (the median's list of
gathered bins overflows).  Against the FP64 oracle: same lines at the same
bins, excess within 1e-9 dB relative as for the other lengths.
"""
import numpy as np
import pytest

import rfi_oracle as RO
import tga

pytestmark = pytest.mark.gpu
FS = 16.368e6
# row_bytes; the transform has 4 row_bytes points
ROWS = {"2^3": 2, "2^5": 8, "2^13": 2048, "2^2x3": 3, "2^4x15": 60, "2^3x7x13": 182, "2^4x11x5^2": 1100, "2^3x3x3x17": 306,
        "2^5x25x33x31": 8 * 25 * 33 * 31}


def _same(got, want):
    for g, w in zip(got, want):
        assert g["dead"] == w["dead"] and len(g["lines"]) == len(w["lines"])
        for a, b in zip(g["lines"], w["lines"]):
            assert a["frequency"] == b["frequency"]
            assert abs(a["excess_db"] - b["excess_db"]) <= 1e-9 * abs(b["excess_db"])


@pytest.mark.parametrize("row_bytes", list(ROWS.values()), ids=list(ROWS))
def test_every_radix(row_bytes):
    n = row_bytes * 8
    rng = np.random.default_rng(row_bytes)
    wave = np.sign(np.cos(2 * np.pi * (1.7e6 / FS) * np.arange(n) + 0.3))
    rows = np.stack([0.8 * wave + rng.standard_normal(n), rng.standard_normal(n)])
    bits = np.packbits(rows >= 0.0, axis=1)
    with tga.Context(0) as ctx:
        got = ctx.rfi_scan(bits, FS)
    _same(got, RO.run(bits, FS))
    if n >= 4096:
        assert got[0]["lines"]


def test_nearly_equal_powers():
    """One sample off in a constant row: every power equals 4 to rounding, so
    thousands of bins share the median's leading bits."""
    bits = np.full((1, 4096), 255, np.uint8)
    bits[0, 1234] = 0xF7
    with tga.Context(0) as ctx:
        got = ctx.rfi_scan(bits, FS)
    _same(got, RO.run(bits, FS))
    assert not got[0]["dead"] and got[0]["lines"] == []
