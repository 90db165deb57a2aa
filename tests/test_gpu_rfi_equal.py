"""RFI scan of rows whose powers are mostly equal, so that the bins sharing the
median's leading digits do not fit the list: constant rows, and a comb of
single samples with one more beside it, whose lines stand on a floor of equal
powers (the median enters their excess).  Alone and beside noise; against the
FP64 oracle.  A constant row must not cost much more than one of noise."""
import time

import numpy as np
import pytest

import rfi_oracle as RO
import tga

pytestmark = pytest.mark.gpu
FS = 16.368e6


def _comb(row_bytes):
    n = row_bytes * 8
    b = np.ones(n, np.uint8)
    b[n // 64::n // 32] = 0
    b[n // 64 + 1] = 0
    return np.packbits(b)


@pytest.mark.parametrize("row_bytes", [4096, 8 * 25 * 33 * 4, 204600])
def test_equal_powers(row_bytes):
    rng = np.random.default_rng(row_bytes)
    bits = np.stack([_comb(row_bytes), np.full(row_bytes, 255, np.uint8), rng.integers(0, 256, row_bytes, dtype=np.uint8),
                     np.zeros(row_bytes, np.uint8), _comb(row_bytes)])
    want = RO.run(bits, FS)
    assert len(want[0]["lines"]) == 3 and want[1]["dead"] and want[3]["dead"]
    with tga.Context(0) as ctx:
        for rows in ([0, 1, 2, 3, 4], [0], [1]):
            got = ctx.rfi_scan(bits[rows], FS)
            for g, w in zip(got, [want[r] for r in rows]):
                assert g["dead"] == w["dead"] and len(g["lines"]) == len(w["lines"])
                for a, b in zip(g["lines"], w["lines"]):
                    assert a["frequency"] == b["frequency"]
                    assert abs(a["excess_db"] - b["excess_db"]) <= 1e-9 * abs(b["excess_db"])


def test_constant_row_costs_like_noise():
    """100 ms of one antenna: 1.4 times the time of noise; one CTA walking the
    row takes six times."""
    n = 204600
    noise = np.random.default_rng(1).integers(0, 256, (1, n), dtype=np.uint8)
    with tga.Context(0) as ctx:
        def best(bits):
            t = []
            for _ in range(12):
                a = time.perf_counter()
                ctx.rfi_scan(bits, FS)
                t.append(time.perf_counter() - a)
            return min(t)
        assert best(np.full((1, n), 255, np.uint8)) < 3.0 * best(noise)
