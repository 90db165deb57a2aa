"""Frequency scan of the fine acquisition at the edges of its tiles: one
antenna, an odd number, more than a tile of 24; scans of one point, within one
tile of 21 points and over two; a window that ends inside a chunk.

The power at the scan's centre must equal tga_fine_eval's at the same point
(both sum the same FP32 products, in other orders: 1e-6 of it), and the scan
must take the refinement to the satellite's frequency from a start that only a
point of its second tile is near.
"""
import numpy as np
import pytest

import tga

pytestmark = pytest.mark.gpu
FS, IF = 16.368e6, 4.092e6
N = 65472 + 5 * 8  # 4 ms and a ragged end


def _rows(n_ant, prn, tau, dop):
    rng = np.random.default_rng(n_ant)
    t = np.arange(N)
    code = tga.code_resampled(tga.GPS, prn, 16368.0, 16368).astype(np.float64)
    x = np.stack([0.5 * code[(t - tau) % 16368] * np.cos(2 * np.pi * ((IF + dop) / FS * t % 1.0) + th)
                  for th in rng.uniform(0, 6.28, n_ant)])
    return np.packbits(x + rng.standard_normal((n_ant, N)) >= 0, axis=1)


@pytest.mark.parametrize("n_ant,half_width", [(1, -1.0), (2, 300.0), (7, 1200.0), (24, 600.0), (26, 1300.0)])
def test_scan_tiles(n_ant, half_width):
    prn, tau, dop = 9, 4321, 1700.0
    bits = _rows(n_ant, prn, tau, dop)
    df = 0.25 * FS / N  # the scan's step
    off = 0.0 if half_width < 0 else -0.8 * half_width
    task = (tga.GPS, prn, float(tau), IF + dop + off, 0, N)
    with tga.Context(0) as ctx:
        res, _ = ctx.fine_acquire(bits, FS, [task, task], scan_half_width_hz=half_width)
        p, _, _ = ctx.fine_eval(bits, FS, *task)
    for r in res:
        assert abs(r["power_start"] - p) <= 1e-6 * p
        assert abs(r["frequency"] - (IF + dop)) < df / 2
