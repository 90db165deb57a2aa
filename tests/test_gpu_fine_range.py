"""Fine acquisition at finite code phases far outside the code: every replica
index stays inside the chip sequence, so the call returns, and a whole number
of code periods more or less gives the same power wherever a double still
holds the samples.  (A power needs no value where it does not.)"""
import numpy as np
import pytest

import tga

pytestmark = pytest.mark.gpu
FS, IF, N = 16.368e6, 4.092e6, 16368


@pytest.mark.parametrize("const,prn,period", [(tga.GPS, 9, 16368), (tga.GALILEO, 3, 65472)])
def test_code_phase_far_away(const, prn, period):
    bits = np.random.default_rng(3).integers(0, 256, size=(2, N // 8), dtype=np.uint8)
    with tga.Context(0) as ctx:
        p0, _, _ = ctx.fine_eval(bits, FS, const, prn, 1234.0, IF, 0, N)
        for m in (1e6, -1e6):  # phases to 2e-5 samples
            p, _, _ = ctx.fine_eval(bits, FS, const, prn, 1234.0 + m * period, IF, 0, N)
            assert abs(p - p0) <= 1e-3 * p0
        for tau in (2.0 ** 40, -2.0 ** 45, 1e17, -1e19, 1e25, 1e300, -1e300):
            ctx.fine_eval(bits, FS, const, prn, tau, IF, 0, N)
            ctx.fine_acquire(bits, FS, [(const, prn, tau, IF, 0, N)])
        p1, _, _ = ctx.fine_eval(bits, FS, const, prn, 1234.0, IF, 0, N)
        assert abs(p1 - p0) <= 1e-12 * p0


@pytest.mark.parametrize("half_widths", [[2.1e6], [1.3e6, 1.3e6], [1e12], [float("inf")]])
def test_too_many_scan_points(half_widths):
    """More than 65535 points over the tasks of a call (steps of 1 / (4 T), 62.5
    Hz for 4 ms) are refused, and the context works on."""
    n = 65472
    bits = np.random.default_rng(4).integers(0, 256, size=(1, n // 8), dtype=np.uint8)
    tasks = [(tga.GPS, 9 + i, 1234.0, IF, 0, n) for i in range(len(half_widths))]
    with tga.Context(0) as ctx:
        with pytest.raises(tga.TgaError):
            ctx.fine_acquire(bits, FS, tasks, scan_half_width_hz=half_widths[0])
        res, _ = ctx.fine_acquire(bits, FS, tasks, scan_half_width_hz=600.0)
        assert all(r["power"] >= r["power_start"] > 0 for r in res)
