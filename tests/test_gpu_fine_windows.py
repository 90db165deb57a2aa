"""Fine acquisition of several windows in one call: scans of different widths
(their points lie one after another), windows of different lengths and starts,
each against the same task alone.  Both sum the same products in FP32; only the
order of the f64 sums over blocks may differ (about 160 of them: 2e-14), which
Newton's last step, converging quadratically, passes on."""
import numpy as np
import pytest

import tga

pytestmark = pytest.mark.gpu
FS, IF = 16.368e6, 4.092e6
N = 163680


@pytest.mark.parametrize("n_ant", [1, 3, 25])
def test_windows_of_one_call(n_ant):
    rng = np.random.default_rng(n_ant)
    t = np.arange(N)
    sats = [(9, 4321, 1700.0), (17, 777, -2300.0), (30, 15000, 400.0)]
    x = rng.standard_normal((n_ant, N))
    for prn, tau, dop in sats:
        code = tga.code_resampled(tga.GPS, prn, 16368.0, 16368).astype(np.float64)
        ph = 2 * np.pi * ((IF + dop) / FS * t % 1.0)
        x += 0.4 * code[(t - tau) % 16368] * np.cos(ph + rng.uniform(0, 6.28, (n_ant, 1)))
    bits = np.packbits(x >= 0, axis=1)
    tasks = []
    for (prn, tau, dop), (start, length) in zip(sats, [(0, 163680), (16368, 32736 + 7), (40000, 65472)]):
        tasks.append((tga.GPS, prn, float(tau) + 0.3, IF + dop + 20.0, start, length))
    tasks += [tasks[1], tasks[0]]
    with tga.Context(0) as ctx:
        every, phases = ctx.fine_acquire(bits, FS, tasks)
        for i, task in enumerate(tasks):
            (one,), ph = ctx.fine_acquire(bits, FS, [task])
            r = every[i]
            assert abs(r["power_start"] - one["power_start"]) <= 1e-12 * one["power_start"]
            assert abs(r["power"] - one["power"]) <= 1e-9 * one["power"]
            assert abs(r["code_phase"] - one["code_phase"]) <= 1e-6
            assert abs(r["frequency"] - one["frequency"]) <= 1e-4
            assert np.max(np.abs(np.exp(1j * phases[i]) - np.exp(1j * ph[0]))) <= 1e-6
