"""Searches over several code lengths: a short one runs each length on a stream
of its own, a long one (and any with per-kernel timing) all on one.  The cells
must not depend on it, nor on which came before on the same context, in eager
calls, captured and replayed ones."""
import numpy as np
import pytest

import tga

pytestmark = pytest.mark.gpu
FIELDS = ("constellation", "prn", "antenna", "best_codephase", "best_freq_idx", "hypothesis", "signal_strength",
          "second_peak", "frequency", "cn0_acr", "cn0_valid")
FS = 4 * 1.023e6
MASK = (1 << tga.GPS) | (1 << tga.GALILEO) | (1 << tga.BEIDOU)


@pytest.mark.parametrize("graphs", [False, True])
@pytest.mark.parametrize("precision", [tga.PRECISION_FP32, tga.PRECISION_FP16_TC])
def test_streams_do_not_change_the_cells(precision, graphs):
    bits = np.random.default_rng(8).integers(0, 256, size=(2, int(FS * 0.021) // 8), dtype=np.uint8)
    short = dict(mask=MASK, prn_filter=list(range(1, 11)), center_freq=0.6e6, search_band=3000.0, cn0=True)
    # 2 antennas x 4001 bins x 10 PRNs x (4092 + 16368 + 40920) lags: 4.9e9, above the limits of both precisions
    long = dict(short, search_band=150.0 * 4000)

    def same(a, b):
        for f in FIELDS:
            assert np.array_equal(a[f], b[f], equal_nan=a[f].dtype.kind == "f"), f

    with tga.Context(0) as ctx:
        ctx.set_precision(precision)
        ctx.set_graphs(graphs)
        ctx.set_profiling(True)
        one = ctx.acquire_cells(bits, FS, **short)
        one_long = ctx.acquire_cells(bits, FS, **long)
        ctx.set_profiling(False)
        for _ in range(4):  # eager, captured, replayed
            same(ctx.acquire_cells(bits, FS, **short), one)
        for _ in range(3):
            same(ctx.acquire_cells(bits, FS, **long), one_long)
            same(ctx.acquire_cells(bits, FS, **short), one)
