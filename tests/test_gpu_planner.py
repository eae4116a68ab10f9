"""The planner's choice between the FFT branch and the tiles where the branch would skip no windows: in a
small window range of a long record, and for thresholds that noise reaches."""
import numpy as np
import pytest

import tremor_b200 as tb

pytestmark = pytest.mark.gpu


def _kernel(ctx, reqs):
    ctx.profile_enable(True)
    ctx.profile_read()
    answers = ctx.scan_batch(reqs)
    return ctx.profile_read()[0], answers


def _same(got, want):
    for i, ((p0, d0), (p1, d1)) in enumerate(zip(got, want)):
        assert np.array_equal(p0, p1) and np.array_equal(d0.view(np.uint32), d1.view(np.uint32)), i


def test_window_range():
    """128 kNN templates of 1024: bounds from the first pieces of 2^22 samples pay, of 60000 they do not."""
    rng = np.random.default_rng(1)
    x = rng.normal(size=1 << 22).astype(np.float32)
    reqs = [tb.Request(rng.normal(size=1024).astype(np.float32), tb.MODE_KNN, k=3, merge_offset=500) for _ in range(128)]
    with tb.Context(x) as ctx:
        assert _kernel(ctx, reqs)[0] == 'fft'
        ctx.set_window_range(1_000_001, 60_000)
        name, got = _kernel(ctx, reqs)
        assert name == 'k_scan_umma'
        ctx.set_tiles(tb.TILES_FFT)
        _same(got, ctx.scan_batch(reqs))


def test_thresholds_that_noise_reaches():
    """128 templates of 1024: at 0.8 almost every window is skipped, at 0.1 few."""
    rng = np.random.default_rng(2)
    x = rng.normal(size=1 << 21).astype(np.float32)
    q = rng.normal(size=(128, 1024)).astype(np.float32)
    with tb.Context(x) as ctx:
        for correlation, kernel in ((0.8, 'fft'), (0.1, 'k_scan_umma')):
            reqs = [tb.Request(t, tb.MODE_THRESHOLD, correlation=correlation) for t in q]
            ctx.set_tiles(tb.TILES_AUTO)
            name, got = _kernel(ctx, reqs)
            assert name == kernel
            ctx.set_tiles(tb.TILES_FFT)
            _same(got, ctx.scan_batch(reqs))
