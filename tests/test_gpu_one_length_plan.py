"""A full tile's worth of templates of one length under the automatic plan: the FFT branch
(window statistics from prefix sums) where its modelled time is the smaller, with the same
answers, bit for bit, as the row tiles (per-length statistics) and the oracle, over a window
range, with missing, constant, loud and quiet stretches and with an offset."""
import numpy as np
import pytest

import tremor_b200 as tb
from tests.test_gpu_batching import _check, _requests, _waveform

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('m,offset,window_range', [(1500, 0.0, None), (2049, 5000.0, None), (4100, 0.0, (7001, 60000)),
                                                   (9000, 0.0, None)])
def test_one_length_auto_equals_row_tiles(m, offset, window_range):
    x = _waveform(1 << 17, m, offset)
    reqs = _requests(x, np.random.default_rng(m + 1), [m] * 130)
    with tb.Context(x) as ctx:
        if window_range:
            ctx.set_window_range(*window_range)
        ctx.profile_enable(True)
        auto = ctx.scan_batch(reqs)
        assert ctx.profile_read()[0] == 'fft'
        ctx.set_tiles(tb.TILES_ROWS)
        rows = ctx.scan_batch(reqs)
        assert ctx.profile_read()[0] == 'k_scan_umma'
    for (p0, d0), (p1, d1) in zip(auto, rows):
        assert np.array_equal(p0, p1) and np.array_equal(d0.view(np.uint32), d1.view(np.uint32))
    if not window_range:
        _check(x, reqs[:4], auto[:4])


def test_short_templates_of_one_length_keep_row_tiles():
    """At 256 samples a full row tile is cheaper than the transforms."""
    x = _waveform(1 << 16, 5)
    reqs = _requests(x, np.random.default_rng(6), [256] * 130)
    with tb.Context(x) as ctx:
        ctx.profile_enable(True)
        answers = ctx.scan_batch(reqs)
        assert ctx.profile_read()[0] == 'k_scan_umma'
    _check(x, reqs[:4], answers[:4])
