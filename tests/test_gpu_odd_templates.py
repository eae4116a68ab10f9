"""A template with a value that is not finite has no answers but constant windows, and leaves the answers
of the others of its length and batch as they are: all equal the oracle's."""
import numpy as np
import pytest

import tremor_b200 as tb
from tests.test_gpu_batching import _check, _waveform

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('tiles', [tb.TILES_AUTO, tb.TILES_ROWS, tb.TILES_COLS_32, tb.TILES_FFT])
@pytest.mark.parametrize('where', [0, 3])
@pytest.mark.parametrize('m', [300, 4000, 9000])
def test_one_among_its_length(m, where, tiles):
    x = _waveform(90_000, 4)
    rng = np.random.default_rng(m)
    reqs = []
    for i in range(5):
        t = x[65_000 + 1000 * i:65_000 + 1000 * i + m].copy()
        t = (np.where(t == tb.MISSING_VALUE, 0, t) + 0.1 * t.std() * rng.normal(size=m)).astype(np.float32)
        if i == where:
            t[m // 3] = np.nan if m != 4000 else np.inf
        reqs.append(tb.Request(t, tb.MODE_KNN, k=4, merge_offset=m // 2) if i % 2 else
                    tb.Request(t, tb.MODE_THRESHOLD, correlation=0.5))
    reqs.append(tb.Request(x[70_000:70_077], tb.MODE_KNN, k=2, merge_offset=10))
    with tb.Context(x) as ctx:
        ctx.set_tiles(tiles)
        answers = ctx.scan_batch(reqs)
        some = range(len(reqs)) if m < 9000 else [where, 1, 5]
        _check(x, [reqs[i] for i in some], [answers[i] for i in some])
        _check(x, reqs[where:where + 1], ctx.scan_batch(reqs[where:where + 1]))
