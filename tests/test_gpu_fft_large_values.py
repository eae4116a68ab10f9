"""Records whose squares pass the largest float within a prefix block: the windows' statistics from the
prefix sums are then not trusted, and the windows are decided by the exact re-scoring, on the FFT
branch as on the tiles. Answers equal the oracle's."""
import numpy as np
import pytest

import tremor_b200 as tb
from tests.test_gpu_batching import _check

pytestmark = pytest.mark.gpu


def _record(kind, n, rng):
    from tremor_b200 import synth
    x = synth.ar2_waveform(n, rng)
    x /= x.std()
    if kind == 'scaled':
        return (x * np.float32(1e17)).astype(np.float32)  # 65536 squares of 1e34
    x[n // 2] = 3e19  # one square of 9e38, and windows of variance below 1e36 around it
    return x


@pytest.mark.parametrize('tiles', [tb.TILES_FFT, tb.TILES_ROWS])
@pytest.mark.parametrize('kind', ['scaled', 'spike'])
@pytest.mark.parametrize('lengths', [[300, 300, 1001], [2049, 2500, 2500], [9000]])
def test_squares_beyond_the_largest_float(kind, lengths, tiles):
    rng = np.random.default_rng(sum(lengths))
    x = _record(kind, 140_000, rng)
    reqs = []
    for i, m in enumerate(lengths):
        p = len(x) // 2 - m // 3 - 7 * i if i % 2 == 0 else 68_000  # over the spike; elsewhere in its block
        t = x[p:p + m].astype(np.float64)
        t = (t + 0.2 * t.std() * rng.normal(size=m)).astype(np.float32)
        reqs.append(tb.Request(t, tb.MODE_THRESHOLD, correlation=0.6))
        reqs.append(tb.Request(t, tb.MODE_KNN, k=6, merge_offset=m // 2))
        reqs.append(tb.Request(t, tb.MODE_KNN, k=3, merge_offset=0))
    with tb.Context(x) as ctx:
        ctx.set_tiles(tiles)
        answers = ctx.scan_batch(reqs)
    _check(x, reqs, answers)
