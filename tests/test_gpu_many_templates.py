"""More kNN templates in one group than a grid is high (65535), with merge offsets below and above a
bucket: the answers of the first, the last and some between equal the oracle's."""
import numpy as np
import pytest

import tremor_b200 as tb
from tests.test_gpu_batching import _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('tiles', [tb.TILES_ROWS, tb.TILES_COLS_128, tb.TILES_FFT])
@pytest.mark.parametrize('merge', [10, 700])
def test_more_templates_than_a_grid_is_high(tiles, merge):
    rng = np.random.default_rng(merge)
    x = rng.normal(size=3000).astype(np.float32)
    count = 65536 + 100
    reqs = [tb.Request(t, tb.MODE_KNN, k=2, merge_offset=merge) for t in rng.normal(size=(count, 20)).astype(np.float32)]
    with tb.Context(x) as ctx:
        ctx.set_tiles(tiles)
        answers = ctx.scan_batch(reqs)
    some = [0, 1, 32767, 32768, 65535, 65536, count - 1]
    _check(x, [reqs[i] for i in some], [answers[i] for i in some])
