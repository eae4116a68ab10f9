"""A batch prepared in one window range and run in another has the answers of a batch of that range."""
import numpy as np
import pytest

import tremor_b200 as tb

pytestmark = pytest.mark.gpu

FULL = (0, 1 << 40)


def _batch_of(kind, rng):
    """The requests and the tiles: several lengths on each branch, and a full tile of one length under the
    automatic plan."""
    lengths = [2100] * 128 if kind == 'one length' else [60, 300, 300, 1100, 2049, 5000, 9000]
    reqs = [tb.Request(rng.normal(size=m).astype(np.float32), tb.MODE_KNN, k=3, merge_offset=m // 2) if i % 2 else
            tb.Request(rng.normal(size=m).astype(np.float32), tb.MODE_THRESHOLD, correlation=3.0 / m ** 0.5)
            for i, m in enumerate(lengths)]
    return reqs, {'rows': tb.TILES_ROWS, 'columns': tb.TILES_COLS_64, 'fft': tb.TILES_FFT, 'one length': tb.TILES_AUTO}[kind]


def _run(kind, ranges):
    rng = np.random.default_rng(len(kind))
    x = rng.normal(size=150_000).astype(np.float32)
    reqs, tiles = _batch_of(kind, rng)
    with tb.Context(x) as ctx:
        ctx.set_tiles(tiles)
        ctx.set_window_range(*ranges[0])
        batch = ctx.batch(reqs)
        for r in ranges:
            ctx.set_window_range(*r)
            for i, ((p, d), (q, e)) in enumerate(zip(batch.run(), ctx.scan_batch(reqs))):
                assert np.array_equal(p, q) and np.array_equal(d.view(np.uint32), e.view(np.uint32)), (r, i)


@pytest.mark.parametrize('kind', ['rows', 'columns', 'fft', 'one length'])
def test_range_widened(kind):
    _run(kind, [(0, 5000), (0, 60_000), FULL])


@pytest.mark.parametrize('kind', ['rows', 'columns', 'fft', 'one length'])
def test_range_moved(kind):
    """To the record's end, where the longest templates have no windows, and past it."""
    _run(kind, [FULL, (70_000, 30_000), (145_500, 1 << 40), (149_990, 5), (200_000, 5), (1, 1 << 40)])
