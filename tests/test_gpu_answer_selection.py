"""The kNN answers' exclusion selection over long candidate runs, and the candidates that a certain
minimum nearby excludes beforehand: smooth records, whose windows near
an event all lie close, and exactly periodic ones, full of equal distances; answer counts around
the fours, warps and blocks that the selection works in, up to its largest."""
import numpy as np
import pytest

import tremor_b200 as tb
from tests import oracle_bindings as ob

pytestmark = pytest.mark.gpu


def _smooth(rng, n):
    return np.convolve(rng.normal(size=n + 199), np.hanning(200), 'valid').astype(np.float32)


def _periodic(rng, n):
    return np.tile(rng.normal(size=500).astype(np.float32), n // 500 + 1)[:n]


@pytest.mark.parametrize('k,merge', [(1, 40), (5, 0), (4, 900), (32, 1), (33, 64), (100, 40), (257, 7), (257, 0), (1024, 20),
                                     (3, 255), (3, 256), (3, 257), (9, 513), (5, 5000), (2, 25_000), (2, 70_000)])
@pytest.mark.parametrize('record', [_smooth, _periodic])
def test_long_runs(record, k, merge):
    rng = np.random.default_rng(k + merge)
    x = record(rng, 60000)
    q = np.stack([x[900:964], x[30000:30064], rng.normal(size=64)]).astype(np.float32)
    Io, Do = ob.scan_knn(x, q, 64, k, merge)
    with tb.Context(x) as ctx:
        for kernel, tiles in [(tb.KERNEL_AUTO, tb.TILES_AUTO), (tb.KERNEL_AUTO, tb.TILES_FFT), (tb.KERNEL_FP32, tb.TILES_AUTO),
                              (tb.KERNEL_SPLIT_BF16, tb.TILES_ROWS)]:
            ctx.set_kernel(kernel)
            ctx.set_tiles(tiles)
            I, D = ctx.search_knn(q, k, merge)
            assert np.array_equal(I, Io) and np.array_equal(D.view(np.uint32), Do.view(np.uint32)), (kernel, tiles)
