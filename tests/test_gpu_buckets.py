"""The kNN bound's buckets: window counts and merge offsets around the 256-window bucket (and the
super-buckets of several), more answers than buckets, and the larger buckets that big groups
get; answers equal the oracle's, or those of the same requests in small groups."""
import numpy as np
import pytest

import tremor_b200 as tb
from tests import oracle_bindings as ob

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('kernel,tiles', [(tb.KERNEL_AUTO, tb.TILES_FFT), (tb.KERNEL_SPLIT_BF16, tb.TILES_ROWS),
                                          (tb.KERNEL_AUTO, tb.TILES_COLS_32), (tb.KERNEL_FP32, tb.TILES_AUTO)])
@pytest.mark.parametrize('windows', [1, 255, 256, 257, 1023, 1025, 7169, 12289])
def test_bucket_edges(kernel, tiles, windows):
    rng = np.random.default_rng(windows)
    m = 40
    x = rng.normal(size=windows + m - 1).astype(np.float32)
    x = np.cumsum(x).astype(np.float32)
    q = rng.normal(size=(3, m)).astype(np.float32)
    with tb.Context(x) as ctx:
        ctx.set_kernel(kernel)
        ctx.set_tiles(tiles)
        for k, merge in [(1, 0), (3, 0), (2, 255), (3, 256), (2, 257), (4, 600), (40, 20), (9, 0)]:
            I, D = ctx.search_knn(q, k, merge)
            Io, Do = ob.scan_knn(x, q, m, k, merge)
            assert np.array_equal(I, Io) and np.array_equal(D.view(np.uint32), Do.view(np.uint32)), (k, merge)


@pytest.mark.parametrize('log_n,count', [(24, 4300), (25, 8300)])
def test_larger_buckets_of_big_groups(log_n, count):
    """Groups whose minima in 256-window buckets would exceed 2 GiB (buckets of 512 and 2048 windows
    here) answer as the same requests in a group of 60."""
    rng = np.random.default_rng(log_n)
    n, m = 1 << log_n, 48
    x = rng.normal(size=n).astype(np.float32)
    x[1000:1200] = 0.5
    q = rng.normal(size=(count, m)).astype(np.float32)
    reqs = [tb.Request(t, tb.MODE_KNN, k=1 + i % 3, merge_offset=(0, 100, 700, 3000)[i % 4]) for i, t in enumerate(q)]
    pick = list(range(0, count, count // 59))[:60]
    with tb.Context(x) as ctx:
        big = ctx.scan_batch(reqs)
        small = ctx.scan_batch([reqs[i] for i in pick])
    for i, (p, d) in zip(pick, small):
        assert np.array_equal(p, big[i][0]) and np.array_equal(d.view(np.uint32), big[i][1].view(np.uint32)), i
