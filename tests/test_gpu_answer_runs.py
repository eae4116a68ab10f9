"""The sort of few answers in shared memory and of many by radix: numbers of answers around powers of
two and the limit of 4096 per template, thresholds and kNN in one batch, templates without
answers; answers equal the oracle's."""
import numpy as np
import pytest

import tremor_b200 as tb
from tests.test_gpu_batching import _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('windows', [1, 2, 3, 31, 512, 513, 4095, 4096, 4097, 9000])
def test_counts_around_the_limits(windows):
    m = 32
    rng = np.random.default_rng(windows)
    x = rng.normal(size=windows + m - 1).astype(np.float32)
    t = rng.normal(size=(5, m)).astype(np.float32)
    reqs = [tb.Request(t[0], tb.MODE_THRESHOLD, correlation=-1.0),  # every window
            tb.Request(t[1], tb.MODE_KNN, k=min(windows, 700), merge_offset=0),
            tb.Request(t[2], tb.MODE_THRESHOLD, correlation=0.999),  # none
            tb.Request(t[3], tb.MODE_KNN, k=5, merge_offset=40),
            tb.Request(t[4], tb.MODE_THRESHOLD, correlation=0.0, merge_offset=3)]
    with tb.Context(x) as ctx:
        _check(x, reqs, ctx.scan_batch(reqs))
        _check(x, reqs[1:2], ctx.scan_batch(reqs[1:2]))


def test_many_templates():
    """Too many answers for every template's block to look at all of them."""
    rng = np.random.default_rng(3)
    x = rng.normal(size=40_000).astype(np.float32)
    reqs = [tb.Request(rng.normal(size=64).astype(np.float32), tb.MODE_THRESHOLD, correlation=0.3) for _ in range(300)]
    with tb.Context(x) as ctx:
        every = ctx.scan_batch(reqs)
        some = ctx.scan_batch(reqs[:7])
    for (p, d), (q, e) in zip(some, every):
        assert np.array_equal(p, q) and np.array_equal(d.view(np.uint32), e.view(np.uint32))
    _check(x, reqs[:2], every[:2])
