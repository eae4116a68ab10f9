"""A loud stretch takes the prefix sums' accuracy from the rest of its block of 65536 samples. The FFT
branch then has the statistics of a group's one length, and does not re-score every window after
the stretch for every template; answers equal the row tiles' and the oracle's."""
import numpy as np
import pytest

import tremor_b200 as tb
from tests.test_gpu_batching import _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('mode', ['knn', 'threshold', 'both'])
@pytest.mark.parametrize('m,templates', [(1500, 130), (300, 40), (4096, 30), (9000, 12)])
def test_windows_after_a_loud_stretch(m, templates, mode):
    from tremor_b200 import synth
    rng = np.random.default_rng(m)
    x = synth.ar2_waveform(1 << 18, rng)
    x[66_000:66_400] *= np.float32(1e5)
    x[90_000:93_000] = x[90_000]
    reqs = []
    for i in range(templates):
        p = int(rng.integers(0, len(x) - m))
        t = (x[p:p + m] + 0.3 * x[p:p + m].std() * rng.normal(size=m)).astype(np.float32)
        if mode == 'knn' or mode == 'both' and i % 2:
            reqs.append(tb.Request(t, tb.MODE_KNN, k=1 + i % 5, merge_offset=(0, m // 2)[i % 2]))
        else:
            reqs.append(tb.Request(t, tb.MODE_THRESHOLD, correlation=0.6))
    with tb.Context(x) as ctx:
        ctx.set_tiles(tb.TILES_ROWS)
        ctx.set_kernel(tb.KERNEL_FP32)  # statistics of the length whatever the number of templates
        want, few = ctx.scan_batch(reqs), ctx.last_candidates()
    with tb.Context(x) as ctx:
        ctx.set_tiles(tb.TILES_FFT)
        for _ in range(2):
            got = ctx.scan_batch(reqs)
            # some 60000 windows per template otherwise
            assert ctx.last_candidates() < 2 * few + 1000 * templates
            for i, ((p0, d0), (p1, d1)) in enumerate(zip(got, want)):
                assert np.array_equal(p0, p1) and np.array_equal(d0.view(np.uint32), d1.view(np.uint32)), i
    _check(x, reqs[:3], got[:3])
