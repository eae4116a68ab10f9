"""Re-scoring of many and of few candidates: short templates and candidates whose rounded statistics the
prefix sums do not decide (on a record that drifts far within a prefix block about half of them), by a
thread each where there are many. Distances equal the oracle's bit for bit."""
import numpy as np
import pytest

import tremor_b200 as tb
from tests.test_gpu_batching import _check

pytestmark = pytest.mark.gpu


def _record(n, slope, rng):
    from tremor_b200 import synth
    x = synth.ar2_waveform(n, rng) + slope * np.arange(n)
    x[n // 3] += 1e5  # a spike, a step and missing samples: some are decided by the chains alone
    x[n // 2:] += 3e3
    x = x.astype(np.float32)
    x[rng.integers(0, n, 30)] = tb.MISSING_VALUE
    return x


@pytest.mark.parametrize('slope', [0.0, 0.05])
@pytest.mark.parametrize('m,templates,correlation', [(33, 1, 0.9), (192, 2, 0.1), (193, 2, 0.1), (400, 1, 0.9995), (400, 6, 0.7),
                                                     (1000, 3, 0.9), (1025, 2, 0.6), (16000, 1, 0.9)])
def test_thresholds_and_few_answers(m, templates, correlation, slope):
    rng = np.random.default_rng(m + templates)
    x = _record(150_000, slope, rng)
    reqs = []
    for i in range(templates):
        p = (20_000 + 9_000 * i, 50_000 - m // 2)[i % 2]
        t = x[p:p + m] + (0.2 * x[p:p + m].std() * rng.normal(size=m)).astype(np.float32)
        reqs += [tb.Request(t, tb.MODE_THRESHOLD, correlation=correlation), tb.Request(t, tb.MODE_KNN, k=1 + 30 * i, merge_offset=i)]
    with tb.Context(x) as ctx:
        ctx.set_tiles(tb.TILES_FFT)
        answers = ctx.scan_batch(reqs)
    _check(x, reqs, answers)


@pytest.mark.parametrize('slope', [0.0, 0.05])
@pytest.mark.parametrize('lengths', [[60, 100], [100, 300, 1500]])
@pytest.mark.parametrize('tiles', [tb.TILES_FFT, tb.TILES_COLS_32])
def test_every_window_a_candidate(tiles, lengths, slope):
    """kNN requests without a bound (too few windows apart) or with one over a thousand buckets, and
    thresholds that every window passes, short and long templates in one group."""
    rng = np.random.default_rng(len(lengths))
    x = _record(120_000, slope, rng)
    reqs = []
    for m in lengths:
        t = (x[30_000:30_000 + m] + 0.5 * x[30_000:30_000 + m].std() * rng.normal(size=m)).astype(np.float32)
        reqs += [tb.Request(t, tb.MODE_KNN, k=3, merge_offset=70_000), tb.Request(t, tb.MODE_KNN, k=1500, merge_offset=0),
                 tb.Request(t, tb.MODE_KNN, k=400, merge_offset=100), tb.Request(t, tb.MODE_THRESHOLD, correlation=-1.0)]
    with tb.Context(x) as ctx:
        ctx.set_tiles(tiles)
        answers = ctx.scan_batch(reqs)
    _check(x, reqs, answers)


def test_undecided_candidates_cost_no_more():
    """Every window of 2^20 a candidate of eight templates of 100: re-scored in the same time whether or not
    the prefix sums decide (three times as long with the chains of 16 candidates to a warp)."""
    from tremor_b200 import synth
    rng = np.random.default_rng(5)
    n = 1 << 20
    x = synth.ar2_waveform(n, rng)
    t = rng.normal(size=(8, 100)).astype(np.float32)
    reqs = [tb.Request(v, tb.MODE_THRESHOLD, correlation=-1.0) for v in t]
    ms = []
    for record in (x, (x + 0.05 * np.arange(n)).astype(np.float32)):
        with tb.Context(record) as ctx:
            ctx.set_tiles(tb.TILES_FFT)
            batch = ctx.batch(reqs)
            batch.run()
            ctx.profile_enable(True)
            best = []
            for _ in range(5):
                ctx.profile_phases()
                batch.run()
                best.append(ctx.profile_phases()['rescore'])
            ms.append(min(best))
    assert ms[1] < 1.6 * ms[0], ms
