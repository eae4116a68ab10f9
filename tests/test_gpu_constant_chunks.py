"""Constant stretches and the chunks' bounds of the FFT branch: windows that are constant for every length
that takes a bound have no part in it; those that a longer window leaves have. Runs around the
lengths of the templates and of the next base; answers equal the oracle's."""
import numpy as np
import pytest

import tremor_b200 as tb
from tests.test_gpu_batching import _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('base', [1, 5, 97, 300, 1102, 2400])
def test_runs_around_the_lengths(base):
    from tremor_b200 import synth
    rng = np.random.default_rng(base)
    nxt = max(base + 1, base * 11 // 10)
    lengths = sorted({base, base + 1, (base + nxt) // 2, nxt - 1, nxt, nxt + 1} - {1})
    x = synth.ar2_waveform(240_000, rng)
    at = 3000
    for run in [v + d for v in lengths for d in (-1, 0, 1)] + [20_000]:
        if run < 1 or at + run > len(x) - 6000:
            continue
        x[at:at + run] = x[at]
        at += run + int(rng.integers(50, 400))
    reqs = []
    for i, m in enumerate(lengths * 6):
        p = int(rng.integers(0, at))
        t = x[p:p + m] + (0.2 * x.std() * rng.normal(size=m)).astype(np.float32)  # over the ends of the runs
        reqs.append(tb.Request(t, tb.MODE_THRESHOLD, correlation=0.999 if m < 20 else 0.8) if i % 3 else
                    tb.Request(t, tb.MODE_KNN, k=4, merge_offset=(0, m // 2)[i % 2]))
    with tb.Context(x) as ctx:
        ctx.set_tiles(tb.TILES_FFT)
        answers = ctx.scan_batch(reqs)
    some = slice(0, 2 * len(lengths)) if base < 1000 else slice(0, len(lengths))
    _check(x, reqs[some], answers[some])


def test_constant_windows_are_skipped():
    """Half the record constant: the correlation takes no longer than on the record without (evaluating
    the constant windows of every template took 1.8 times as long)."""
    from tremor_b200 import synth
    rng = np.random.default_rng(2)
    plain = synth.ar2_waveform(1 << 22, rng)
    half = plain.copy()
    for p in range(0, len(half), 100_000):
        half[p:p + 50_000] = 0
    reqs = [tb.Request(rng.normal(size=1500).astype(np.float32), tb.MODE_THRESHOLD, correlation=0.7) for _ in range(64)]
    ms = []
    for x in (plain, half):
        with tb.Context(x) as ctx:
            ctx.set_tiles(tb.TILES_FFT)
            batch = ctx.batch(reqs)
            batch.run()
            ctx.profile_enable(True)
            best = []
            for _ in range(5):
                ctx.profile_read()
                batch.run()
                best.append(ctx.profile_read()[2])
            ms.append(min(best))
    assert ms[1] < 1.3 * ms[0], ms
