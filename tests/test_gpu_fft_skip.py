"""The FFT branch's chunks of windows that a template's cut lets it skip: answers equal the oracle's
with thresholds and with kNN bounds known from the first part of the record, over lengths at, above
and below those that the chunks' bounds are kept at, and over records whose deviation jumps, that
stand constant, miss samples, carry an offset or cross a prefix block."""
import numpy as np
import pytest

import tremor_b200 as tb
from tests import oracle_bindings as ob

pytestmark = pytest.mark.gpu


def _record(kind, n, rng):
    from tremor_b200 import synth
    x = synth.ar2_waveform(n, rng)
    if kind == 'jumps':
        x *= np.repeat(rng.choice([1e-3, 1.0, 50.0], n // 700 + 1), 700)[:n].astype(np.float32)
    elif kind == 'constant':
        for p in rng.integers(0, n - 3000, 12):
            x[p:p + rng.integers(100, 3000)] = x[p]
        x[rng.integers(0, n, 40)] = tb.MISSING_VALUE
    elif kind == 'offset':
        x += np.float32(3000.0)
    return x


def _check(x, reqs, answers):
    for r, (pos, dist) in zip(reqs, answers):
        m, t = len(r.template), r.template[None, :]
        if r.mode == tb.MODE_KNN:
            I, D = ob.scan_knn(x, t, m, r.k, r.merge_offset)
            p, d = I[0], D[0]
        else:
            _, p, d = ob.scan_threshold(x, t, m, r.correlation, r.merge_offset)
        assert np.array_equal(pos, p), (m, r.mode, r.k, r.merge_offset)
        assert np.array_equal(dist.view(np.uint32), d.view(np.uint32)), (m, r.mode)


@pytest.mark.parametrize('kind', ['plain', 'jumps', 'constant', 'offset'])
@pytest.mark.parametrize('lengths', [[300, 301, 329, 330, 331, 400, 400, 440, 441] * 2 + [3, 16, 17, 21],
                                     [2049, 2049, 1500, 1254, 1255] * 4, [4097, 4000, 3700, 2050] * 4,
                                     [8192, 8000, 4098] * 3 + [8193, 9000, 16384] * 3])
def test_thresholds(kind, lengths):
    """Enough pieces and templates of each class for windows to be skipped."""
    rng = np.random.default_rng(sum(lengths))
    x = _record(kind, 170_000, rng)
    reqs = []
    for i, m in enumerate(lengths):
        p = int(rng.integers(0, len(x) - m))
        t = np.where(x[p:p + m] == tb.MISSING_VALUE, 0, x[p:p + m]) + rng.normal(size=m) * x[p:p + m].std() * 0.3
        reqs.append(tb.Request(t.astype(np.float32), tb.MODE_THRESHOLD, correlation=(0.9, 0.6, 0.3)[i % 3]))
    with tb.Context(x) as ctx:
        ctx.set_tiles(tb.TILES_FFT)
        answers = ctx.scan_batch(reqs)
        ctx.set_tiles(tb.TILES_ROWS)
        rows = ctx.scan_batch(reqs)
    for i, ((p, d), (pr, dr)) in enumerate(zip(answers, rows)):
        assert np.array_equal(p, pr) and np.array_equal(d.view(np.uint32), dr.view(np.uint32)), i
    _check(x, reqs[-4:], answers[-4:])


@pytest.mark.parametrize('kind', ['plain', 'jumps', 'constant', 'offset'])
def test_bounds_from_the_first_pieces(kind):
    """Enough pieces and templates for three launches; the best windows at the end of the record, and a
    template with too few windows apart for a bound."""
    rng = np.random.default_rng(5)
    n = 2_000_000
    x = _record(kind, n, rng)
    reqs = []
    for i in range(48):
        m = 300 + 9 * (i // 2)
        t = x[n - 5000 - m:n - 5000] if i % 4 == 0 else rng.normal(size=m)
        t = np.where(t == tb.MISSING_VALUE, 0, t).astype(np.float32)
        if i % 5 == 4:
            reqs.append(tb.Request(t, tb.MODE_THRESHOLD, correlation=0.5))
        else:
            reqs.append(tb.Request(t, tb.MODE_KNN, k=(1, 7, 40)[i % 3], merge_offset=(0, 150, 2000, 400_000)[i % 4]))
    with tb.Context(x) as ctx:
        ctx.set_tiles(tb.TILES_FFT)
        answers = ctx.scan_batch(reqs)
        ctx.set_tiles(tb.TILES_ROWS)
        rows = ctx.scan_batch(reqs)
    for i, ((p, d), (pr, dr)) in enumerate(zip(answers, rows)):
        assert np.array_equal(p, pr) and np.array_equal(d.view(np.uint32), dr.view(np.uint32)), i
    _check(x, reqs[:4], answers[:4])


def test_contexts_give_the_bounds_back():
    """Twelve contexts, each with the bounds of some 40 lengths (10 MB of them), leave no more memory
    taken than one of them does."""
    import torch
    rng = np.random.default_rng(9)
    x = _record('plain', 1 << 21, rng)
    reqs = [tb.Request(rng.normal(size=int(64 * 1.1 ** i)).astype(np.float32), tb.MODE_THRESHOLD, correlation=0.9)
            for i in range(40)]
    free = []
    for _ in range(12):
        with tb.Context(x) as ctx:
            ctx.set_tiles(tb.TILES_FFT)
            ctx.scan_batch(reqs)
        free.append(torch.cuda.mem_get_info()[0])
    assert free[0] - free[-1] < 10 * (1 << 20)
