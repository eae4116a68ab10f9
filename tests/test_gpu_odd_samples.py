"""Samples that are not finite: a window with one has the distance NaN in the reference, so it is in no
answer, and the windows around it are found as ever, through every contraction: a single one, some
of each kind, a stretch, one within a constant stretch and one within the best match, over which a
bound must not be taken. Answers equal the oracle's."""
import numpy as np
import pytest

import tremor_b200 as tb
from tests.test_gpu_batching import TILES, _check

pytestmark = pytest.mark.gpu


def _record(kind, n, rng):
    from tremor_b200 import synth
    x = synth.ar2_waveform(n, rng)
    x[9000:9900] = 0.0
    if kind == 'one':
        x[n // 2 + 5] = np.nan
    elif kind == 'some':
        x[rng.integers(0, n, 9)] = np.nan
        x[rng.integers(0, n, 9)] = np.inf
        x[rng.integers(0, n, 9)] = -np.inf
        x[[0, 9400, n - 1]] = np.nan
    else:
        x[40_000:40_700] = np.nan
        x[50_000:52_000:200] = np.inf  # too close for windows of the longer templates
    return x


def _requests(x, rng, lengths):
    reqs, odd = [], np.flatnonzero(~np.isfinite(x))
    for i, m in enumerate(lengths):
        p = min(max(0, int(odd[i % len(odd)]) - m // 2), len(x) - m) if i % 2 else int(rng.integers(20_000, len(x) - m))
        t = np.nan_to_num(x[p:p + m], nan=0.0, posinf=0.0, neginf=0.0)
        t = t + 0.1 * (t.std() + 0.1) * rng.normal(size=m)
        reqs += [tb.Request(t, tb.MODE_KNN, k=(1, 7, 30)[i % 3], merge_offset=(0, m // 2)[i % 2]),
                 tb.Request(t, tb.MODE_THRESHOLD, correlation=0.5)]
    return reqs


@pytest.mark.parametrize('tiles', TILES)
@pytest.mark.parametrize('kind', ['one', 'some', 'stretch'])
def test_several_lengths(kind, tiles):
    rng = np.random.default_rng(len(kind))
    x = _record(kind, 100_000, rng)
    reqs = _requests(x, rng, [40, 128, 190, 333, 1000, 2500])
    with tb.Context(x) as ctx:
        ctx.set_tiles(tiles)
        answers = ctx.scan_batch(reqs)
    _check(x, reqs, answers)


@pytest.mark.parametrize('tiles,kernel', [(tb.TILES_ROWS, tb.KERNEL_AUTO), (tb.TILES_COLS_32, tb.KERNEL_AUTO),
                                          (tb.TILES_AUTO, tb.KERNEL_FP32)])
@pytest.mark.parametrize('kind', ['one', 'some', 'stretch'])
def test_one_length(kind, tiles, kernel):
    """Statistics per length; the whole record's windows asked for, the constant ones among them."""
    rng = np.random.default_rng(len(kind))
    x = _record(kind, 100_000, rng)
    reqs = _requests(x, rng, [200] * 64) + [tb.Request(x[20_000:20_200], tb.MODE_KNN, k=600, merge_offset=150)]
    with tb.Context(x) as ctx:
        ctx.set_kernel(kernel)
        ctx.set_tiles(tiles)
        answers = ctx.scan_batch(reqs)
    some = list(range(8)) + [len(reqs) - 1]
    _check(x, [reqs[i] for i in some], [answers[i] for i in some])


def test_bounds_from_the_first_pieces():
    """Bounds and cuts along the way: the best match has a NaN within, and begins in the first pieces."""
    rng = np.random.default_rng(3)
    from tremor_b200 import synth
    n = 2_000_000
    x = synth.ar2_waveform(n, rng)
    reqs = []
    for i in range(40):
        m = 300 + 7 * i
        p = 2000 + 1500 * i
        t = x[p:p + m].copy()
        q = n - 3000 - 1500 * i  # the second best, found last
        x[q:q + m] += 1.5 * t
        x[p + m // 2] = np.nan
        reqs.append(tb.Request(t, tb.MODE_KNN, k=1 + i % 3, merge_offset=(0, 100)[i % 2]))
    with tb.Context(x) as ctx:
        ctx.set_tiles(tb.TILES_FFT)
        answers = ctx.scan_batch(reqs)
        ctx.set_tiles(tb.TILES_ROWS)
        rows = ctx.scan_batch(reqs)
    for i, ((p, d), (pr, dr)) in enumerate(zip(answers, rows)):
        assert np.array_equal(p, pr) and np.array_equal(d.view(np.uint32), dr.view(np.uint32)), i
    _check(x, reqs[:6], answers[:6])


@pytest.mark.parametrize('scale', [1e30, 1e36])
def test_dot_products_beyond_the_largest_float(scale):
    rng = np.random.default_rng(8)
    from tremor_b200 import synth
    x = synth.ar2_waveform(30_000, rng)
    x = (x * (scale / np.abs(x).max())).astype(np.float32)
    reqs = [tb.Request((x[p:p + m] / scale + 0.02 * rng.normal(size=m)).astype(np.float32), tb.MODE_THRESHOLD, correlation=0.5)
            for p, m in ((9000, 300), (100, 2500), (17_000, 9000))]
    with tb.Context(x) as ctx:
        ctx.set_tiles(tb.TILES_FFT)
        answers = ctx.scan_batch(reqs)
    _check(x, reqs, answers)
