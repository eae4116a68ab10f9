"""Paths of the kNN selection that need many buckets, many pieces or the longest templates: a bucket list
that has to be made again, bounds from the first pieces of a window range, and windows skipped by
templates cut in two parts. Answers equal the oracle's, and the row tiles' bit for bit."""
import numpy as np
import pytest

import tremor_b200 as tb
from tests import oracle_bindings as ob
from tests.test_gpu_batching import _check

pytestmark = pytest.mark.gpu


def _same(got, want):
    for i, ((p0, d0), (p1, d1)) in enumerate(zip(got, want)):
        assert np.array_equal(p0, p1) and np.array_equal(d0.view(np.uint32), d1.view(np.uint32)), i


@pytest.mark.parametrize('tiles', [tb.TILES_ROWS, tb.TILES_FFT])
def test_bucket_list_made_again(tiles):
    """A record of period 256: every bucket of every template holds a best match, 36 x 32769 of them, more
    than the 2^20 that the list first has room for."""
    rng = np.random.default_rng(3)
    n, m = (1 << 23) + 300, 64
    period = rng.normal(size=256).astype(np.float32)
    x = np.tile(period, n // 256 + 2)[:n]
    reqs = []
    for i in range(40):
        t = (x[7 * i:7 * i + m] + 0.2 * rng.normal(size=m)).astype(np.float32)
        if i % 10 == 9:
            reqs.append(tb.Request(t, tb.MODE_THRESHOLD, correlation=0.95, merge_offset=5000))
        else:
            reqs.append(tb.Request(t, tb.MODE_KNN, k=1 + i % 7, merge_offset=(0, 100, 700)[i % 3]))
    with tb.Context(x) as ctx:
        ctx.set_tiles(tiles)
        ctx.scan_batch(reqs[:2])  # what the record and the length need once
        ctx.profile_read()
        first = ctx.scan_batch(reqs)
        launches = ctx.profile_read()[4]
        _same(ctx.scan_batch(reqs), first)
        assert launches > ctx.profile_read()[4]  # the list and the re-pass a second time
    some = [0, 1, 2, 9, 38, 39]
    _check(x, [reqs[i] for i in some], [first[i] for i in some])


def _check_range(x, first, count, reqs, answers):
    for r, (pos, dist) in zip(reqs, answers):
        m = len(r.template)
        I, D = ob.scan_knn(x[first:first + count + m - 1], r.template[None, :], m, r.k, r.merge_offset)
        assert np.array_equal(pos, I[0] + np.uint64(first)), (m, r.k, r.merge_offset)
        assert np.array_equal(dist.view(np.uint32), D[0].view(np.uint32)), (m, r.k)


@pytest.mark.parametrize('first,count', [(100_003, 1_700_000), (1, 1_900_000), (500_000, 1_111_111)])
def test_bounds_from_the_first_pieces_of_a_range(first, count):
    """Three launches over the range's pieces; matches just before it, at its ends and in its middle."""
    from tremor_b200 import synth
    rng = np.random.default_rng(first)
    x = synth.ar2_waveform(2_000_000, rng)
    reqs = []
    for i in range(60):
        m = 300 + 13 * (i // 2)
        p = (max(first - 1, 0), first, first + count // 2, first + count - 1, first + count - m)[i % 5]
        t = (x[p:p + m] + 0.05 * rng.normal(size=m)).astype(np.float32)
        reqs.append(tb.Request(t, tb.MODE_KNN, k=(1, 7, 30)[i % 3], merge_offset=(0, 150, 2000)[i % 3]))
    with tb.Context(x) as ctx:
        ctx.set_window_range(first, count)
        ctx.set_tiles(tb.TILES_FFT)
        answers = ctx.scan_batch(reqs)
        ctx.set_tiles(tb.TILES_ROWS)
        _same(answers, ctx.scan_batch(reqs))
    _check_range(x, first, count, reqs[:6], answers[:6])


@pytest.mark.parametrize('mode', ['knn', 'threshold'])
def test_two_parts_skip_windows(mode):
    """16 templates of 8194 to 16384 samples on 2^20: 128 pieces, so that thresholds skip windows throughout and
    kNN templates past the first pieces."""
    from tremor_b200 import synth
    rng = np.random.default_rng(7)
    x = synth.ar2_waveform(1 << 20, rng)
    x[300_000:310_000] *= np.float32(40)
    reqs = []
    for i, m in enumerate([8194, 9000, 9900, 12_000, 12_000, 16_000, 16_383, 16_384] * 2):
        p = (len(x) - m, 290_000 + 1000 * i, 5000 * i)[i % 3]
        t = (x[p:p + m] + 0.3 * x[p:p + m].std() * rng.normal(size=m)).astype(np.float32)
        reqs.append(tb.Request(t, tb.MODE_KNN, k=1 + i % 4, merge_offset=(0, m // 2)[i % 2]) if mode == 'knn' else
                    tb.Request(t, tb.MODE_THRESHOLD, correlation=(0.05, 0.5, 0.9)[i % 3]))
    with tb.Context(x) as ctx:
        ctx.set_tiles(tb.TILES_FFT)
        answers = ctx.scan_batch(reqs)
        ctx.set_tiles(tb.TILES_ROWS)
        _same(answers, ctx.scan_batch(reqs))
    _check(x, reqs[1:2], answers[1:2])
