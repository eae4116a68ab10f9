"""Searches with little device memory left: what does not fit is done in less, with the same answers."""
import numpy as np
import pytest

import tremor_b200 as tb

pytestmark = pytest.mark.gpu


class _Taken:
    """All but `left` bytes of the device's free memory."""

    def __init__(self, left):
        import torch
        torch.cuda.synchronize()
        self.hold = [torch.empty(max(0, torch.cuda.mem_get_info()[0] - left), dtype=torch.uint8, device='cuda')]

    def __enter__(self):
        return self

    def __exit__(self, *exc):
        import torch
        self.hold.clear()
        torch.cuda.empty_cache()


def _record(n):
    from tremor_b200 import synth
    rng = np.random.default_rng(n)
    return synth.ar2_waveform(n, rng), rng


def _same(got, want):
    for i, ((p0, d0), (p1, d1)) in enumerate(zip(got, want)):
        assert np.array_equal(p0, p1) and np.array_equal(d0.view(np.uint32), d1.view(np.uint32)), i


@pytest.mark.parametrize('tiles', [tb.TILES_AUTO, tb.TILES_FFT])
def test_spectra_of_fewer_classes(tiles):
    """2^24 samples: the prefix sums take 302 MB, spectra of the four classes 154, 180, 179 and 268 MB: with
    room for 0.8 of 900 MB the longest pieces serve every template."""
    x, rng = _record(1 << 24)
    reqs = [tb.Request(rng.normal(size=m).astype(np.float32), tb.MODE_KNN, k=3, merge_offset=m // 2)
            for m in (700, 1900, 3900, 8000, 12000)]
    with tb.Context(x) as ctx:
        ctx.set_tiles(tiles)
        want = ctx.scan_batch(reqs)
    with tb.Context(x) as ctx:
        ctx.set_tiles(tiles)
        ctx.profile_enable(True)
        with _Taken(900 << 20):
            got = ctx.scan_batch(reqs)
        assert ctx.profile_read()[0] == 'fft'
        _same(got, want)
        _same(ctx.scan_batch(reqs), want)  # with memory again, and one class resident


def test_chunk_bounds_stay_small():
    """The bounds of 2^22 samples' chunks, 0.5 MB for each of some ninety lengths, with 300 MB free: no more
    of them are kept than take a tenth of that, and the answers are those of all windows evaluated."""
    import torch
    x, rng = _record(1 << 22)
    lengths = [20]
    while lengths[-1] < 15_000:
        lengths.append(int(lengths[-1] * 1.08) + 1)
    batches = [[tb.Request(rng.normal(size=m).astype(np.float32), tb.MODE_THRESHOLD, correlation=0.3 + 8 / m ** 0.5)
                for m in lengths[i::9]] for i in range(9)]
    with tb.Context(x) as ctx:
        ctx.set_tiles(tb.TILES_ROWS)
        want = [ctx.scan_batch(b) for b in batches]
    with tb.Context(x) as ctx:
        ctx.set_tiles(tb.TILES_FFT)
        _same(ctx.scan_batch(batches[0]), want[0])  # its other buffers are there now
        with _Taken(300 << 20):
            before = torch.cuda.mem_get_info()[0]
            for b, w in zip(batches, want):
                _same(ctx.scan_batch(b), w)
            assert before - torch.cuda.mem_get_info()[0] < 36 << 20
        for b, w in zip(batches, want):
            _same(ctx.scan_batch(b), w)


def test_a_search_after_one_that_ran_out():
    """The failure of one search is not that of the next on the same thread, nor of a new context."""
    x, rng = _record(1 << 24)
    reqs = [tb.Request(rng.normal(size=300).astype(np.float32), tb.MODE_KNN, k=3, merge_offset=100) for _ in range(3)]
    with tb.Context(x) as ctx:
        ctx.set_tiles(tb.TILES_FFT)
        with _Taken(60 << 20):
            with pytest.raises(tb.TremorError) as e:
                ctx.scan_batch(reqs)
        assert e.value.code == -3
        got = ctx.scan_batch(reqs)
    with tb.Context(x) as ctx:
        _same(got, ctx.scan_batch(reqs))


def test_larger_buckets():
    """The minima of 1000 kNN templates over 2^23 windows take 268 MB in buckets of 256 windows, 34 in buckets
    of 2048: with 150 MB left the larger ones serve."""
    x, rng = _record(1 << 23)
    reqs = [tb.Request(rng.normal(size=64).astype(np.float32), tb.MODE_KNN, k=1 + i % 3, merge_offset=(0, 40, 300)[i % 3])
            for i in range(1000)]
    with tb.Context(x) as ctx:
        ctx.set_tiles(tb.TILES_FFT)
        ctx.scan_batch(reqs[:2])  # the record's own arrays
        with _Taken(150 << 20):
            got = ctx.scan_batch(reqs)
        _same(got, ctx.scan_batch(reqs))
