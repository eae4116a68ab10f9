"""Records that drift many standard deviations within a prefix block, whose centre is the FFT branch's
shift: its bound holds, and is no looser for it than the other kernels'."""
import numpy as np
import pytest

import tremor_b200 as tb

pytestmark = pytest.mark.gpu


def _drifting(n, slope, rng):
    from tremor_b200 import synth
    return (synth.ar2_waveform(n, rng) + slope * np.arange(n) + 100.0).astype(np.float32)


@pytest.mark.parametrize('slope', [0.05, 3.0])
@pytest.mark.parametrize('m', [30, 1000, 2500, 8192, 16384])
def test_bound_holds(m, slope):
    rng = np.random.default_rng(m)
    x = _drifting(140_000, slope, rng)
    q = np.stack([x[p:p + m] + (0.5 * x[p:p + m].std() * rng.normal(size=m)).astype(np.float32) for p in (100, 50_000, 110_000)])
    with tb.Context(x) as ctx:
        ctx.set_tiles(tb.TILES_FFT)
        d, e, exact = ctx.bound_diagnostics(q)
    ok = np.isfinite(d)
    err = np.abs(d[ok].astype(np.float64) - exact[ok].astype(np.float64))
    assert ok.any() and np.all(err <= e[ok]), (m, float(np.max(err / e[ok])))  # a short window on a steep record is not trusted


@pytest.mark.parametrize('m', [1500, 4096])
@pytest.mark.parametrize('merge', [0, 1])
def test_few_candidates(m, merge):
    """kNN candidates, against those of the FP32 kernel, whose shifts and statistics are the windows' own: at
    most four times as many (the re-pass that emits them has the same bound; the kNN bound itself may
    be looser)."""
    rng = np.random.default_rng(m + merge)
    x = _drifting(1 << 19, 0.05, rng)
    reqs = [tb.Request(rng.normal(size=m).astype(np.float32), tb.MODE_KNN, k=10, merge_offset=merge * m // 2) for _ in range(24)]
    with tb.Context(x) as ctx:
        ctx.set_tiles(tb.TILES_FFT)
        got, many = ctx.scan_batch(reqs), ctx.last_candidates()
        ctx.set_kernel(tb.KERNEL_FP32)
        ctx.set_tiles(tb.TILES_AUTO)
        want, few = ctx.scan_batch(reqs), ctx.last_candidates()
    for i, ((p0, d0), (p1, d1)) in enumerate(zip(got, want)):
        assert np.array_equal(p0, p1) and np.array_equal(d0.view(np.uint32), d1.view(np.uint32)), i
    print(m, merge, 'candidates', many, few)
    assert many <= 4 * few
