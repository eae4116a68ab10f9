"""Windows that end just before a sample far louder than they are: the prefix sums up to there must not carry
its rounding. Distances equal the oracle's bit for bit, and the bound holds."""
import numpy as np
import pytest

import tremor_b200 as tb
from tests.test_gpu_batching import _check

pytestmark = pytest.mark.gpu


def _record(rng):
    from tremor_b200 import synth
    x = synth.ar2_waveform(14 * 65536, rng)
    # the first of its prefix block, at each place among the 8 samples that a thread sums
    at = 65536 * np.arange(14) + 8 * rng.integers(300, 500, size=14) + np.arange(14) % 8
    x[at] = (10.0 ** rng.uniform(5, 7.5, size=14) * x.std()).astype(np.float32)
    return x


@pytest.mark.parametrize('m', [8, 29, 100, 250])
def test_distances(m):
    rng = np.random.default_rng(m)
    x = _record(rng)
    t = rng.normal(size=(2, m)).astype(np.float32)
    reqs = [tb.Request(t[0], tb.MODE_THRESHOLD, correlation=-1.0), tb.Request(t[1], tb.MODE_KNN, k=600, merge_offset=0)]
    for tiles in (tb.TILES_FFT, tb.TILES_COLS_32):
        with tb.Context(x) as ctx:
            ctx.set_tiles(tiles)
            for repeat in (1, 8):  # few candidates, and enough for a thread each
                answers = ctx.scan_batch(reqs * repeat)
                _check(x, reqs, answers[-2:])


@pytest.mark.parametrize('m', [29, 100, 250])
def test_bound(m):
    rng = np.random.default_rng(m + 1)
    x = _record(rng)
    with tb.Context(x) as ctx:
        ctx.set_tiles(tb.TILES_FFT)
        d, e, exact = ctx.bound_diagnostics(rng.normal(size=(3, m)).astype(np.float32))
    ok = np.isfinite(d)
    err = np.abs(d[ok].astype(np.float64) - exact[ok].astype(np.float64))
    assert ok.any() and np.all(err <= e[ok]), float(np.max(err / e[ok]))
