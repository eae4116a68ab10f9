"""The constant runs that decide which windows are searched.

Every (template, window) pair of small records through tm_bound_diagnostics: the windows
without a distance are exactly the constant ones and those that start at a missing sample
(NumPy decides), and elsewhere |d - exact| <= e, the bound itself (no tolerance)."""
import numpy as np
import pytest

import tremor_b200 as tb
from tests.test_gpu_parity import _templates

pytestmark = pytest.mark.gpu


def _searched(x, m):
    """Windows that are searched: first sample present, samples (missing as 0) not all equal."""
    clean = np.where(x == tb.MISSING_VALUE, np.float32(0), x)
    last = np.full(len(x), len(x) - 1)  # last index of the run of equal samples from i on
    ends = np.flatnonzero(clean[1:] != clean[:-1])
    where = np.searchsorted(ends, np.arange(len(x)))
    inside = where < len(ends)
    last[inside] = ends[where[inside]]
    W = len(x) - m + 1
    return (x[:W] != tb.MISSING_VALUE) & (last[:W] - np.arange(W) + 1 < m)


def _check(x, m, tiles):
    q = _templates(x, m, np.random.default_rng(m + 7), 3)
    with tb.Context(x) as ctx:
        ctx.set_tiles(tiles)
        d, e, exact = ctx.bound_diagnostics(q)
    ok = _searched(x, m)
    assert np.array_equal(np.isfinite(d), np.broadcast_to(ok, d.shape)), m
    assert np.all(np.abs(d[:, ok].astype(np.float64) - exact[:, ok]) <= e[:, ok]), m


@pytest.mark.parametrize('tiles', [tb.TILES_FFT, tb.TILES_COLS_64])
@pytest.mark.parametrize('m', [8, 300])
def test_constant_runs(m, tiles):
    """Runs that start or end at the edges of the 8192-sample chunks in which they are found, one
    over several chunks, one longer than 65535, one up to the record's end, missing samples
    within and next to them."""
    rng = np.random.default_rng(m)
    n = 200003
    x = rng.normal(size=n).astype(np.float32)
    x[8192:8192 + 400] = 3.0
    x[3 * 8192 - 400:3 * 8192] = -2.0
    x[5 * 8192 - 7:8 * 8192 + 9] = 0.0
    x[6 * 8192:6 * 8192 + 500] = tb.MISSING_VALUE  # counts as 0: the run goes on
    x[90000:90000 + 70000] = 0.25
    x[n - 350:] = 1.0
    x[8192 + 400] = tb.MISSING_VALUE
    _check(x, m, tiles)
