"""The claims behind skipped windows (chunk_limit, tm_fftk.cu), in float64: what 1 / std and the mean of
the windows of m0 samples say about the longer windows that begin at the same places, and that
the base lengths are close enough below every length."""
import numpy as np
import pytest


def _windows(x, m):
    w = np.lib.stride_tricks.sliding_window_view(x, m)
    return w.mean(1), w.std(1)


@pytest.mark.parametrize('kind', ['noise', 'offset', 'drift', 'steps', 'quiet_then_loud', 'spike'])
@pytest.mark.parametrize('m0,m', [(2, 2), (2, 3), (10, 11), (64, 70), (300, 329), (1000, 1099)])
def test_longer_windows_are_bounded(kind, m0, m):
    rng = np.random.default_rng(m)
    x = rng.normal(size=6000)
    if kind == 'offset':
        x += 1e4
    elif kind == 'drift':
        x = np.cumsum(x)
    elif kind == 'steps':
        x += np.repeat(rng.normal(size=60) * 100, 100)
    elif kind == 'quiet_then_loud':
        x[:3000] *= 1e-3
    elif kind == 'spike':
        x[::500] = 1e5
    mu0, sd0 = _windows(x, m0)
    mu, sd = _windows(x, m)
    mu0, sd0 = mu0[:len(mu)], sd0[:len(mu)]
    g, h = np.sqrt(m / m0), np.sqrt((m - m0) / m0)
    slack = 1e-9 * (1 + np.abs(mu)) / sd0  # of this float64 evaluation
    assert np.all(1 / sd <= g / sd0 * (1 + slack))
    for shift in (0.0, float(x[0]), 1e3):
        assert np.all(np.abs(mu - shift) / sd <= g * np.abs(mu0 - shift) / sd0 * (1 + slack) + h + slack)


def test_base_lengths():
    """fft_base_next's sequence from 1 on, 100 entries: reaches 16384, and the largest entry that a
    length reaches is at most a tenth below it."""
    bases = [1]
    while len(bases) < 100:
        b = bases[-1]
        bases.append(max(b + 1, b * 11 // 10))
    assert bases[-1] > 16384
    for m in range(1, 16385):
        b = max(v for v in bases if v <= m)
        assert b == m or 10 * m <= 11 * b + 9, m
