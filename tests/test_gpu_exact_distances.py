"""The exact re-scoring equals the oracle's distance profile, bit for bit, at every window: where
the rounded mean and std are decided from the prefix sums (FFT branch) or from lane sums
(per-length statistics), and where the FP64 chains run; lengths around the 16- and 32-sample
steps; records with a zero mean (means near a float boundary), offsets, level steps, loud and
quiet stretches, constant and missing samples."""
import numpy as np
import pytest

import tremor_b200 as tb
from tests import oracle_bindings as ob
from tests.test_gpu_parity import _templates

pytestmark = pytest.mark.gpu


def _record(kind, n, rng):
    x = rng.normal(size=n).astype(np.float32)
    if kind == 'offset':
        x += np.float32(30000.0)
    if kind == 'steps':
        x[n // 3:] += np.float32(1000.0)
        x[n // 2:n // 2 + 900] *= np.float32(1e5)
        x[n // 2 + 900:n // 2 + 3000] *= np.float32(1e-6)
    if kind == 'gaps':
        x[1000:1400] = 2.5
        x[3000:3300] = tb.MISSING_VALUE
        x[rng.integers(0, n, 40)] = tb.MISSING_VALUE
        x[5000:5400] *= np.float32(1e-14)
    if kind == 'tiny':
        x *= np.float32(1e-9)
        x[::7] *= np.float32(1e-12)
    return x


@pytest.mark.parametrize('tiles', [tb.TILES_FFT, tb.TILES_ROWS])
@pytest.mark.parametrize('kind', ['zero', 'offset', 'steps', 'gaps', 'tiny'])
@pytest.mark.parametrize('m', [2, 15, 16, 17, 31, 32, 33, 64, 257, 1000, 4111])
def test_exact_distances(m, kind, tiles):
    rng = np.random.default_rng(m)
    x = _record(kind, 9001 + m, rng)
    if kind != 'gaps':  # the second of these crosses prefix blocks
        x = np.concatenate([x, _record(kind, 66000 - len(x), rng)]) if m in (33, 1000) else x
    q = _templates(x, m, rng, 2)
    with tb.Context(x) as ctx:
        ctx.set_tiles(tiles)
        _, _, exact = ctx.bound_diagnostics(q)
    present = x[:len(x) - m + 1] != tb.MISSING_VALUE
    for i in range(2):
        want = ob.distance_profile(x, q[i], m)
        assert np.array_equal(exact[i][present].view(np.uint32), want[present].view(np.uint32)), i
