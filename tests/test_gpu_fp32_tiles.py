"""The FP32 kernel's tiles by what remains of a group beyond whole tiles of 64 templates (8, 16, 32 or
64 templates by 2048 to 256 windows), on records long enough for the narrow ones and too short
for them, around the edges of a warp's windows and a tile's: answers equal the oracle's, and those
of the templates searched one by one."""
import numpy as np
import pytest

import tremor_b200 as tb
from tests import oracle_bindings as ob

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('count', [1, 8, 9, 16, 17, 32, 33, 64, 65, 73, 90])
@pytest.mark.parametrize('windows,m', [(2047, 70), (1 << 16, 128), (2048 * 148 + 1, 40), (303_000, 150)])
def test_remainder_tiles(count, windows, m):
    rng = np.random.default_rng(count + m)
    n = windows + m - 1
    x = np.cumsum(rng.normal(size=n)).astype(np.float32)
    x[n // 2:n // 2 + 300] = 1.0
    q = rng.normal(size=(count, m)).astype(np.float32)
    q[-1] = x[n - m:]
    with tb.Context(x) as ctx:
        ctx.set_kernel(tb.KERNEL_FP32)
        I, D = ctx.search_knn(q, 3, 20)
        hits = ctx.search_threshold(q, 0.8)
        for i in {0, count // 2, count - 1}:
            I1, D1 = ctx.search_knn(q[i:i + 1], 3, 20)
            assert np.array_equal(I[i:i + 1], I1) and np.array_equal(D[i:i + 1].view(np.uint32), D1.view(np.uint32)), i
    last = q[-1:]
    Io, Do = ob.scan_knn(x, last, m, 3, 20)
    assert np.array_equal(I[-1:], Io) and np.array_equal(D[-1:].view(np.uint32), Do.view(np.uint32))
    _, p, d = ob.scan_threshold(x, last, m, 0.8, 0)
    assert np.array_equal(hits[-1][0], p) and np.array_equal(hits[-1][1].view(np.uint32), d.view(np.uint32))
