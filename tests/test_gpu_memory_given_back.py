"""Device memory of one call is given back when it ends."""
import numpy as np
import pytest

import tremor_b200 as tb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('tiles', [tb.TILES_ROWS, tb.TILES_COLS_64, tb.TILES_FFT])
def test_diagnostics(tiles):
    """Six calls with the exact distances, of 24 bytes per window and template (19 MB) each."""
    import torch
    rng = np.random.default_rng(1)
    x = rng.normal(size=100_000).astype(np.float32)
    q = rng.normal(size=(8, 300)).astype(np.float32)
    free = []
    with tb.Context(x) as ctx:
        ctx.set_tiles(tiles)
        for _ in range(6):
            ctx.bound_diagnostics(q)
            torch.cuda.synchronize()
            free.append(torch.cuda.mem_get_info()[0])
    assert free[1] - free[-1] < 10 << 20
