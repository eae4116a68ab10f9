"""Batches destroyed after their context: their buffers and the context's memory pool go with the last of
them, and the device stays usable."""
import numpy as np
import pytest

import tremor_b200 as tb

pytestmark = pytest.mark.gpu


def test_batches_outlive_their_context():
    """40 contexts with three batches each, closed before, after and along with them; 60 MB of templates a
    context."""
    import torch
    rng = np.random.default_rng(1)
    x = rng.normal(size=50_000).astype(np.float32)
    reqs = [tb.Request(rng.normal(size=m).astype(np.float32), tb.MODE_KNN, k=2, merge_offset=m // 2)
            for m in [100, 300, 4000] + [9000] * 200]
    free, held = [], []
    for i in range(40):
        ctx = tb.Context(x)
        ctx.set_tiles((tb.TILES_FFT, tb.TILES_ROWS)[i % 2])
        batches = [ctx.batch(reqs) for _ in range(3)]
        out = batches[0].run()
        assert len(out) == len(reqs)
        batches.pop(i % 3).close()
        ctx.close()
        held.append(batches)
        if i % 4 == 3:  # some contexts later
            for kept in held:
                for b in kept:
                    b.close()
            held.clear()
            torch.cuda.synchronize()
            free.append(torch.cuda.mem_get_info()[0])
    assert free[0] - free[-1] < 16 << 20
