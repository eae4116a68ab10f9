"""What the server counts for a request before it admits it."""
import numpy as np
import pytest

import tremor_b200 as tb

pytestmark = pytest.mark.gpu


def _served(x, reqs, **config):
    with tb.Context(x) as ctx:
        server = ctx.serve(workers=1, max_batch=64, **config)
        tickets = [server.submit(r) for r in reqs]
        sizes = {}
        while len(sizes) < len(tickets):
            for c in server.poll():
                assert c.status == 0
                sizes[c.ticket] = c.batch_size
        server.stop()
    return [sizes[t] for t in tickets]


def test_bucket_minima_count():
    """2^24 windows: a kNN request's minima take 0.5 MB, the rest of its estimate 0.2: with a budget of 1 MB
    one is admitted at a time."""
    rng = np.random.default_rng(1)
    x = rng.normal(size=1 << 24).astype(np.float32)
    reqs = [tb.Request(rng.normal(size=200).astype(np.float32), tb.MODE_KNN, k=1, merge_offset=100) for _ in range(8)]
    assert max(_served(x, reqs, memory_budget=1_000_000)) == 1
