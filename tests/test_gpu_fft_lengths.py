"""The FFT branch at the edges of its length classes and pieces.

Every (template, window) pair of small records through tm_bound_diagnostics: the windows
without a distance are exactly the constant ones and those that start at a missing sample
(NumPy decides), and elsewhere |d - exact| <= e, the bound itself (no tolerance). Three
templates of one length, so that the window statistics kept for the second and third are
used; records whose last piece is full, nearly empty, or one sample long."""
import numpy as np
import pytest

import tremor_b200 as tb
from tests.test_gpu_runs import _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('m,extra', [(31, 1), (1025, 0), (1026, 6143), (2049, 6145), (2050, 1), (4097, 12288),
                                     (4098, 0), (8192, 8191), (8193, 1), (12000, 4097), (16384, 8193)])
def test_length_classes(m, extra):
    """Lengths on both sides of the class edges (1025, 2049, 4097, 8192); `extra` windows beyond
    the first piece's, around whole numbers of steps."""
    rng = np.random.default_rng(m)
    step = 7168 if m <= 1025 else 6144 if m <= 2049 else 12288 if m <= 4097 else 8192
    x = rng.normal(size=step + extra + m - 1).astype(np.float32) + np.float32(2.0)
    x[100:100 + m + 5] = 1.5  # constant windows at the start
    x[rng.integers(0, len(x), 20)] = tb.MISSING_VALUE
    _check(x, m, tb.TILES_FFT)
