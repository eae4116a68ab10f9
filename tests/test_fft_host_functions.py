"""The FFT branch's host functions (tm_fft.cuh), compiled as they are: classes and parts of every length,
and the base lengths of the chunks' bounds."""
import os
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parents[1] / 'tremor_b200' / 'csrc'
NVCC = shutil.which('nvcc') or '/usr/local/cuda/bin/nvcc'

MAIN = r'''
#include <cstdio>
#include "tm_fft.cuh"
int main()
{
    using namespace tmb;
    for (int m = 1; m <= kFftMaxM; m++)
    {
        const int cls = fft_class_of(m), base = fft_base(m);
        std::printf("%d %d %d %u %d %d %d\n", m, cls, fft_class(cls).n, fft_class(cls).step, fft_parts(m, cls), base,
                    fft_base_length(base));
    }
    return 0;
}
'''


@pytest.fixture(scope='module')
def table(tmp_path_factory):
    if not os.path.exists(NVCC):
        pytest.skip('nvcc not found')
    d = tmp_path_factory.mktemp('fft_host')
    (d / 'main.cu').write_text(MAIN)
    subprocess.run([NVCC, '-std=c++17', '-gencode', 'arch=compute_100a,code=sm_100a', f'-I{CSRC}', str(d / 'main.cu'), '-o',
                    str(d / 'main')], check=True, capture_output=True)
    out = subprocess.run([str(d / 'main')], check=True, capture_output=True, text=True).stdout
    return np.array([line.split() for line in out.splitlines()], dtype=np.int64)


def test_every_length_has_its_windows_without_wrapping(table):
    m, cls, n, step, parts, _, _ = table.T
    assert np.array_equal(m, np.arange(1, 16385)) and np.all(np.diff(cls) >= 0)
    one = parts == 1
    assert np.all(m[one] <= 2 * n[one] - step[one] + 1)  # outputs o + m - 1 of 2 n, o < step
    assert np.all(m[~one] > 2 * n[~one] - step[~one] + 1)
    assert np.all(parts * step >= np.where(one, 0, m)) and parts.max() == 2


def test_base_lengths_are_near_below(table):
    m, base, length = table[:, 0], table[:, 5], table[:, 6]
    assert base.min() >= 0 and base.max() < 100 and np.all(np.diff(base) >= 0)
    assert np.all(length <= m) and np.all((length == m) | (10 * m <= 11 * length + 9))
    for b in np.unique(base):
        assert len(np.unique(length[base == b])) == 1
