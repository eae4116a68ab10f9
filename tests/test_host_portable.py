"""The host library's source asks for x86 code on x86 only: preprocessed for another machine (the
macros taken away, empty headers), no function is cloned for an x86 feature."""
import re
import subprocess
from pathlib import Path

SOURCE = Path(__file__).resolve().parents[1] / 'tremor_b200' / 'csrc' / 'tm_host.cpp'


def _preprocessed(tmp_path, *flags):
    for name in re.findall(r'#include <([^>]+)>', SOURCE.read_text() + SOURCE.with_suffix('.h').read_text()):
        (tmp_path / name).parent.mkdir(parents=True, exist_ok=True)
        (tmp_path / name).touch()
    return subprocess.run(['g++', '-E', '-nostdinc', '-nostdinc++', f'-I{tmp_path}', *flags, str(SOURCE)], check=True,
                          capture_output=True, text=True).stdout


def test_no_x86_clones_elsewhere(tmp_path):
    assert 'target_clones' not in _preprocessed(tmp_path, '-U__x86_64__', '-U__i386__')
    assert 'znormalize' in _preprocessed(tmp_path)
