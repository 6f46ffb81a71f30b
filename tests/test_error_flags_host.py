"""The device error flags are words, numbered by LC3D_FLAG_*: no source may
use such a number as a bit of one word."""
import glob
import re

from conftest import ROOT


def test_flag_numbers_are_not_used_as_bits():
    internal = open(f'{ROOT}/lcode3d_b200/csrc/lc3d_internal.cuh').read()
    flags = {n: int(v) for n, v in re.findall(r'#define (LC3D_FLAG_\w+) (\d+)', internal)}
    count = int(re.search(r'#define LC3D_FLAGS (\d+)', internal).group(1))
    assert sorted(flags.values()) == list(range(count))
    for path in glob.glob(f'{ROOT}/lcode3d_b200/csrc/*.cu*'):
        for line in open(path):
            if any(n in line for n in flags) and '#define' not in line:
                assert 'raise_flag(' in line or re.search(r'flags\[LC3D_FLAG_\w+\]', line), (path, line)
