"""Which strided slices share memory (``csrc/slices.cuh``, plain C++, compiled here):
against the sets of the values themselves.  Tensor-core applies run side by side
where this says that they share none."""

import ctypes as C
from pathlib import Path
import subprocess

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parent.parent/'pyfr_gb300'/'csrc'


@pytest.fixture(scope='module')
def overlap(tmp_path_factory):
    d = tmp_path_factory.mktemp('slices')
    (d/'s.cpp').write_text('''
#include "slices.cuh"
extern "C" int ov(long pa, long ra, long la, long sa, long na, long pb,
                  long rb, long lb, long sb, long nb) {
    return b200::overlap({(void *)pa, ra, la, sa, na}, {(void *)pb, rb, lb, sb, nb});
}
''')
    subprocess.run(['g++', '-std=c++17', '-shared', '-fPIC', '-I', str(CSRC),
                    str(d/'s.cpp'), '-o', str(d/'s.so')], check=True)
    fn = C.CDLL(str(d/'s.so')).ov
    fn.argtypes = [C.c_long]*10
    return lambda a, b: bool(fn(*a, *b))


def _values(p, rows, ld, stride, n):
    return {p//4 + z*stride + i for z in range(n) for i in range(rows*ld)}


def test_overlap_of_slices(overlap):
    rng = np.random.default_rng(0)
    seen = {True: 0, False: 0}
    for _ in range(6000):
        n, s = int(rng.integers(1, 5)), int(rng.integers(0, 40))
        a, b = ((int(4*rng.integers(100, 300)), int(rng.integers(1, 6)),
                 int(rng.integers(1, 6)), s, n) for _ in range(2))
        if rng.random() < 0.3:
            b = b[:3] + (int(rng.integers(0, 40)), int(rng.integers(1, 5)))
        share = bool(_values(*a) & _values(*b))
        got = overlap(a, b)
        if a[3] == b[3] and a[3] > 0:
            assert got == share, (a, b)
        # (other strides: never less than there is)
        assert got or not share, (a, b)
        seen[share] += 1
    assert min(seen.values()) > 500


def test_interleaved_rows_and_slices(overlap):
    ld, m, n = 128, 96, 3
    a = (4096, 32, ld, m*ld, n)
    # other rows of the same slices
    assert not overlap(a, (4096 + 4*32*ld, 64, ld, m*ld, n))
    # the same rows of the next slice, and a stride below the rows
    assert overlap(a, (4096 + 4*m*ld, 32, ld, m*ld, n))
    assert overlap((4096, 32, ld, 16*ld, n), (4096 + 4*32*ld, 32, ld, 16*ld, n))
    # one more slice than there are
    assert not overlap(a, (4096 + 4*n*m*ld, 32, ld, m*ld, n))
    assert not overlap(a, (0, 32, ld, m*ld, n))
