"""The FP64 reciprocal, square root and quotient of the flux kernels
(``csrc/common.cuh``) against the correctly rounded ones, over the range that
they refine single-precision estimates in (magnitudes of [2^-100, 2^100)), at its
edges, where they hand over to the IEEE operations, and beyond.

Bounds: the reciprocal's last step is one rounding of a value within 2^-64 of
the exact one, and the root's of one within 2^-60: one unit in the last place
of the correctly rounded result.  The quotient is a product with that
reciprocal: two units.  Beyond the range reciprocal and root are the IEEE ones.
"""

import ctypes as C
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SRC = '''
#include "common.cuh"
__global__ void k(int n, const double *x, const double *y, double *r, double *s, double *q) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    r[i] = b200::rcp(x[i]);
    s[i] = b200::root(x[i]);
    q[i] = b200::quot(y[i], x[i]);
}
extern "C" int run(int n, const double *x, const double *y, double *r, double *s, double *q) {
    k<<<(n + 127) / 128, 128>>>(n, x, y, r, s, q);
    return (int)cudaDeviceSynchronize();
}
'''


@pytest.fixture(scope='module')
def functions(tmp_path_factory):
    import torch

    from pyfr_gb300.build import ARCH, CSRC, NVCC_FLAGS, nvcc_path

    d = tmp_path_factory.mktemp('fluxmath')
    (d/'m.cu').write_text(SRC)
    subprocess.run([nvcc_path(), *ARCH, *NVCC_FLAGS, '-I', str(CSRC),
                    '-shared', str(d/'m.cu'), '-o', str(d/'m.so')], check=True)
    run = C.CDLL(str(d/'m.so')).run
    run.argtypes = [C.c_int] + [C.c_void_p]*5

    def call(x, y):
        t = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (x, y)]
        t += [torch.empty_like(t[0]) for _ in range(3)]
        torch.cuda.synchronize()
        assert run(len(x), *(a.data_ptr() for a in t)) == 0
        return [a.cpu().numpy() for a in t[2:]]
    return call


def _ulps(got, want):
    with np.errstate(all='ignore'):
        return np.abs(got - want)/np.spacing(np.abs(want))


def test_inside_the_range(functions):
    rng = np.random.default_rng(2)
    n = 1 << 20
    m = 1 + rng.random(n)
    # (mantissas next to powers of two, and every exponent of the range)
    m[::7] = 1 + 2.0**-52*rng.integers(0, 4, len(m[::7]))
    m[1::7] = 2 - 2.0**-52*rng.integers(1, 4, len(m[1::7]))
    x = m*2.0**rng.integers(-100, 100, n)
    y = rng.standard_normal(n)*2.0**rng.integers(-100, 100, n)
    r, s, q = functions(x, y)
    assert _ulps(r, 1/x).max() <= 1 and _ulps(s, np.sqrt(x)).max() <= 1
    assert _ulps(q, y/x).max() <= 2
    r, s, q = functions(-x, y)
    assert _ulps(r, -1/x).max() <= 1 and np.isnan(s).all()
    assert _ulps(q, -y/x).max() <= 2


def test_edges_and_beyond(functions):
    lo, hi = 2.0**-100, 2.0**100
    x = np.array([lo, np.nextafter(lo, 0), np.nextafter(lo, 1), hi,
                  np.nextafter(hi, 0), np.nextafter(hi, np.inf), 1e-300, 1e300,
                  5e-324, 2.0**-1022, 1.7e308, 0.0, -0.0, np.inf, -np.inf,
                  np.nan, -1.0, -1e-320])
    r, s, _ = functions(x, np.ones_like(x))
    with np.errstate(all='ignore'):
        ri, si = 1/x, np.sqrt(x)
    mid = (np.abs(x) >= lo) & (np.abs(x) < hi)
    for got, want in ((r, ri), (s, si)):
        assert np.array_equal(got[~mid], want[~mid], equal_nan=True)
        assert np.array_equal(np.isnan(got), np.isnan(want))
        f = mid & np.isfinite(want)
        assert _ulps(got[f], want[f]).max() <= 1
