"""FP64 operator applies in fixed point (``csrc/mul.cu``) against FP64 sums in
extended precision.

The bound of one output: its final rounding, the truncation of B below the
column's largest value and of A below the row's absolute sum, each at most
2^-53 (row sum)(largest |B| the row touches) by the kernel's support test
(see the kernel's notes), so 4 2^-53 of that product is allowed, and with
beta = 1 one rounding of the sum more.  Outputs that are formed with FP64
FMAs (narrow or short rows, small supports) have the classical bound, one
2^-53 of the terms' absolute sum per term, the old output being one of the
terms with beta = 1.
"""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = 2.0**-53


def _operator(kind, p):
    from pyfr_gb300.shapes import get_shape
    if kind == 'tet':
        return get_shape('tet', p, 'alpha-opt', 'alpha-opt').m4
    if kind == 'wide':
        # (rows up to the longest that the fixed-point form takes, an empty
        # row, and a row of one entry)
        a = np.cos(1.0 + np.arange(9*64).reshape(9, 64)*0.37)
        a[3] = 0.0
        a[4, :-1] = 0.0
        return a
    s = get_shape('hex', p)
    return {'m0': s.m0, 'm3': s.m3, 'm4': s.opmat('M4 - M6*M0'),
            'm132': s.opmat('M1 - M3*M2')}[kind]


def _data(what, k, n, rng):
    col = np.arange(n)
    b = np.sin(0.1*np.arange(k)[:, None] + 0.37*col)
    match what:
        case 'mean':
            b = 178.0 + 0.01*b
        case 'zeros':
            b[:, ::3] = 0.0
            b[k//2:, 1::3] = 0.0
            b[1::2, 2::3] = -0.0
        case 'range':
            b = b*2.0**rng.integers(-70, 70, (k, n))
        case 'ends':
            b = b*np.where(col % 2, 1e300, 1e-300)
            b[:, ::5] = 5e-324*rng.integers(0, 9, (k, len(b[0, ::5])))
        case 'special':
            b[0, ::4] = np.inf
            b[k - 1, 1::4] = np.nan
            b[k//2, 2::4] = -np.inf
    return b


@pytest.mark.parametrize('ncol', [1, 31, 64, 65, 9728, 9735, 20002])
@pytest.mark.parametrize('kind,p', [('m0', 3), ('m3', 3), ('m4', 3),
                                    ('m132', 3), ('m4', 1), ('tet', 3),
                                    ('wide', 0), ('m0', 2), ('m0', 4)])
@pytest.mark.parametrize('what', ['smooth', 'mean', 'zeros', 'range', 'ends',
                                  'special'])
def test_fixed_point_apply(kind, p, ncol, what):
    if ncol > 9735 and what != 'smooth':
        pytest.skip('the largest width: one kind of data')
    import torch
    from pyfr_gb300.backend import B200Backend
    from pyfr_gb300.inifile import Inifile

    lib = B200Backend(Inifile()).lib
    a = np.ascontiguousarray(_operator(kind, p), dtype=np.float64)
    m, k = a.shape
    rng = np.random.default_rng(7)
    b = _data(what, k, ncol, rng)
    c0 = rng.standard_normal((m, ncol))

    h = C.c_void_p()
    lib.mul_create(a.ctypes.data_as(C.POINTER(C.c_double)), m, k, C.byref(h))
    # (an even leading dimension takes the 16-byte accesses, an odd one
    # does not)
    for ld, beta in ((ncol + ncol % 2, 0.0), (ncol + 1 - ncol % 2, 1.0)):
        db = torch.zeros((k, ld), dtype=torch.float64, device='cuda')
        dc = torch.full((m, ld), 7.0, dtype=torch.float64, device='cuda')
        db[:, :ncol] = torch.from_numpy(b).cuda()
        dc[:, :ncol] = torch.from_numpy(c0).cuda()
        torch.cuda.synchronize()
        lib.mul_f64(h, db.data_ptr(), ld, dc.data_ptr(), ld, ncol,
                    C.c_double(1.0), C.c_double(beta), None)
        torch.cuda.synchronize()
        got = dc.cpu().numpy()
        assert np.all(got[:, ncol:] == 7.0)
        got = got[:, :ncol]

        with np.errstate(all='ignore'):
            ref = np.zeros((m, ncol), dtype=np.longdouble)
            absum = np.zeros((m, ncol), dtype=np.longdouble)
            top = np.zeros((m, ncol))
            for j in range(k):
                nz = np.flatnonzero(a[:, j])
                t = a[nz, j].astype(np.longdouble)[:, None]*b[j]
                ref[nz] += t
                absum[nz] += abs(t)
                top[nz] = np.maximum(top[nz], abs(b[j]))
            l1 = abs(a).sum(axis=1)[:, None].astype(np.longdouble)
            nnz = (a != 0).sum(axis=1)[:, None]
            if beta:
                ref = ref + c0
            old = abs(c0) if beta else 0.0
            tol = np.maximum(4*l1*top, nnz*(absum + old))*EPS + \
                EPS*(abs(ref) + old) + 1e-322
            r64 = ref.astype(np.float64)
            fin = np.isfinite(r64)
            # (infinities and NaNs where FP64 sums have them)
            assert np.array_equal(np.isnan(got), np.isnan(r64))
            ninf = ~fin & ~np.isnan(r64)
            assert np.array_equal(got[ninf], r64[ninf])
            err = abs(got[fin].astype(np.longdouble) - ref[fin])
            assert np.all(err <= tol[fin]), float((err/tol[fin]).max())
    lib.mul_destroy(h)


def test_in_place_apply():
    """An apply onto its own input is formed as before (no input is read
    after an output of its column is written)."""
    import torch
    from pyfr_gb300.backend import B200Backend
    from pyfr_gb300.inifile import Inifile

    lib = B200Backend(Inifile()).lib
    rng = np.random.default_rng(3)
    a = rng.standard_normal((8, 8))
    b = rng.standard_normal((8, 200))*2.0**rng.integers(-60, 60, (8, 200))
    h = C.c_void_p()
    lib.mul_create(a.ctypes.data_as(C.POINTER(C.c_double)), 8, 8, C.byref(h))
    d = torch.from_numpy(b).cuda()
    torch.cuda.synchronize()
    lib.mul_f64(h, d.data_ptr(), 200, d.data_ptr(), 200, 200, C.c_double(1.0),
                C.c_double(0.0), None)
    torch.cuda.synchronize()
    tol = 8*EPS*(abs(a) @ abs(b))
    assert np.all(abs(d.cpu().numpy() - a @ b) <= 2*tol)
    lib.mul_destroy(h)
