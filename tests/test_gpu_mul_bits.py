"""FP64 operator applies where the largest entries of a row meet zeros or small
values, and operators whose entries span many orders of magnitude: every output
against extended precision with a bound over its own terms.

Bound, u = 2^-53: an output of n terms is within n u of their absolute sum,
as FP64 sums are, and rounded once more.  Operators whose rows come in groups
of one support of 3 to 6 entries (of n and n - 1), none of them below 1/16 of the
largest row's mean, are summed in fixed point with a bound of (1 + 5 n/8) u/16 of
(largest row sum)(largest value of the support), if that is more.
"""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

U = 2.0**-53


def _operator(kind):
    from pyfr_gb300.shapes import get_shape

    rng = np.random.default_rng(1)
    if kind == 'groups-spread':
        # 24 rows by fours over supports of four columns, entries over 2^-40..1
        a = np.zeros((24, 24))
        for g in range(6):
            a[4*g:4*g + 4, 4*g:4*g + 4] = \
                rng.standard_normal((4, 4))*2.0**-np.arange(0, 40, 10)
        return a
    if kind == 'dense-spread':
        return rng.standard_normal((30, 24))*2.0**-rng.integers(0, 50, (30, 24))
    name, p, op = kind.split('-')
    s = get_shape(name, int(p), *(('alpha-opt',)*2 if name == 'tet' else ()))
    ops = {'grad': 'M4 - M6*M0', 'm132': 'M1 - M3*M2'}
    return s.opmat(ops[op]) if op in ops else getattr(s, op)


def _grouped(a):
    """The rule of the grouped form, on the rows' supports and entries."""
    by, l1 = {}, np.abs(a).sum(1)
    for r in a != 0:
        by[r.tobytes()] = by.get(r.tobytes(), 0) + 1
    n = (a != 0).sum(1)
    least = np.abs(a[a != 0]).min()
    return 3 <= n.min() and n.max() <= min(6, n.min() + 1) and \
        l1.min() >= l1.max()/16 and 16*n.max()*least >= l1.max() and \
        len(a) >= 2*sum(-(-c//4) for c in by.values())


def _data(what, k, n, rng):
    b = rng.standard_normal((k, n))
    if what == 'sparse':
        # one to three values of a column, of any size to one another
        keep = rng.random((k, n)).argsort(0) < rng.integers(1, 4, n)
        b *= keep*2.0**-rng.integers(0, 30, (k, n))
    elif what == 'pulse':
        x = np.linspace(-1, 1, k)[:, None]
        b = (1 + 0.1*b)*np.exp(-((x + 1)/rng.uniform(0.1, 0.6, n))**2/2)
    elif what == 'positive':
        b = 1.5 + 0.2*b
    elif what == 'exponents':
        b *= 2.0**rng.integers(-90, 90, (k, n))
    return b


@pytest.mark.parametrize('ncol', [37, 9730, 19461])
@pytest.mark.parametrize('what', ['normal', 'positive', 'sparse', 'pulse',
                                  'exponents'])
@pytest.mark.parametrize('kind', ['tet-3-grad', 'tet-4-m6', 'tet-4-m3',
                                  'hex-2-m0', 'hex-3-grad', 'hex-3-m0',
                                  'hex-4-grad', 'hex-5-m0', 'quad-4-m132',
                                  'groups-spread',
                                  'dense-spread'])
def test_terms_keep_their_bits(kind, what, ncol):
    if ncol > 9730 and kind not in ('tet-3-grad', 'tet-4-m3', 'dense-spread'):
        pytest.skip('the largest width: dense rows')
    import torch

    from pyfr_gb300.backend import B200Backend
    from pyfr_gb300.inifile import Inifile

    lib = B200Backend(Inifile()).lib
    a = np.ascontiguousarray(_operator(kind), dtype=np.float64)
    m, k = a.shape
    rng = np.random.default_rng(3)
    b = _data(what, k, ncol, rng)
    c0 = rng.standard_normal((m, ncol))

    ref = np.zeros((m, ncol), dtype=np.longdouble)
    absum, top = np.zeros((m, ncol)), np.zeros((m, ncol))
    for j in range(k):
        nz = np.flatnonzero(a[:, j])
        t = a[nz, j].astype(np.longdouble)[:, None]*b[j]
        ref[nz] += t
        absum[nz] += np.abs(t).astype(np.float64)
        top[nz] = np.maximum(top[nz], np.abs(b[j]))
    n = (a != 0).sum(1)[:, None]
    tol = (n + 2)*absum
    if _grouped(a):
        l1 = np.abs(a).sum(1).max()
        tol = np.maximum(tol, (1 + 5*n.max()/8)/16*l1*top + absum)
    tol = U*tol*(1 + 1e-9)

    h = C.c_void_p()
    lib.mul_create(a.ctypes.data_as(C.POINTER(C.c_double)), m, k, C.byref(h))
    db = torch.from_numpy(b).cuda()
    for alpha, beta in ((1.0, 0.0), (1.0, 1.0), (2.0, 0.0), (-0.5, 0.25)):
        dc = torch.from_numpy(c0).cuda()
        torch.cuda.synchronize()
        lib.mul_f64(h, db.data_ptr(), ncol, dc.data_ptr(), ncol, ncol,
                    C.c_double(alpha), C.c_double(beta), None)
        torch.cuda.synchronize()
        want = alpha*ref + beta*c0
        # (the sum, its scaling and the old output's, and their sum rounded;
        # with the FP64 form the old output is one of the terms)
        old = np.abs(beta*c0)
        lim = abs(alpha)*(tol + 2*U*np.abs(ref)) + (n + 3)*U*old
        err = np.abs(dc.cpu().numpy() - want)
        assert np.all(err <= lim), (alpha, beta, float((err/(lim + 1e-300)).max()))
    lib.mul_destroy(h)


@pytest.mark.parametrize('ncol', [33, 200, 9731, 19461])
@pytest.mark.parametrize('what', ['normal', 'sparse', 'exponents'])
@pytest.mark.parametrize('kind', ['groups', 'dense', 'short'])
def test_in_place(kind, what, ncol):
    """An apply onto its own input, for an operator of each form (rows in
    groups of one support; twenty entries a row, whose fixed-point form has to
    be declined, since it reads the input again for outputs of small terms; two
    entries a row): as the same apply to a copy, and within its bound."""
    import torch

    from pyfr_gb300.backend import B200Backend
    from pyfr_gb300.inifile import Inifile

    lib = B200Backend(Inifile()).lib
    rng = np.random.default_rng(5)
    m = 24
    if kind == 'groups':
        a = np.kron(np.eye(6), 1 + rng.random((4, 4)))
        assert _grouped(a)
    elif kind == 'dense':
        a = rng.standard_normal((m, m))
        a[:, 20:] = 0
        a[:, :20] += np.sign(a[:, :20])
    else:
        a = np.kron(np.eye(12), rng.standard_normal((2, 2)))
    a = np.ascontiguousarray(a)
    b = _data(what, m, ncol, rng)
    h = C.c_void_p()
    lib.mul_create(a.ctypes.data_as(C.POINTER(C.c_double)), m, m, C.byref(h))
    d, e = torch.from_numpy(b).cuda(), torch.from_numpy(b).cuda()
    out = torch.empty_like(d)
    torch.cuda.synchronize()
    for src, dst in ((d, out), (e, e)):
        lib.mul_f64(h, src.data_ptr(), ncol, dst.data_ptr(), ncol, ncol,
                    C.c_double(1.0), C.c_double(0.0), None)
    torch.cuda.synchronize()
    lib.mul_destroy(h)
    ref = (a.astype(np.longdouble)[:, :, None]*b).sum(1)
    n = (a != 0).sum(1)[:, None]
    tol = U*(n + 2)*(np.abs(a) @ np.abs(b))*(1 + 1e-9)
    if kind == 'groups':
        sup = np.repeat(np.abs(b).reshape(6, 4, ncol).max(1), 4, axis=0)
        tol = np.maximum(tol, U*((1 + 5*4/8)/16*np.abs(a).sum(1).max()*sup +
                                 np.abs(a) @ np.abs(b)))
    for t in (out, e):
        assert np.all(np.abs(t.cpu().numpy() - ref) <= tol)
    assert kind == 'dense' or torch.equal(out, e)
