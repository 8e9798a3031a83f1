"""FP64 element kernels on elements whose fluxes span many orders of magnitude:
every output of the divergence and of the lift against extended precision, with
a bound over that output's own operands.

The mass equation is used: its flux is the momentum itself, and with unit metric
terms (the diagonal form) that of the elements' reference coordinates, so what
goes into the products is known to the last bit.

Bound of one output, u = 2^-53, R the line matrix's largest row sum, B the
output's own largest operand: each line's integer sum is truncated by at most
one unit for its low products' carry, 7/2 for the products of low parts that
are left out, 1/4 for the 60 bits of B and one where it is shifted to a larger
line's exponent, a unit being 2^-56 R B or less: 6/8 u R B a line and so
below 3 u R B; another u R B is allowed for the rounding of the sum to FP64 and
the scaling.  The middle point of an odd line is no operand of its own output;
where it is more than four times the others the line is formed by FMAs, and below
that the units of such an output are four times as large: below 9 u R B.  The
two-dimensional Euler form makes one sum of both lines, with B in 58 bits, over
the output's operands alone: units of 2^-54 R B, one and 7 and 1/2 of them,
below 5 u R B.  Where outputs are formed with FP64 operations the classical bound
holds, u (n + 2) times the absolute sum of the n terms.
"""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

U = 2.0**-53


def _lines(nd, q):
    from pyfr_gb300.backend.tensorele import _line_points, line_operators
    from pyfr_gb300.shapes import get_shape

    b = get_shape({2: 'quad', 3: 'hex'}[nd], q - 1)
    grad, interp, div, fpt = line_operators(
        nd, q, b.m0, b.opmat('M1 - M3*M2'), b.m3, b.opmat('M4 - M6*M0'), b.m6)
    mats = [np.ascontiguousarray(m) for m in (grad, interp, div)]
    return mats, np.ascontiguousarray(fpt, dtype=np.int32), _line_points(nd, q)


def _pulse(what, x, ne, rng):
    """Values at the points x (npts, nd) of every element."""
    shape = (len(x), ne)
    noise = 1 + 0.1*rng.standard_normal(shape)
    if what == 'smooth':
        return noise + np.sin(x.sum(1))[:, None]
    if what == 'zeros':
        return noise*rng.integers(0, 2, shape)
    if what == 'exponents':
        return noise*2.0**rng.integers(-120, 120, shape)
    if what == 'middle':
        # tall on the middle planes of the element, by up to 2^60
        tall = (np.abs(x) < 1e-9).sum(1)[:, None]
        return noise*2.0**(tall*rng.integers(0, 20, ne))
    # a Gaussian pulse in a corner of the element, of this width
    r2 = ((x + 1)**2).sum(1)
    return noise*np.exp(-r2/(2*float(what)**2))[:, None]


def _dev(a, nv=1):
    """(npts, nv, neles) in blocks of 32 elements, variables within."""
    import torch

    npts, _, ne = a.shape
    nb = -(-ne//32)
    out = np.zeros((npts, nb, nv, 32))
    for e in range(ne):
        out[:, e//32, :, e % 32] = a[:, :, e]
    return torch.from_numpy(out.reshape(npts, -1)).cuda()


def _host(t, npts, nv, ne):
    a = t.cpu().numpy().reshape(npts, -1, nv, 32).transpose(0, 2, 1, 3)
    return a.reshape(npts, nv, -1)[:, :, :ne]


def _sums(terms):
    """(sum, absolute sum, largest operand) of (coefficient, values) terms in
    extended precision, of one output point."""
    s = a = t = 0
    for c, x in terms:
        if c == 0:
            continue
        p = np.longdouble(c)*x
        s, a, t = s + p, a + abs(p), np.maximum(t, abs(x))
    return s, a, t


@pytest.mark.parametrize('what', ['0.5', '0.3', '0.2', '0.15', 'smooth',
                                  'zeros', 'exponents', 'middle'])
@pytest.mark.parametrize('kernel', ['euler', 'gradflux', 'lift'])
@pytest.mark.parametrize('nd,q', [(2, 3), (2, 4), (2, 5), (3, 3), (3, 4),
                                  (3, 5)])
def test_outputs_keep_their_own_bits(nd, q, kernel, what):
    import torch

    from pyfr_gb300.backend import B200Backend
    from pyfr_gb300.backend.lib import Gas
    from pyfr_gb300.inifile import Inifile
    from pyfr_gb300.shapes import get_shape

    lib = B200Backend(Inifile()).lib
    (grad, interp, div), fpt, lines = _lines(nd, q)
    basis = get_shape({2: 'quad', 3: 'hex'}[nd], q - 1)
    ne, nv, npts, nf = 37, nd + 2, q**nd, basis.nfpts
    rng = np.random.default_rng(100*nd + q)
    pd = C.POINTER(C.c_double)
    h = C.c_void_p()
    lib.te_create(nd, q, *(m.ctypes.data_as(pd) for m in (grad, interp, div)),
                  fpt.ctypes.data_as(C.POINTER(C.c_int)), C.byref(h))

    mom = [_pulse(what, basis.upts, ne, rng) for _ in range(nd)]
    u = np.zeros((npts, nv, ne))
    u[:, 0] = 1.0
    u[:, 1:-1] = np.stack(mom, axis=1)
    u[:, -1] = 2.5 + 0.5*(u[:, 1:-1]**2).sum(1)
    fc = np.zeros((nf, nv, ne))
    fc[:, 0] = _pulse(what, basis.fpts, ne, rng)
    old = np.zeros((npts, nv, ne))
    old[:, 0] = _pulse(what, basis.upts, ne, rng)

    du, dfc, dr = _dev(u, nv), _dev(fc, nv), _dev(old, nv)
    ld = du.shape[1]
    sm = torch.ones((nd, -(-ne//32)*nd*32), dtype=torch.float64, device='cuda')
    rj = torch.ones((1, ld), dtype=torch.float64, device='cuda')
    gf = torch.zeros((nd*nf, ld), dtype=torch.float64, device='cuda')
    diag = 3
    torch.cuda.synchronize()
    if kernel == 'euler':
        lib.te_euler_f64(h, ne, diag, C.c_double(1.4), du.data_ptr(), ld,
                         dfc.data_ptr(), ld, sm.data_ptr(), sm.shape[1],
                         rj.data_ptr(), ld, dr.data_ptr(), ld, None)
    elif kernel == 'gradflux':
        gas = Gas()
        gas.gamma, gas.mu, gas.pr = 1.4, 1e-3, 0.7
        lib.te_gradflux_ns_f64(h, ne, diag, C.byref(gas), du.data_ptr(), ld,
                               dfc.data_ptr(), ld, gf.data_ptr(), ld,
                               4**nd - 1, 0, sm.data_ptr(), sm.shape[1],
                               rj.data_ptr(), ld, dr.data_ptr(), ld, None)
    else:
        lib.te_lift_f64(h, ne, dfc.data_ptr(), ld, rj.data_ptr(), 0,
                        dr.data_ptr(), ld, None)
    torch.cuda.synchronize()
    got = _host(dr, npts, nv, ne)[:, 0]
    lib.te_destroy(h)

    top = np.abs(div).sum(1).max()
    bad = []
    for p in range(npts):
        terms, mid = [], False
        for d in range(nd):
            (l,), (i,) = np.nonzero(lines[d] == p)
            mid = mid or (q % 2 and i == q//2)
            if kernel != 'lift':
                terms += [(div[i, j], mom[d][k])
                          for j, k in enumerate(lines[d, l])]
            if kernel != 'gradflux':
                terms += [(div[i, q + e], fc[fpt[d, l, e], 0])
                          for e in range(2)]
        s, a, t = _sums(terms)
        c = 6 if (kernel, nd) == ('euler', 2) else \
            10 if mid and kernel != 'lift' else 4
        tol = np.maximum(c*top*t, (len(terms) + 2)*a)
        if kernel == 'lift':
            s, tol = s + old[p, 0], tol + 2*abs(old[p, 0])
        if kernel != 'gradflux':
            s = -s
        err = abs(got[p] - s)/(U*tol + 1e-300)
        assert np.all(np.isfinite(err))
        bad.append(float(err.max()))
    assert max(bad) <= 1.0, bad
