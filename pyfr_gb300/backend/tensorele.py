"""Element kernels of tensor-product elements (``csrc/tensor_ele.cu``): the
operator applies and pointwise kernels of one element in one launch, the
operators applied line by line.

``te_interp`` takes the place of ``disu``; ``te_gradflux`` that of
``tgradpcoru_upts``, ``tgradcoru_upts``, ``tdisf_fused``, ``gradcoru_fpts`` and
``tdivtpcorf``; ``te_lift`` that of ``tdivtconf`` and ``negdivconf``; and
``te_euler`` that of ``tdisf``, ``tdivtpcorf``, ``tdivtconf`` and ``negdivconf``
(``pyfr/solvers/baseadvec/elements.py:91-120``,
``pyfr/solvers/baseadvecdiff/elements.py:47-116``).
"""

import ctypes as C
import weakref

import numpy as np

from pyfr_gb300.backend.types import Kernel


def _line_points(nd, q):
    """Point indices (nd, q**(nd - 1), q) of the lines of each direction,
    the first coordinate being the fastest; lines in the order of their
    first point."""
    p = np.arange(q**nd).reshape((q,)*nd)
    return np.stack([np.moveaxis(p, nd - 1 - d, -1).reshape(-1, q)
                     for d in range(nd)])


def _gauss_line(q):
    """The line matrices (grad, interp, div) of q Gauss-Legendre points in
    extended precision: the full operators' entries carry a few roundings of
    their own, alike on every line, which differentiating a large mean
    (pressure, energy) shows; these are rounded once."""
    ld = np.longdouble
    x = np.polynomial.legendre.leggauss(q)[0].astype(ld)

    def legendre(t):
        p0, p1 = np.ones_like(t), t
        for k in range(1, q):
            p0, p1 = p1, ((2*k + 1)*t*p1 - k*p0)/(k + 1)
        return p1, q*(t*p1 - p0)/(t*t - 1)

    for _ in range(3):
        p, dp = legendre(x)
        x = x - p/dp
    dp = legendre(x)[1]
    w = 2/((1 - x*x)*dp*dp)
    b = np.array([1/np.prod(x[j] - np.delete(x, j)) for j in range(q)])
    D = np.zeros((q, q), dtype=ld)
    for i in range(q):
        for j in range(q):
            if i != j:
                D[i, j] = b[j]/b[i]/(x[i] - x[j])
        D[i, i] = -D[i].sum()
    lo, hi = (np.array([np.prod(e - np.delete(x, j))*b[j] for j in range(q)])
              for e in (ld(-1), ld(1)))
    # (correction by the lift of both ends; the common solution enters the
    # gradient, the outward common flux the divergence)
    own = D - np.outer(hi/w, hi) + np.outer(lo/w, lo)
    if q % 2:
        own[q//2, q//2] = 0
    lift = np.stack([lo/w, hi/w], axis=1)
    return [a.astype(np.float64)
            for a in (np.hstack([own, lift*[-1, 1]]), np.stack([lo, hi]),
                      np.hstack([own, lift]))]


def line_operators(nd, q, m0, m132, m3, m460=None, m6=None, tol=1e-12):
    """The one-dimensional matrices (grad, interp, div) and the flux points
    (nd, lines, 2) of operators that are products of them, or None where the
    given ones are not (to ``tol`` of each operator's largest entry)."""
    nu, nl, nf = q**nd, q**(nd - 1), 2*nd*q**(nd - 1)
    if m0.shape != (nf, nu) or nd not in (2, 3) or not 3 <= q <= 5:
        return None
    lines = _line_points(nd, q)

    # The two flux points of a line are those that interpolate from its
    # points alone; the low end's largest coefficient is the first point's
    on = np.abs(m0) > tol*np.abs(m0).max()
    rows = {}
    for f in range(nf):
        rows.setdefault(tuple(np.flatnonzero(on[f])), []).append(f)
    fpt = np.empty((nd, nl, 2), dtype=np.int32)
    for d in range(nd):
        for l in range(nl):
            fs = rows.get(tuple(sorted(lines[d, l])), [])
            if len(fs) != 2:
                return None
            lead = [np.argmax(np.abs(m0[f, lines[d, l]])) for f in fs]
            if sorted(lead) != [0, q - 1]:
                return None
            fpt[d, l] = fs if lead[0] == 0 else fs[::-1]

    l0, f0 = lines[0, 0], fpt[0, 0]
    interp = m0[np.ix_(f0, l0)]
    div = np.hstack([m132[np.ix_(l0, l0)], m3[np.ix_(l0, f0)]])
    grad = np.zeros((q, q + 2)) if m460 is None else \
        np.hstack([m460[np.ix_(l0, l0)], m6[np.ix_(l0, f0)]])

    # Gauss-Legendre lines: the same matrices, rounded once
    for m, g in zip((grad, interp, div), _gauss_line(q)):
        if np.any(m) and np.abs(m - g).max() <= tol*np.abs(m).max():
            m[...] = g

    # (an odd line's middle point is no part of its own derivative)
    for m in (grad, div):
        c = q//2
        if q % 2 and abs(m[c, c]) <= tol*np.abs(m).max():
            m[c, c] = 0.0
        elif q % 2:
            return None

    full = dict(m0=np.zeros_like(m0), m132=np.zeros_like(m132),
                m3=np.zeros_like(m3))
    if m460 is not None:
        full |= dict(m460=np.zeros_like(m460), m6=np.zeros_like(m6))
    for d in range(nd):
        for l in range(nl):
            p, f = lines[d, l], fpt[d, l]
            full['m0'][np.ix_(f, p)] = interp
            full['m132'][np.ix_(p, d*nu + p)] = div[:, :q]
            full['m3'][np.ix_(p, f)] = div[:, q:]
            if m460 is not None:
                full['m460'][np.ix_(d*nu + p, p)] = grad[:, :q]
                full['m6'][np.ix_(d*nu + p, f)] = grad[:, q:]
    given = dict(m0=m0, m132=m132, m3=m3, m460=m460, m6=m6)
    if any(np.abs(full[k] - given[k]).max() > tol*np.abs(given[k]).max()
           for k in full):
        return None
    return grad, interp, div, fpt


class TensorElementKernels:
    def __init__(self, backend):
        from pyfr_gb300.backend.base import release
        self.backend = backend
        self._handles = {}
        weakref.finalize(self, release, self._destroy,
                         backend.lib.te_destroy, self._handles)

    @staticmethod
    def _destroy(destroy, handles):
        for h in handles.values():
            if h is not None:
                destroy(h[0])
        handles.clear()

    def handle(self, basis, viscous):
        """(handle, flux points of the lines) of a shape's operators, or
        None where they are not products of line matrices that the kernels
        are built for."""
        key = (basis.name, basis.order, basis.upts.tobytes(),
               basis.fpts.tobytes(), viscous)
        if key not in self._handles:
            nd, q = basis.ndims, basis.order + 1
            self._handles[key] = None
            if basis.name in ('quad', 'hex') and basis.nupts == q**nd:
                ops = line_operators(
                    nd, q, basis.m0, basis.opmat('M1 - M3*M2'), basis.m3,
                    *((basis.opmat('M4 - M6*M0'), basis.m6)
                      if viscous else ()))
                if ops is not None:
                    *mats, fpt = ops
                    mats = [np.ascontiguousarray(m, dtype=np.float64)
                            for m in mats]
                    pd = C.POINTER(C.c_double)
                    h = C.c_void_p()
                    if not viscous:
                        # (te_create asks for a derivative matrix)
                        mats[0] = mats[2]
                    self.backend.lib.te_create(
                        nd, q, *(m.ctypes.data_as(pd) for m in mats),
                        fpt.ctypes.data_as(C.POINTER(C.c_int)), C.byref(h))
                    self._handles[key] = (h.value, fpt)
        return self._handles[key]

    def _fn(self, name):
        sfx = 'f64' if self.backend.fpdtype == np.float64 else 'f32'
        return getattr(self.backend.lib, f'te_{name}_{sfx}')

    def te_interp(self, handle, u, out, neles):
        fn, h = self._fn('interp'), handle
        args = (neles, u.data, u.leaddim, out.data, out.leaddim)

        def run(stream):
            fn(h, *args, stream)

        return Kernel(run, mats=[u, out], name='te_interp',
                      meta=dict(kind='te_interp', u=u, out=out))

    def te_gradflux(self, handle, tplargs, neles, u, comm, gradf, facemask, r,
                    geom, refgrad=False):
        from pyfr_gb300.backend.pointwise import _gas
        lin, (sp, sl), (rp, rl), _, _ = geom
        gas = _gas(tplargs['c'], tplargs.get('visc_corr', 'none'))
        fn, h = self._fn('gradflux_ns'), handle
        args = (u.data, u.leaddim, comm.data, comm.leaddim, gradf.data,
                gradf.leaddim, facemask, int(refgrad), sp, sl, rp, rl, r.data, r.leaddim)

        def run(stream):
            fn(h, neles, lin, C.byref(gas), *args, stream)

        return Kernel(run, mats=[u, comm, gradf, r], misc=[gas],
                      name='te_gradflux',
                      meta=dict(kind='te_gradflux', tplargs=tplargs, u=u,
                                comm=comm, gradf=gradf, r=r,
                                geom_mode=lin, facemask=facemask))

    def te_euler(self, handle, tplargs, neles, u, fc, r, geom):
        lin, (sp, sl), (rp, rl), _, _ = geom
        fn, h = self._fn('euler'), handle
        gamma = tplargs['c']['gamma']
        args = (u.data, u.leaddim, fc.data, fc.leaddim, sp, sl, rp, rl,
                r.data, r.leaddim)

        def run(stream):
            fn(h, neles, lin, gamma, *args, stream)

        return Kernel(run, mats=[u, fc, r], name='te_euler',
                      meta=dict(kind='te_euler', tplargs=tplargs, u=u, fc=fc, r=r,
                                geom_mode=lin))

    def te_lift(self, handle, tplargs, neles, fc, r, geom):
        lin, _, (rp, rl), _, _ = geom
        fn, h = self._fn('lift'), handle
        # (one 1/|J| per element: every point reads the same row)
        args = (neles, fc.data, fc.leaddim, rp, rl if lin == 0 else 0, r.data,
                r.leaddim)

        def run(stream):
            fn(h, *args, stream)

        return Kernel(run, mats=[fc, r], name='te_lift',
                      meta=dict(kind='te_lift', fc=fc, r=r))
