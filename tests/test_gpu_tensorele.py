"""Element kernels of tensor-product elements (``csrc/tensor_ele.cu``) against
the operator applies and pointwise kernels that they take the place of
(``element-kernels = general``), and the host's recognition of their operators.

Both sides are sums of the same products in another order: with the derivative
and lift matrices' row sums (at most about 50 at p = 4) two passes of rounding
stay below 1e-12 of the right-hand side's largest value in FP64 when the
pressure (71 against fluctuations of 1) is differentiated, and below 2e-4 in
FP32."""

import numpy as np
import pytest

from pyfr_gb300.backend.tensorele import line_operators
from pyfr_gb300.shapes import get_shape


@pytest.mark.parametrize('name', ['quad', 'hex'])
@pytest.mark.parametrize('order', [1, 2, 3, 4, 5])
def test_line_operators(name, order):
    b = get_shape(name, order)
    ops = line_operators(b.ndims, order + 1, b.m0, b.opmat('M1 - M3*M2'),
                         b.m3, b.opmat('M4 - M6*M0'), b.m6)
    assert (ops is not None) == (2 <= order <= 4)
    if ops:
        grad, interp, div, fpt = ops
        # Exact on the line's polynomials, the common solution being the
        # interpolated one
        x = b.upts[:order + 1, 0]
        for k in range(order + 1):
            ends = np.array([(-1.0)**k, 1.0])
            assert np.allclose(interp @ x**k, ends, atol=1e-12)
            d = k*x**max(k - 1, 0)
            full = np.concatenate([x**k, ends])
            assert np.allclose(grad @ full, d, atol=1e-11)
            # (outward: the low end's normal flux is minus the flux)
            full[-2] *= -1
            assert np.allclose(div @ full, d, atol=1e-11)
        assert sorted(fpt.ravel()) == list(range(b.nfpts))


def test_line_operators_refused():
    """Operators that are not products of line matrices are left to the
    general kernels."""
    b = get_shape('hex', 3, 'gauss-legendre-lobatto', 'gauss-legendre-lobatto')
    ops = [b.m0, b.opmat('M1 - M3*M2'), b.m3, b.opmat('M4 - M6*M0'), b.m6]
    assert line_operators(3, 4, *ops) is None
    b = get_shape('hex', 3)
    ops = [b.m0, b.opmat('M1 - M3*M2'), b.m3, b.opmat('M4 - M6*M0'), b.m6]
    for i in range(5):
        bad = [o.copy() for o in ops]
        bad[i][3, 5] += 1e-6
        assert line_operators(3, 4, *bad) is None


def _system(nd, flow, order, n, prec, mesh_form, beta, rs, kernels):
    from pyfr_gb300.backend import B200Backend
    from pyfr_gb300.cases import euler_vortex, ns_tgv
    from pyfr_gb300.mesh import periodic_box
    from pyfr_gb300.solvers.system import EulerSystem, NavierStokesSystem

    cfg, mesh = ns_tgv(n=2, order=order, precision=prec, beta=beta, rsolver=rs)
    et = {2: 'quad', 3: 'hex'}[nd]
    if nd == 2:
        cfg.set('solver-interfaces-line', 'flux-pts', 'gauss-legendre')
        cfg.set('solver-elements-quad', 'soln-pts', 'gauss-legendre')
    cfg.set('backend-b200', 'element-kernels', kernels)
    mesh = periodic_box(et, n, -np.pi, np.pi)
    x = mesh.spts[et]
    if mesh_form == 'sheared':
        x[..., 0] += 0.3*x[..., 1]
    elif mesh_form == 'bent':
        y = x.copy()
        x[..., 0] += 0.2*np.sin(y[..., 1])
        x[..., 1] += 0.2*np.sin(y[..., 0])
    cls = EulerSystem if flow == 'euler' else NavierStokesSystem

    rng = np.random.default_rng(11)
    ne = x.shape[1]
    nu = (order + 1)**nd
    v = 0.3*rng.standard_normal((nd, nu, ne))
    rho = 1 + 0.01*rng.standard_normal((nu, ne))
    p = 71.4 + rng.standard_normal((nu, ne))
    u = np.stack([rho, *(rho*v), p/0.4 + 0.5*rho*(v*v).sum(0)], axis=1)
    return cls(B200Backend(cfg), mesh, {et: u}, 2, cfg)


@pytest.mark.gpu
@pytest.mark.parametrize('prec,tol', [('double', 1e-12), ('single', 2e-4)])
@pytest.mark.parametrize('nd,order,n', [
    (2, 2, 5), (2, 3, (33, 1)), (2, 4, 6), (3, 2, (3, 11, 1)), (3, 3, 3),
    (3, 4, (2, 3, 1))])
@pytest.mark.parametrize('flow,mesh_form,beta,rs', [
    ('euler', 'uniform', 0.5, 'rusanov'), ('euler', 'bent', 0.5, 'hllc'),
    ('ns', 'uniform', 0.5, 'rusanov'), ('ns', 'sheared', -0.5, 'rusanov'),
    ('ns', 'bent', 0.0, 'hllc')])
def test_element_kernels(nd, order, n, flow, mesh_form, beta, rs, prec, tol):
    got = {}
    for kernels in ('auto', 'general'):
        s = _system(nd, flow, order, n, prec, mesh_form, beta, rs, kernels)
        s.commit()
        names = {k.name or '' for g in s.rhs_graphs(0, 1)
                 for k in g.klist}
        assert any(x.startswith('te_') for x in names) == (kernels == 'auto')
        s.rhs(0.0, 0, 1)
        s.backend.wait()
        a = s.ele_scal_upts(1)[0]
        # (onto its own input, as the integrator's later stages do)
        s.rhs(0.0, 0, 0)
        s.backend.wait()
        assert np.array_equal(s.ele_scal_upts(0)[0], a)
        got[kernels] = a
    a, b = got['auto'], got['general']
    assert np.all(np.isfinite(b))
    for q in range(a.shape[1]):
        assert np.abs(a[:, q] - b[:, q]).max() <= tol*np.abs(b[:, q]).max()


@pytest.mark.gpu
@pytest.mark.parametrize('flow', ['euler', 'ns'])
def test_element_kernels_special_values(flow):
    """A NaN, an infinity, zeros and values at the ends of the exponent range
    reach the same values of the right-hand side through both kernels, and
    no others."""
    got = {}
    for kernels in ('auto', 'general'):
        s = _system(3, flow, 3, 4, 'double', 'uniform', 0.5, 'rusanov',
                    kernels)
        s.commit()
        (u,) = s.ele_scal_upts(0)
        u[:, 1:4, 10] = 0.0
        u[:, 2, 20] *= 1e-310
        u[5, 0, 40] = np.nan
        u[7, 4, 55] = np.inf
        s.set_ele_scal_upts(0, [u])
        s.rhs(0.0, 0, 1)
        s.backend.wait()
        got[kernels] = s.ele_scal_upts(1)[0]
    a, b = got['auto'], got['general']
    fin = np.isfinite(b)
    assert 0 < fin.sum() < fin.size
    assert np.array_equal(np.isfinite(a), fin)
    assert np.abs(a - b)[fin].max() <= 1e-12*np.abs(b[fin]).max()


@pytest.mark.gpu
@pytest.mark.parametrize('mesh_form', ['uniform', 'sheared', 'bent'])
@pytest.mark.parametrize('flow', ['euler', 'ns'])
def test_element_kernels_without_host_geometry(flow, mesh_form, monkeypatch):
    """The set-up of a large mesh drops the host copies of its vertices, and
    a right-hand side's kernels are made after that: the same bits as with
    the copies kept."""
    from pyfr_gb300.backend import base

    got = []
    for keep in (base.HOST_KEEP, 50):
        monkeypatch.setattr(base, 'HOST_KEEP', keep)
        s = _system(3, flow, 3, 3, 'double', mesh_form, 0.5, 'rusanov',
                    'auto')
        s.commit()
        names = {k.name or '' for g in s.rhs_graphs(0, 1) for k in g.klist}
        assert any(x.startswith('te_') for x in names)
        s.rhs(0.0, 0, 1)
        s.rhs(0.0, 0, 0)
        s.backend.wait()
        got.append([s.ele_scal_upts(i)[0] for i in (0, 1)])
    assert all(np.array_equal(a, b) for a, b in zip(*got))
