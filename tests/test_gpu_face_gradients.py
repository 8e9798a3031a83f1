"""Face gradients that reach the interface kernel in reference space (single
precision, every element affine, no boundaries): the right-hand side against
FP64's and against the one with the gradients transformed at the points.

The viscosity is large enough (0.1, gradients of 0.3 noise) that the
interfaces' viscous flux is some percent of the largest value, so gradients
that are not transformed show.  Bounds: FP32 inputs of the pressure (71 against
fluctuations of 1) carry 178 2^-24 = 1e-5 of the fluctuations, which the
derivative and lift matrices' row sums (at most about 50 at p = 4, a tenth of
it in the mean) take below 2e-4 of the largest; of the two FP32 forms each
other's roundings alone, within the same.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rhs(nd, order, n, shear, beta, prec, kernels, facegrad):
    from pyfr_gb300.backend import B200Backend
    from pyfr_gb300.cases import ns_tgv
    from pyfr_gb300.mesh import periodic_box
    from pyfr_gb300.solvers.system import NavierStokesSystem

    et = {2: 'quad', 3: 'hex'}[nd]
    cfg, _ = ns_tgv(n=2, order=order, precision=prec, beta=beta)
    cfg.set('constants', 'mu', '0.1')
    cfg.set('solver-interfaces-line', 'flux-pts', 'gauss-legendre')
    cfg.set('solver-elements-quad', 'soln-pts', 'gauss-legendre')
    cfg.set('backend-b200', 'element-kernels', kernels)
    cfg.set('backend-b200', 'face-gradients', facegrad)
    mesh = periodic_box(et, n, -np.pi, np.pi)
    mesh.spts[et][..., 0] += shear*mesh.spts[et][..., 1]

    rng = np.random.default_rng(5)
    ne, nu = mesh.spts[et].shape[1], (order + 1)**nd
    v = 0.3*rng.standard_normal((nd, nu, ne))
    rho = 1 + 0.01*rng.standard_normal((nu, ne))
    p = 71.4 + rng.standard_normal((nu, ne))
    u = np.stack([rho, *(rho*v), p/0.4 + 0.5*rho*(v*v).sum(0)], axis=1)
    s = NavierStokesSystem(B200Backend(cfg), mesh, {et: u}, 2, cfg)
    s.commit()
    s.rhs(0.0, 0, 1)
    s.backend.wait()
    return s.ele_scal_upts(1)[0]


@pytest.mark.parametrize('kernels', ['auto', 'general'])
@pytest.mark.parametrize('beta', [0.5, -0.5, 0.0])
@pytest.mark.parametrize('shear', [0.0, 0.3])
@pytest.mark.parametrize('nd,order,n', [(2, 1, (3, 5)), (2, 2, (33, 2)),
                                        (2, 3, 6), (2, 4, 3), (3, 3, 3)])
def test_reference_space_face_gradients(nd, order, n, shear, beta, kernels):
    a = _rhs(nd, order, n, shear, beta, 'single', kernels, 'auto')
    b = _rhs(nd, order, n, shear, beta, 'single', kernels, 'physical')
    c = _rhs(nd, order, n, shear, beta, 'double', 'general', 'auto')
    for q in range(c.shape[1]):
        top = np.abs(c[:, q]).max()
        assert np.abs(a[:, q] - b[:, q]).max() <= 2e-4*top
        assert np.abs(a[:, q] - c[:, q]).max() <= 2e-4*top
