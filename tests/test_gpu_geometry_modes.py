"""The element kernels' forms of the metric terms against one another on a
mesh that all of them take (a uniform box: per point, per element, diagonal),
and on a sheared one that the diagonal form has to decline.

The forms differ by rounding alone: each output is a sum of a few hundred
products of one FP64 (FP32) rounding each, so 1e-12 (1e-5 in FP32, where the
pressure terms of Ma = 0.1 cancel to a hundredth) of the largest is
allowed."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rhs(nd, flow, prec, per_ele, shear):
    from pyfr_gb300.backend import B200Backend
    from pyfr_gb300.cases import euler_vortex, ns_tgv
    from pyfr_gb300.solvers.system import EulerSystem, NavierStokesSystem

    if flow == 'ns':
        cfg, mesh = ns_tgv(n=5, order=2, precision=prec)
        cls = NavierStokesSystem
    else:
        cfg, mesh = euler_vortex(n=7, order=3, precision=prec)
        cls = EulerSystem
    cfg.set('backend-b200', 'per-element-metrics', str(per_ele).lower())
    (et,) = mesh.spts
    mesh.spts[et][..., 0] += shear*mesh.spts[et][..., 1]
    s = cls(B200Backend(cfg), mesh, None, 2, cfg)
    s.commit()
    modes = {k.meta['geom_mode'] for g in s.rhs_graphs(0, 1) for k in g.klist
             if 'geom_mode' in getattr(k, 'meta', {})}
    s.rhs(0.0, 0, 1)
    s.backend.wait()
    return s.ele_scal_upts(1)[0], modes


@pytest.mark.parametrize('prec,tol', [('double', 1e-12), ('single', 1e-5)])
@pytest.mark.parametrize('nd,flow', [(2, 'euler'), (3, 'ns')])
@pytest.mark.parametrize('shear', [0.0, 1e-9, 0.25])
def test_metric_forms_agree(nd, flow, prec, tol, shear):
    a, ma = _rhs(nd, flow, prec, True, shear)
    b, mb = _rhs(nd, flow, prec, False, shear)
    assert ma == {2 if shear else 3} and mb == {0}
    assert np.all(np.isfinite(a))
    assert np.abs(a - b).max() <= tol*np.abs(b).max()
