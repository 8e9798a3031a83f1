"""Right-hand sides and steps whose captured graph has branches (several element
types side by side, the flux beside the interfaces) against the same kernels one
after the other, bit for bit: a missing wait would show as another result."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _case(kinds, flow, prec):
    from pyfr_gb300.cases import euler_mixed

    cfg, mesh = euler_mixed(n=6, kinds=kinds, precision=prec)
    if flow == 'navier-stokes':
        cfg.set('solver', 'system', flow)
        cfg.set('constants', 'mu', '0.05')
        cfg.set('constants', 'Pr', '0.72')
        cfg.set('solver-interfaces', 'ldg-beta', '0.5')
        cfg.set('solver-interfaces', 'ldg-tau', '0.1')
        cfg.set('soln-ics', 'p', '10 + cos(x)*sin(y)')
    return cfg, mesh


@pytest.mark.parametrize('prec', ['double', 'single'])
@pytest.mark.parametrize('flow', ['euler', 'navier-stokes'])
@pytest.mark.parametrize('kinds', ['hex-pri', 'hex-pyr-tet', 'pri-tet'])
def test_branches_equal_the_serial_order(kinds, flow, prec):
    from pyfr_gb300.backend import B200Backend
    from pyfr_gb300.integrators import MixedRKIntegrator, RKVdH2Integrator
    from pyfr_gb300.solvers.system import EulerSystem, NavierStokesSystem

    cls = EulerSystem if flow == 'euler' else NavierStokesSystem
    icls = RKVdH2Integrator if prec == 'double' else MixedRKIntegrator
    got = []
    for graphs in (True, False):
        cfg, mesh = _case(kinds, flow, prec)
        cfg.set('backend-b200', 'cuda-graphs', str(graphs).lower())
        it = icls(B200Backend(cfg), cls, mesh, cfg)
        assert it.use_step_graph == graphs
        assert (it.step_nodes(0, it.dt) is not None) or not graphs
        it.system.rhs(0.0, 0, 1)
        it.backend.wait()
        out = [a.copy() for a in it.system.ele_scal_upts(1)]
        it.run_steps(3)
        it.backend.wait()
        got.append(out + [np.array(a) for a in it.soln])
    assert all(np.all(np.isfinite(a)) for a in got[0])
    assert all(np.array_equal(a, b) for a, b in zip(*got))
