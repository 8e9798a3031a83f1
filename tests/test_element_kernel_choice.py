"""The choice between the element kernels and the general ones is made once, when
a system is committed: what an integrator does to the backend afterwards does
not change which kernels a right-hand side of another register pair has.  On
the library stand-in, no GPU."""

import pytest

from tests.fake_lib import FakeLib


@pytest.mark.parametrize('case', ['vortex', 'tgv'])
@pytest.mark.parametrize('before', [False, True])
def test_choice_is_made_at_commit(case, before, monkeypatch):
    from pyfr_gb300.backend import B200Backend
    from pyfr_gb300.backend import lib as liblib
    from pyfr_gb300.cases import euler_vortex, ns_tgv
    from pyfr_gb300.solvers.system import EulerSystem, NavierStokesSystem

    monkeypatch.setattr(liblib, '_LIB', FakeLib())
    cfg, mesh = euler_vortex(n=3) if case == 'vortex' else ns_tgv(n=2)
    cls = EulerSystem if case == 'vortex' else NavierStokesSystem
    be = B200Backend(cfg)
    if before:
        be.ref_state = (1.0, 71.4)
    s = cls(be, mesh, None, 3, cfg)
    s.commit()

    def names(uin, fout):
        return sorted(k.name or '' for g in s.rhs_graphs(uin, fout)
                      for k in g.klist)

    want = names(0, 1)
    assert any(n.startswith('te_') for n in want) == (not before)
    be.ref_state = None if before else (1.0, 71.4)
    assert names(1, 1) == want and names(2, 0) == want
