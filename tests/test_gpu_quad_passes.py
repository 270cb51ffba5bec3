"""The quad passes of the optimised step around their block sizes against the CPU
restatement: corner faces, node solve and RHS on random data, and one whole step
(the RHS pass with its update, with and without U^n; full degree).

Tolerance: as for the triangle passes, about 100 terms that cancel by up to four
digits: 100 * 2.2e-16 * 1e4 = 2e-10 of the field's scale; the step adds dt M^-1 of
that to the state, less than the same of it.
"""
import numpy as np
import pytest

from lag2d_b200.config import StepConfig
from lag2d_b200.mesh import quad_mesh
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(31, 1), (8, 4), (11, 3), (9, 7), (16, 4), (13, 5), (43, 3)])
@pytest.mark.parametrize("mdegr,nstag", [(6, 3), (6, 2), (3, 2)])
def test_rhs_and_step(shape, mdegr, nstag):
    from lag2d_b200.api import Lag2DSolver
    m = quad_mesh(*shape, jitter=0.1, curve=0.05)
    c = StepConfig(ncase=1, gamlg=5.0 / 3.0, nstag=nstag, cfl=0.02, tend=10.0, mdegr=mdegr)
    s, o = Lag2DSolver(m, c), Oracle(m, c)
    geoel, amatr, u = s.init_fields()
    rng = np.random.default_rng(3)
    n = m.ncell
    u[:n, :, 0] *= 1.0 + 1.0e-3 * rng.standard_normal((n, 4))
    us = 0.1 * rng.standard_normal(m.coord.shape)
    s.set_state(u, m.coord, us)
    uo, uso = u.copy(), us.copy()
    ro, _ = o.rhs(uso, uo, geoel, m.coord, m.coord, amatr)
    r, _ = s.rhs()
    assert np.abs(s.get_state()[2] - uso).max() < 2e-11 * np.abs(uso).max()
    for q in range(4):
        assert np.abs(r[:n, q] - ro[:n, q]).max() < 2e-10 * np.abs(ro[:n, q]).max()
    if mdegr < 6:
        return  # the restatement's step truncates elsewhere than the RHS
    s.set_state(u, m.coord, us)
    x, uso = m.coord.copy(), us.copy()
    _, dt, _ = o.run(u, x, m.coord, geoel, amatr, uso, 1, 1, c.dtfix, 0.0)
    s.step()
    u2, x2, us2, _ = s.get_state()
    assert abs(s.dtfix - dt) <= 2e-11 * dt
    for q in range(4):
        assert np.abs(u2[:n, q] - u[:n, q]).max() < 2e-10 * np.abs(u[:n, q]).max()
    assert np.abs(x2 - x).max() < 2e-11 and np.abs(us2 - uso).max() < 2e-10 * np.abs(uso).max()
