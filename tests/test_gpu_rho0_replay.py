"""A density set after a handle has stepped reaches its later steps and adjoint windows:
on states whose interior quads WENO replaces (it weighs its stencils by the initial
density) they give the bits of a handle that had the density from the start, in both
directions, step by step, in runs and with checkpoints."""
import numpy as np
import pytest

from lag2d_b200.config import StepConfig
from lag2d_b200.mesh import quad_mesh

pytestmark = pytest.mark.gpu


def _renew(s, m, rho0):
    s.set_rho0(rho0)
    geoel, amatr, u = s.init_fields()
    rng = np.random.default_rng(11)
    inner = np.zeros((7, 9))
    inner[1:-1, 1:-1] = 1.0
    u[:m.ncell, 0, 3:] += 0.01 * rng.standard_normal((m.ncell, 3)) * inner.reshape(-1, 1)
    s.set_state(u, m.coord, np.zeros_like(m.coord))


def _advance(s, call):
    if call == "step":
        s.step()
        s.step()
    elif call == "run":
        s.run(2)
    else:
        return s.adjoint(3, 2)[:4] + s.get_state() + (s.dtfix, s.tacru)
    return s.get_state() + (s.dtfix, s.tacru)


@pytest.mark.parametrize("call,exact", [("step", False), ("run", False), ("adjoint", False), ("step", True), ("run", True)])
@pytest.mark.parametrize("back", [False, True])
def test_density_after_steps(call, back, exact):
    from lag2d_b200.api import Lag2DSolver
    m = quad_mesh(9, 7, 0.0, 1.0, 0.0, 1.0, jitter=0.1, curve=0.05)
    c = StepConfig(ncase=1, gamlg=5.0 / 3.0, nstag=3, cfl=0.02, tend=10.0)
    x = m.coord[m.ipqua[:, 8] - 1]
    rho0 = 1.0 + 0.5 * np.sin(4.0 * x[:, 0]) * np.cos(3.0 * x[:, 1])
    first, then = (rho0, None) if back else (None, rho0)
    used, fresh = Lag2DSolver(m, c, order_exact=exact), Lag2DSolver(m, c, order_exact=exact)
    _renew(used, m, first)
    _advance(used, call)
    _renew(used, m, then)
    _renew(fresh, m, then)
    assert np.count_nonzero(fresh.rhs()[1]) > 20  # troubled quads there are
    _renew(fresh, m, then)
    for a, b in zip(_advance(used, call), _advance(fresh, call)):
        assert np.array_equal(a, b)
