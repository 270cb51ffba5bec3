"""The sub-cell density corrections of a quad that WENO replaces come from its limited
moments alone: one step on states whose raw tau passes zero (to rounding) along a row of
sub-cell Gauss points of a marked quad, against the CPU restatement, which limits first.

Tolerance: that of the reconstruction itself, 1e-8 of the field's scale.
"""
import numpy as np
import pytest

from lag2d_b200.config import StepConfig, workload
from lag2d_b200.mesh import quad_mesh
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu

G = 0.9061798459386639927976269


def _compare(m, c, u, geoel, amatr, s, o, tol):
    us = np.zeros_like(m.coord)
    s.set_state(u, m.coord, us)
    x = m.coord.copy()
    _, dt, _ = o.run(u, x, m.coord, geoel, amatr, us, 1, 1, c.dtfix, 0.0)
    s.step()
    ug, xg, vg, _ = s.get_state()
    n = m.ncell
    assert abs(s.dtfix - dt) <= tol * dt
    for q in range(4):
        assert np.abs(ug[:n, q] - u[:n, q]).max() < tol * np.abs(u[:n, q]).max()
    assert np.abs(xg - x).max() < tol and np.abs(vg - us).max() < tol * np.abs(us).max()


@pytest.mark.parametrize("r0", [0.5 * (G + 1.0), 0.5, -0.5, -0.5 * (G + 1.0)])
@pytest.mark.parametrize("along", [0, 1])  # the row lies across r or across s
def test_raw_tau_through_zero(r0, along):
    from lag2d_b200.api import Lag2DSolver
    m = quad_mesh(7, 7, jitter=0.05)
    c = StepConfig(ncase=1, gamlg=5.0 / 3.0, nstag=3, cfl=0.05, tend=10.0)
    s, o = Lag2DSolver(m, c), Oracle(m, c)
    geoel, amatr, u = s.init_fields()
    e, t3 = 24, 0.3
    c0, g = geoel[e, along], geoel[e, 18 + along]
    tau = u[e, 0, 0]
    u[e, 0, 1:] = 0.0
    u[e, 0, 3 + along] = t3
    u[e, 0, 1 + along] = -(tau + t3 * (0.5 * (r0 - c0) ** 2 - g)) / (r0 - c0)
    Oracle.counts()
    _compare(m, c, u, geoel, amatr, s, o, 1e-8)
    assert Oracle.counts()[1] >= 1  # replaced


def test_blast():
    from lag2d_b200.api import Lag2DSolver
    m, c = workload("sedov16")
    s, o = Lag2DSolver(m, c), Oracle(m, c)
    geoel, amatr, u = s.init_fields()
    _compare(m, c, u, geoel, amatr, s, o, 1e-8)
