"""The node partial sums of the optimised step: three rows a node in FP64, five in
the FP32-mixed step, on quads and triangles.  One RHS of each against the
restatement, on a mesh with every kind of node (corner, edge, centre, shared by
triangles and quads, walls).

Tolerance: u* is a quotient of sums of about 16 positive terms, m u and sigma.n A
cancelling by up to three digits: 100 * 2.2e-16 * 1e3 = 2e-11 of the field; the
FP32-mixed sums carry 6e-8 instead, 100 * 6e-8 * 1e1.
"""
import numpy as np
import pytest

from lag2d_b200.config import StepConfig
from lag2d_b200.mesh import hybrid_mesh, quad_mesh
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["quads", "hybrid"])
@pytest.mark.parametrize("precision,tol", [(0, 2e-11), (1, 6e-5)])
def test_node_velocity(kind, precision, tol):
    from lag2d_b200.api import Lag2DSolver
    m = quad_mesh(5, 3, jitter=0.05) if kind == "quads" else hybrid_mesh(7, 5, 0.0, 1.0, 0.0, 1.0, jitter=0.05)
    c = StepConfig(ncase=1, gamlg=5.0 / 3.0, nstag=3, cfl=0.05, tend=10.0)
    s, o = Lag2DSolver(m, c, precision=precision), Oracle(m, c)
    geoel, amatr, u = s.init_fields()
    us = 0.1 * np.random.default_rng(5).standard_normal(m.coord.shape)
    s.set_state(u, m.coord, us)
    uo, uso = u.copy(), us.copy()
    ro, _ = o.rhs(uso, uo, geoel, m.coord, m.coord, amatr)
    r, _ = s.rhs()
    assert np.abs(s.get_state()[2] - uso).max() < tol * np.abs(uso).max()
    n = m.ncell
    for q in range(4):
        assert np.abs(r[:n, q] - ro[:n, q]).max() < 10.0 * tol * np.abs(ro[:n, q]).max()
