"""The triangle passes of the optimised step against the CPU restatement: sizes
around the block of 64 triangles, a stretched and a curved mesh, mdegr below
ndegr, and the recorded corner coefficients of the adjoint.

Tolerance: the RHS is a sum of about 100 terms that cancel by up to four digits
(the tau equation), so 100 * 2.2e-16 * 1e4 = 2e-10 of the field's scale.
"""
import numpy as np
import pytest

from lag2d_b200.config import StepConfig
from lag2d_b200.mesh import hybrid_mesh, polar_mesh
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


def _mesh(kind):
    if kind == "polar":
        return polar_mesh(6, 5, 1.0), 3
    nx, ny, jit, curve = {"one block": (16, 4, 0.0, 0.0), "one more": (33, 2, 0.0, 0.0), "curved": (17, 12, 0.1, 0.05),
                          "flat": (70, 3, 0.05, 0.0)}[kind]
    return hybrid_mesh(nx, ny, 0.0, 1.0, 0.0, 0.3 if kind == "flat" else 1.0, jitter=jit, curve=curve), 1


@pytest.mark.parametrize("kind", ["one block", "one more", "curved", "flat", "polar"])
@pytest.mark.parametrize("mdegr", [6, 3])
def test_rhs(kind, mdegr):
    from lag2d_b200.api import Lag2DSolver
    m, ncase = _mesh(kind)
    c = StepConfig(ncase=ncase, gamlg=5.0 / 3.0, nstag=3, cfl=0.05, tend=10.0, mdegr=mdegr)
    s, o = Lag2DSolver(m, c), Oracle(m, c)
    geoel, amatr, u = s.init_fields()
    rng = np.random.default_rng(3)
    n, nt = m.ncell, m.ntria
    u[:nt] *= 1.0 + 1.0e-3 * rng.standard_normal((nt, 4, 1))
    us = 0.1 * rng.standard_normal(m.coord.shape)
    s.set_state(u, m.coord, us)
    uo, uso = u.copy(), us.copy()
    ro, _ = o.rhs(uso, uo, geoel, m.coord, m.coord, amatr)
    r, _ = s.rhs()
    assert np.abs(s.get_state()[2] - uso).max() < 1e-11 * np.abs(uso).max()
    for q in range(4):
        assert np.abs(r[:nt, q] - ro[:nt, q]).max() < 2e-10 * np.abs(ro[:n, q]).max()
