"""The block-per-quad WENO of the optimised step against the CPU restatement on
states in which every interior quad is marked: one quad, more quads than a
wave of blocks, odd sizes.

Tolerance: the reconstruction solves 5 x 5 systems whose matrices (products of
the scaled local basis, entries O(1)) have condition numbers up to ~1e4, the
Hermite ones as normal matrices up to its square; 1e8 * 2.2e-16 * ~25 terms is
5e-7 at worst and the mean candidate is three orders better, so 1e-8 of the
field's scale.
"""
import numpy as np
import pytest

from lag2d_b200.config import StepConfig
from lag2d_b200.mesh import quad_mesh
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(3, 3), (5, 4), (27, 23), (41, 37)])
def test_marked_quads(nx, ny):
    from lag2d_b200.api import Lag2DSolver
    m = quad_mesh(nx, ny, 0.0, 1.0, 0.0, 1.0, jitter=0.1, curve=0.05)
    c = StepConfig(ncase=1, gamlg=5.0 / 3.0, nstag=3, cfl=0.05, tend=10.0)
    s, o = Lag2DSolver(m, c), Oracle(m, c)
    geoel, amatr, u = s.init_fields()
    rng = np.random.default_rng(11)
    # tau moments of a few percent: far above the indicator's threshold in every quad
    # (not along the boundary, where the reference limits nothing)
    inner = np.zeros((ny, nx))
    inner[1:-1, 1:-1] = 1.0
    u[:m.ncell, 0, 3:] += 0.03 * rng.standard_normal((m.ncell, 3)) * inner.reshape(-1, 1)
    u[:m.ncell, 1:3] += 1.0e-2 * rng.standard_normal((m.ncell, 2, 6))
    us = np.zeros_like(m.coord)
    s.set_state(u, m.coord, us)
    uo = u.copy()
    Oracle.counts()
    _, fo = o.rhs(us.copy(), uo, geoel, m.coord, m.coord, amatr)
    marked, replaced = Oracle.counts()
    _, f = s.rhs()
    ug = s.get_state()[0]
    assert marked == replaced >= 0.99 * (nx - 2) * (ny - 2)
    assert np.array_equal(f, fo)
    n = m.ncell
    for q in range(4):
        assert np.abs(ug[:n, q] - uo[:n, q]).max() < 1e-8 * np.abs(uo[:n, q]).max()
