"""The cell integrals of the optimised step: the Taylor-Green source in each range
of cell sizes its cosines are expanded for, and the Persson marks on random data.

At rest and at uniform pressure the energy equation holds the source and what the
rounding of the coordinates leaves of the pressure forces; the same state without
a source (ncase 3) takes that off.  The source is a sum of 25 terms of products
of cosines, rounded at some 1e-15 of the largest on either side: 1e-11 leaves room
for a mesh near a zero of the source.  A mark is a comparison: none may differ
where the ratio is off the threshold by more than a rounding.
"""
import numpy as np
import pytest

from lag2d_b200.config import StepConfig
from lag2d_b200.mesh import quad_mesh
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h", [0.0004, 0.0011, 0.0013, 0.0075, 0.009, 0.17, 0.2, 0.5])
def test_source(h):
    """h: cell size; half of it is the distance the expansions are chosen by."""
    from lag2d_b200.api import Lag2DSolver
    m = quad_mesh(4, 3, 0.31, 0.31 + 4 * h, 0.11, 0.11 + 3 * h, jitter=0.1)
    got = []
    for ncase in (1, 3):
        c = StepConfig(ncase=ncase, gamlg=5.0 / 3.0, nstag=3, cfl=0.05, tend=10.0)
        s, o = Lag2DSolver(m, c), Oracle(m, c)
        geoel, amatr, u = s.init_fields()
        u[:] = 0.0
        u[:, 0, 0], u[:, 3, 0] = 1.0, 2.0
        us = np.zeros_like(m.coord)
        s.set_state(u, m.coord, us)
        ro, _ = o.rhs(us.copy(), u.copy(), geoel, m.coord, m.coord, amatr)
        got.append((s.rhs()[0][:m.ncell, 3], ro[:m.ncell, 3]))
    src, ref = got[0][0] - got[1][0], got[0][1] - got[1][1]
    assert np.abs(src - ref).max() < 1e-11 * np.abs(ref).max()


@pytest.mark.parametrize("shape", [(16, 8), (43, 5)])
def test_marks(shape):
    from lag2d_b200.api import Lag2DSolver
    m = quad_mesh(*shape, jitter=0.1, curve=0.05)
    c = StepConfig(ncase=1, gamlg=5.0 / 3.0, nstag=3, cfl=0.05, tend=10.0)
    s, o = Lag2DSolver(m, c), Oracle(m, c)
    geoel, amatr, u = s.init_fields()
    rng = np.random.default_rng(11)
    n = m.ncell
    size = 10.0 ** rng.uniform(-6.0, -1.0, n)
    u[:n, 0, 1:3] = 0.1 * rng.standard_normal((n, 2))
    u[:n, 0, 3:] = size[:, None] * rng.standard_normal((n, 3))
    i, j = np.arange(n) % shape[0], np.arange(n) // shape[0]
    u[:n, 0, 3:][(i == 0) | (i == shape[0] - 1) | (j == 0) | (j == shape[1] - 1)] = 0.0  # WENO rejects marked corners
    us = np.zeros_like(m.coord)
    s.set_state(u, m.coord, us)
    _, fo = o.rhs(us.copy(), u.copy(), geoel, m.coord, m.coord, amatr)
    _, marks = s.rhs()
    assert 0 < np.count_nonzero(fo[:n]) < n
    assert np.array_equal(marks[:n] != 0, np.asarray(fo)[:n] != 0)
