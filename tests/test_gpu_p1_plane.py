"""The plane linear branch runs one arithmetic on meshes of every size: cells and nodes
near the lower wall of a strip that does not vary along y get the same bits on a
mesh of 64 x 40 cells and on one of 64 x 1024 (65,536 cells), as long as the upper wall is
out of reach.

A stage reaches two cells far (the limited states around the neighbours' vertices), so
two SSP-RK2 steps reach eight rows; rows are 2^-8 high, so that every difference of
their coordinates is exact, and the step size is fixed.
"""
import numpy as np
import pytest

from lag2d_b200 import workload
from lag2d_b200.mesh import linear_quad_mesh

pytestmark = pytest.mark.gpu

NX, ROWS = 64, 20


def _run(ny, mdegr, steps):
    from lag2d_b200.api import Lag2DSolver
    m = linear_quad_mesh(NX, ny, 0.0, 1.0, 0.0, ny / 256.0)
    c = workload("sod200")[1]
    c.mdegr, c.ndt, c.dtfix, c.tend = mdegr, 0, 5.0e-4, 10.0  # half the CFL limit of the flat cells
    s = Lag2DSolver(m, c)
    _, _, u = s.init_fields()
    n = m.ncell
    rng = np.random.default_rng(5)
    f = 1.0 + 0.05 * rng.standard_normal((4, NX))
    for q, k in ((0, 0), (3, 0)):
        u[:n, q, k] *= np.tile(f[q], ny)
    u[:n, 1, 0] += np.tile(0.1 * f[1] - 0.1, ny)
    u[:n, 0, 1] += np.tile(0.01 * f[2] - 0.01, ny)
    s.set_state(u, m.coord, np.zeros_like(m.coord))
    if steps:
        assert s.run(steps) == steps
        got = s.get_state()[:3]
    else:
        r = s.rhs()[0]
        got = (r,) + tuple(s.get_state()[:3])
    s.close()
    return [a[:ROWS * (NX if len(a.shape) == 3 else NX + 1)] for a in got]


@pytest.mark.parametrize("mdegr", [1, 2, 3])
@pytest.mark.parametrize("steps", [0, 2])
def test_bits_do_not_depend_on_the_size(mdegr, steps):
    for a, b in zip(_run(40, mdegr, steps), _run(1024, mdegr, steps)):
        assert np.array_equal(a, b)
