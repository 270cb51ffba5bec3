"""Area-weighted RZ meshes whose last block of the cell pass has lanes, or whole warps,
past the last cell: these work on the last cell and must store nothing, its mass centre
and mass matrix included.  Runs repeat themselves to the bit, and the last cells end
where the reference-order kernels put them.

Tolerance: 1e-12 of the fields' scale per step, as for the other steps against the
reference order.
"""
import numpy as np
import pytest

from lag2d_b200 import workload
from lag2d_b200.mesh import linear_quad_mesh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(3, 11), (5, 8), (7, 7), (8, 7), (10, 10), (100, 100)])  # 1, 8, 17, 24, 4, 16 of 32
def test_last_cells(nx, ny):
    from lag2d_b200.api import Lag2DSolver
    m = linear_quad_mesh(nx, ny, 0.0, 1.0, 0.0, 1.0, jitter=0.1)
    c = workload("noh_rzaw8")[1]
    c.cfl, c.tend = 0.1, 10.0
    got = []
    for exact in (False, False, True):
        s = Lag2DSolver(m, c, order_exact=exact)
        g, a, u = s.init_fields()
        x, n = m.coord[m.ipqua - 1].mean(axis=1), m.ncell
        u = u.copy()
        u[:n, 0, 0] *= 1.0 + 0.1 * np.sin(3.0 * x[:, 0] + 2.0 * x[:, 1])
        u[:n, 3, 0] += 1.0 + 0.2 * np.cos(2.0 * x[:, 0] - 3.0 * x[:, 1])
        s.set_state(u, m.coord, np.zeros_like(m.coord), g, a)
        assert s.run(4) == 4
        got.append(s.get_state())
        s.close()
    for p, q in zip(got[0], got[1]):
        assert np.array_equal(p, q)
    (uf, _, _, gf), (ue, _, _, ge) = got[0], got[2]
    last = slice(m.ncell - 4, m.ncell)
    scale = np.abs(ue[:m.ncell, :, 0]).max(axis=0)
    assert (np.abs(uf[last, :, 0] - ue[last, :, 0]).max(axis=0) < 4e-12 * scale).all()
    assert np.abs(gf[last, :2] - ge[last, :2]).max() < 4e-11  # centres: a quotient of sums with a digit cancelled
