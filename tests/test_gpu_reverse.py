"""The reverse RHS and corner-face passes around their block sizes (64 quads, 32 quads
with four lanes each), with a limited degree, and on cells too large for the source's
series: the gradient must not know the numbering, so a mesh with its quads in another
order gives the same gradient, every quad in another place of its block.  (That the
gradient is right is checked by differences elsewhere.)

Tolerance: the sums of about 100 terms cancel by up to four digits, 2e-10 of the
largest entry.
"""
import numpy as np
import pytest

from lag2d_b200.config import StepConfig
from lag2d_b200.mesh import Mesh, quad_mesh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,mdegr,size", [((8, 4), 6, 1.0), ((11, 3), 6, 1.0), ((16, 4), 6, 1.0), ((13, 5), 6, 1.0),
                                              ((9, 7), 3, 1.0), ((43, 3), 6, 1.0), ((5, 4), 6, 2.5)])
def test_renumbered_quads(shape, mdegr, size):
    from lag2d_b200.api import Lag2DSolver
    m = quad_mesh(*shape, 0.0, size, 0.0, size, jitter=0.1, curve=0.05, seed=4)
    n, rng = m.ncell, np.random.default_rng(7)
    order = rng.permutation(n)
    c = StepConfig(ncase=1, gamlg=5.0 / 3.0, nstag=3, cfl=0.05, tend=10.0, ndt=0, mdegr=mdegr)
    us, noise, got = 1e-3 * rng.standard_normal(m.coord.shape), rng.standard_normal((n, 4, 3)), []
    for p in (np.arange(n), order):
        s = Lag2DSolver(Mesh(coord=m.coord, ipqua=m.ipqua[p], iptri=m.iptri, bface=m.bface), c)
        geoel, amatr, u = s.init_fields()
        u[:n, :, :3] += np.array([2e-4, 1e-4, 1e-4]) * noise[p]
        s.set_state(u, m.coord, us, geoel, amatr)
        s.itime, s.dtfix, s.tacru = 1, c.dtfix, 0.0
        J, gU, gX, gS, _ = s.adjoint(2, 1)
        back = np.empty_like(gU[:n])
        back[p] = gU[:n]
        got.append((J, back, gX, gS))
        s.close()
    assert abs(got[0][0] - got[1][0]) <= 1e-13 * got[0][0]
    for a, b in zip(got[0][1:], got[1][1:]):
        assert np.abs(a - b).max() < 2e-10 * np.abs(a).max()
