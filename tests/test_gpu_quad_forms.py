"""The corner-face and RHS passes with four lanes and with one thread per quad: mesh
sizes just within and just beyond each line, the nodal solve and two steps against
the reference-order kernels.  (The RHS itself is left to the small meshes: at
h = 1/512 the rounding of the coordinates alone is 1e-9 of its tau equation.)

Tolerance: as around the block sizes, 100 * 2.2e-16 * 1e4 = 2e-10 of the field.
"""
import numpy as np
import pytest

from lag2d_b200.config import StepConfig
from lag2d_b200.mesh import quad_mesh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(96, 98), (97, 98), (512, 512), (513, 512)])
def test_both_forms(shape):
    from lag2d_b200.api import Lag2DSolver
    m = quad_mesh(*shape, jitter=0.1)
    c = StepConfig(ncase=1, gamlg=5.0 / 3.0, nstag=3, cfl=0.02, tend=10.0)
    n, got = m.ncell, []
    for exact in (False, True):
        s = Lag2DSolver(m, c, order_exact=exact)
        _, _, u = s.init_fields()
        rng = np.random.default_rng(3)
        u[:n, :, 0] *= 1.0 + 1.0e-4 * rng.standard_normal((n, 4))
        us = 0.1 * rng.standard_normal(m.coord.shape)
        s.set_state(u, m.coord, us)
        s.rhs()
        v = s.get_state()[2]
        s.set_state(u, m.coord, us)
        s.run(2)
        got.append((v,) + tuple(s.get_state()[:3]))
        s.close()
    (vf, uf, xf, wf), (ve, ue, xe, we) = got
    assert np.abs(vf - ve).max() < 2e-11 * np.abs(ve).max()
    for q in range(4):
        assert np.abs(uf[:n, q] - ue[:n, q]).max() < 2e-10 * np.abs(ue[:n, q]).max()
    assert np.abs(xf - xe).max() < 2e-11 and np.abs(wf - we).max() < 2e-10 * np.abs(we).max()
