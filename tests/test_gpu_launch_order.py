"""Passes that come up behind one another read ahead of the wait only what the pass
before them leaves alone: runs of the captured step give the bits of the same steps
launched one by one with a record between every two passes, whatever the mesh and
the path, also beyond the size the early launch ends at."""
import numpy as np
import pytest

from lag2d_b200 import workload
from lag2d_b200.config import StepConfig
from lag2d_b200.mesh import hybrid_mesh, linear_quad_mesh, quad_mesh

pytestmark = pytest.mark.gpu


def _case(kind):
    c = StepConfig(ncase=1, gamlg=5.0 / 3.0, nstag=3, cfl=0.02, tend=10.0)
    if kind == "hybrid":
        return hybrid_mesh(24, 17, 0.0, 1.0, 0.0, 1.0), c
    if isinstance(kind, tuple):
        return quad_mesh(*kind, jitter=0.05), c
    if kind == "sod80":
        c = workload("sod200")[1]
        return linear_quad_mesh(80, 9, 0.0, 1.0, 0.0, 0.1, jitter=0.1), c
    return workload(kind)


@pytest.mark.parametrize("kind,steps", [((12, 9), 60), ((97, 61), 40), ((120, 110), 30), ((363, 361), 6), ((363, 362), 6),
                                        ("sedov32", 40), ("hybrid", 40), ("sod80", 60), ("noh_rz32", 40),
                                        ("noh_rzaw32", 40)])
def test_run_and_timed_agree(kind, steps):
    from lag2d_b200.api import Lag2DSolver
    m, c = _case(kind)
    got = []
    for timed in (False, True):
        s = Lag2DSolver(m, c)
        s.init_fields()
        s.timing(timed)
        assert s.run(steps) == steps
        got.append((s.get_state(), s.dtfix, s.tacru))
        s.close()
    assert got[0][1:] == got[1][1:]
    for a, b in zip(got[0][0], got[1][0]):
        assert np.array_equal(a, b)
