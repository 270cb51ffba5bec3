"""The timed families: a pass of several kernels counts once, so that the average is the
pass's time whatever its kernels are; a pass per RK stage, the time step's per step."""
import pytest

from lag2d_b200 import workload
from lag2d_b200.config import StepConfig
from lag2d_b200.mesh import hybrid_mesh, quad_mesh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,precision,exact", [(k, 0, e) for k in ("quads", "hybrid", "sod40", "noh_rz8")
                                                  for e in (False, True)] + [("quads", 1, False), ("hybrid", 1, False)])
def test_passes(kind, precision, exact):
    from lag2d_b200.api import Lag2DSolver
    if kind in ("quads", "hybrid"):
        m = quad_mesh(12, 9) if kind == "quads" else hybrid_mesh(7, 5, 0.0, 1.0, 0.0, 1.0)
        c = StepConfig(ncase=1, gamlg=5.0 / 3.0, nstag=3, ndt=0, dtfix=1.0e-4, tend=10.0)
        stage = ("persson", "weno", "corner", "node", "rhs")
    else:
        m, c = workload(kind)
        stage = ("cell", "node", "rhs")
    s = Lag2DSolver(m, c, precision=precision, order_exact=exact)
    s.init_fields()
    s.timing(True)
    for calls in (1, 2):
        s.run(2)
        for f in stage:
            assert s.kernel_ms(f)[1] == 2 * calls * c.nstag, f
        assert s.kernel_ms("dt")[1] == 2 * calls
    s.close()
