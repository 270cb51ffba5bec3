"""An adjoint window on a handle with timing on and no captured step yet: same bits as
without timing, real times in the families, and the steps after it as ever."""
import numpy as np
import pytest

from lag2d_b200.config import StepConfig
from lag2d_b200.mesh import quad_mesh

pytestmark = pytest.mark.gpu


def test_timed_window():
    from lag2d_b200.api import Lag2DSolver
    m = quad_mesh(12, 9, jitter=0.05)
    c = StepConfig(ncase=1, gamlg=5.0 / 3.0, nstag=3, cfl=0.02, tend=10.0)
    got = []
    for timed in (False, True):
        s = Lag2DSolver(m, c)
        s.init_fields()
        s.timing(timed)
        out = [s.adjoint(3, 2)[:4]]
        s.step()
        if timed:
            for family in ("persson", "node", "rhs", "dt"):
                ms, n = s.kernel_ms(family)
                assert n > 0 and ms > 1.0e-3  # a launch takes microseconds
        s.timing(False)
        assert s.run(2) == 2
        out += [s.get_state(), (s.dtfix, s.tacru)]
        got.append(out)
        s.close()
    for a, b in zip(*got):
        for x, y in zip(a, b):
            assert np.array_equal(x, y)
