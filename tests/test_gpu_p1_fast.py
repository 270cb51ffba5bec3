"""The optimised linear path against the reference-order kernels on the device:
sizes around a block and around the line between its two plane forms, node
valences 3 to 5, every mdegr, and the same bits run, stepped or timed.

Tolerance: a step within 1e-12 of the fields' scale (some 1e3 roundings of
2.2e-16, as for the steps against the restatement), twice that after two; the
RHS cancels by up to three digits more, 1e-9.
"""
import numpy as np
import pytest

from lag2d_b200 import workload
from lag2d_b200.mesh import Mesh, linear_quad_mesh

pytestmark = pytest.mark.gpu


def _fan(n, k):
    """A regular n-gon around (0.6, 0.7): n quads around its centre, k x k each."""
    ang = 2.0 * np.pi * np.arange(n) / n + 0.1
    c = np.array([0.6, 0.7])
    v = c + 0.4 * np.stack([np.cos(ang), np.sin(ang)], axis=1)
    ids, xy, quads, edges = {}, [], [], {}

    def node(p):
        key = (round(p[0] * 1e9), round(p[1] * 1e9))
        if key not in ids:
            ids[key] = len(xy) + 1
            xy.append(p)
        return ids[key]

    for i in range(n):
        a, b, d = 0.5 * (v[i - 1] + v[i]), v[i], 0.5 * (v[i] + v[(i + 1) % n])
        at = lambda s, t: (1 - s) * (1 - t) * c + s * (1 - t) * a + s * t * b + (1 - s) * t * d
        for j in range(k):
            for l in range(k):
                q = [node(at((j + p) / k, (l + r) / k)) for p, r in ((0, 0), (1, 0), (1, 1), (0, 1))]
                quads.append(q)
                for e in range(4):
                    edges[(q[e], q[(e + 1) % 4])] = 1
    bf = [(a, b, 22, 221, 0) for a, b in edges if (b, a) not in edges]
    return Mesh(coord=np.array(xy), ipqua=np.array(quads), iptri=np.zeros((0, 3), np.int32),
                bface=np.array(bf), nvqua=4)


def _case(kind, nrz, mdegr):
    c = workload({0: "sod40", 1: "noh_rz8", 2: "noh_rzaw8"}[nrz])[1]
    c.mdegr, c.cfl, c.tend = mdegr, 0.1, 10.0
    if isinstance(kind, int):
        return _fan(kind, 3), c
    return linear_quad_mesh(*kind, 0.0, 1.0, 0.0, 1.0, jitter=0.1), c


def _solver(m, c, exact):
    from lag2d_b200.api import Lag2DSolver
    s = Lag2DSolver(m, c, order_exact=exact)
    g, a, u = s.init_fields()
    # slopes and strain far above the limiter's thresholds everywhere
    u = u.copy()
    x, y = m.coord[:, 0], m.coord[:, 1]
    cx = m.coord[m.ipqua - 1].mean(axis=1)
    u[:m.ncell, 0, 0] *= 1.0 + 0.1 * np.sin(3.0 * cx[:, 0] + 2.0 * cx[:, 1])
    u[:m.ncell, 3, 0] += 1.0 + 0.2 * np.cos(2.0 * cx[:, 0] - 3.0 * cx[:, 1])
    us = np.stack([0.1 * np.sin(3.0 * x + y), 0.1 * np.cos(2.0 * y - x)], axis=1)
    s.set_state(u, m.coord, us, g, a)
    return s


def _err(a, b):
    sc = np.abs(b).max(axis=(0, 2), keepdims=True)
    sc[0, 1] = sc[0, 2] = max(sc[0, 1, 0], sc[0, 2, 0])
    return (np.abs(a - b) / np.maximum(sc, 1e-300)).max()


MESHES = [(2, 2), (8, 4), (11, 3), (16, 8), (43, 3), 3, 5]


@pytest.mark.parametrize("kind,nrz,mdegr", [(k, r, d) for k in MESHES for r in (0, 1, 2) for d in (1, 2, 3)] +
                         [(k, 0, d) for k in ((257, 255), (256, 256)) for d in (1, 3)])
def test_reference_order(kind, nrz, mdegr):
    m, c = _case(kind, nrz, mdegr)
    f, e = _solver(m, c, False), _solver(m, c, True)
    n = m.ncell
    (rf, _), (re, _) = f.rhs(), e.rhs()
    assert _err(rf[:n], re[:n]) < 1e-9
    (uf, _, vf, _), (ue, _, ve, _) = f.get_state(), e.get_state()
    assert _err(uf[:n], ue[:n]) < 1e-11
    assert np.abs(vf - ve).max() < 1e-11 * np.abs(ve).max()
    f, e = _solver(m, c, False), _solver(m, c, True)
    assert f.run(2) == e.run(2) == 2
    (uf, xf, _, gf), (ue, xe, _, ge) = f.get_state(), e.get_state()
    assert _err(uf[:n, :, :1], ue[:n, :, :1]) < 2e-12
    assert np.abs(xf - xe).max() < 2e-12
    assert np.abs(gf[:n, 2] / ge[:n, 2] - 1.0).max() < 1e-11
    assert abs(f.dtfix - e.dtfix) <= 2e-12 * e.dtfix


@pytest.mark.parametrize("kind,nrz", [((11, 3), 0), ((256, 256), 0), ((11, 3), 1), ((11, 3), 2), (5, 0), (3, 2)])
def test_same_bits(kind, nrz):
    m, c = _case(kind, nrz, 3)
    got = []
    for mode in ("run", "step", "timed"):
        s = _solver(m, c, False)
        s.timing(mode == "timed")
        if mode == "step":
            for _ in range(3):
                s.step()
        else:
            assert s.run(3) == 3
        got.append((s.get_state(), s.dtfix, s.tacru))
        if mode == "run":
            keep = s
    for g in got[1:]:
        assert g[1:] == got[0][1:]
        for a, b in zip(g[0], got[0][0]):
            assert np.array_equal(a, b)
    # the RHS of the state the steps left, and of the same state uploaded
    u, x, us, geoel = got[0][0]
    t = _solver(m, c, False)
    t.run(3)
    t.set_state(u, x, us)
    (ra, _), (rb, _) = keep.rhs(), t.rhs()
    assert np.array_equal(ra, rb)
