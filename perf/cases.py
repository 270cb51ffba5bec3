"""The work that users of the time step have it do, as measurable cases.

Every case is one call sequence of the public host API
(:class:`lag2d_b200.api.Lag2DSolver`): upload a state from pinned host
buffers, advance it (``run``: many steps on the device, ``step``: one call
per step, ``adjoint`` / ``adjoint_step``: gradients of a window or a step),
and read the whole result back.  Windows are as long as a last-bit change of
the state stays small in them.  The families:

  tgv      Taylor-Green vortex on curved P2 quads, SSP-RK3, CFL time step
  sedov    Sedov blast on P2 quads (Persson marks, WENO replaces cells)
  hybrid   Taylor-Green on a mesh of triangles and quads at a fixed time step
  sod      Sod shock tube on straight quads, linear P1 branch, SSP-RK2
  rz       Noh implosion in RZ on straight quads (nrz = 1 true volume,
           nrz = 2 area-weighted), SSP-RK2

A case holds the family, the mesh size (nx, ny), the number of steps, the
precision (0 FP64, 1 FP32-mixed) and the mode of the call.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from lag2d_b200.api import Lag2DSolver
from lag2d_b200.config import StepConfig
from lag2d_b200.mesh import Mesh, hybrid_mesh, linear_quad_mesh, quad_mesh
from lag2d_b200.roofline import stage_bytes, stage_bytes_p1

LARGEST = 1024 * 1024 * 20  # cells x steps of the largest run


def _case(family, nx, ny, steps, mode="run", **kw):
    c = {"family": family, "nx": nx, "ny": ny, "steps": steps, "mode": mode, "precision": 0, "curved": 0,
         "checkpoint": 0, "nrz": 0, "noise": 0}
    c.update(kw)
    return c


def listed():
    cases = {
        # a host code that drives the step itself, one call per step, on a small mesh: latency
        "tgv16_step": _case("tgv", 16, 16, 10, "step"),
        # an ordinary small run on a general mesh: odd sizes, moved vertices, curved edges
        "tgv97x61_curved": _case("tgv", 97, 61, 40, curved=1),
        # a medium run, whose state stays in L2
        "tgv256": _case("tgv", 256, 256, 30),
        # the benchmark's mesh: the largest run, far beyond L2
        "tgv1024": _case("tgv", 1024, 1024, 20),
        # the FP32-mixed form; few steps: its FP32 sums amplify a last-bit change of the state to 1e-9 at once
        "tgv512_mixed": _case("tgv", 512, 512, 4, precision=1),
        # the blast the limiter works on: marks and WENO replacements in every stage
        "sedov128": _case("sedov", 128, 128, 60),
        # gradient of a window from a noisy guess of the state: forward, recompute from checkpoints, reverse
        "tgv256_adjoint": _case("tgv", 256, 256, 4, "adjoint", checkpoint=2, noise=1),
        # triangles and quads together
        "hybrid128": _case("hybrid", 128, 128, 20),
        # the linear branch: the shock tube's usual 200 x 10 cells, and a large mesh
        "sod200x10": _case("sod", 200, 10, 60),
        "sod1024x512": _case("sod", 1024, 512, 30),
        # axisymmetric runs, both RZ forms; short: the cold implosion amplifies a last-bit change fast
        "noh_rz100": _case("rz", 100, 100, 20, nrz=1),
        "noh_rzaw100": _case("rz", 100, 100, 40, nrz=2),
    }
    return [dict(c, name=n) for n, c in cases.items()]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: a family by how often it is run, sizes over the
    logarithm of their range, square and odd ones."""
    kind = rng.choice(["tgv", "tgv", "tgv", "mixed", "sedov", "adjoint", "adjoint_step", "hybrid", "sod", "sod", "rz",
                       "rz"])
    steps = _log(rng, 4, 60)
    if kind in ("tgv", "mixed"):
        nx, ny = _log(rng, 12, 1024), _log(rng, 12, 1024)
        steps = max(2, min(steps, LARGEST // (nx * ny)))
        if kind == "mixed":
            return _case("tgv", nx, ny, min(steps, 4), precision=1, curved=rng.randint(0, 1))
        return _case("tgv", nx, ny, steps, rng.choice(["run", "run", "step"]), curved=rng.randint(0, 1))
    if kind == "sedov":
        n = 2 * _log(rng, 12, 80)
        return _case("sedov", n, n, steps)
    if kind in ("adjoint", "adjoint_step"):
        nx, ny = _log(rng, 12, 320), _log(rng, 12, 320)
        if kind == "adjoint_step":
            return _case("tgv", nx, ny, 1, "adjoint_step", curved=1, noise=1)
        return _case("tgv", nx, ny, rng.randint(2, 6), "adjoint", checkpoint=rng.randint(1, 4),
                     curved=rng.randint(0, 1), noise=1)
    if kind == "hybrid":
        return _case("hybrid", _log(rng, 8, 160), _log(rng, 8, 160), min(steps, 20))
    if kind == "sod":
        return _case("sod", _log(rng, 40, 1024), _log(rng, 4, 512), min(steps, 20))
    return _case("rz", _log(rng, 12, 256), _log(rng, 12, 256), min(steps, 20), nrz=rng.randint(1, 2))


def _straight_rz(nx, ny):
    """Axis at y = 0, slip wall at x = 0, pressure boundaries on the outer sides."""
    m = linear_quad_mesh(nx, ny, 0.0, 1.0, 0.0, ny / nx)
    bf = m.bface.copy()
    bf[:nx, 2:4] = (22, 221)
    bf[nx:2 * nx + ny, 2:4] = (21, 0)
    bf[2 * nx + ny:, 2:4] = (22, 222)
    return Mesh(coord=m.coord, ipqua=m.ipqua, iptri=m.iptri, bface=bf, nvqua=4)


@functools.lru_cache(maxsize=2)
def _problem(family, nx, ny, curved, nrz):
    """Mesh and configuration, which a user's program reads from its files once."""
    if family == "tgv":
        m = quad_mesh(nx, ny, 0.0, 1.0, 0.0, 1.0, jitter=0.08 * curved, curve=0.04 * curved)
        c = StepConfig(ncase=1, gamlg=5.0 / 3.0, nstag=3, cfl=0.05, tend=10.0)
    elif family == "sedov":
        m = quad_mesh(nx, ny, -1.2, 1.2, -1.2, 1.2)
        h = nx // 2
        cells = ((h - 1) * nx + h, (h - 1) * nx + h + 1, h * nx + h, h * nx + h + 1)
        c = StepConfig(ncase=7, gamlg=1.4, nstag=3, cfl=0.3, tend=1.0, sedov_cells=cells)
    elif family == "hybrid":
        # the CFL step comes from the quads only and is too long for the triangles
        m = hybrid_mesh(nx, ny, 0.0, 1.0, 0.0, 1.0)
        c = StepConfig(ncase=1, gamlg=5.0 / 3.0, nstag=3, ndt=0, dtfix=0.005 / max(nx, ny), tend=10.0)
    elif family == "sod":
        m = linear_quad_mesh(nx, ny, 0.0, 1.0, 0.0, ny / (2.0 * nx) if ny < nx else 0.5)
        c = StepConfig(npoly=1, ndegr=3, mdegr=3, ncase=6, gamlg=1.4, nstag=2, cfl=0.3, tend=0.2)
    else:
        m = _straight_rz(nx, ny)
        c = StepConfig(npoly=1, ndegr=3, mdegr=3, ncase=3, gamlg=5.0 / 3.0, nstag=2, cfl=0.3, tend=0.6, nrz=nrz)
    return m, c


def _of(case):
    return _problem(case["family"], case["nx"], case["ny"], case["curved"], case["nrz"])


def _factor(mesh, seed):
    """Smooth factor per cell, 1 within a percent, for the velocities (its
    square for the energies): another seed is another initial state."""
    rng = np.random.default_rng(seed)
    corners = mesh.ipqua[:, :4] - 1
    xc = mesh.coord[corners].mean(axis=1)
    if mesh.ntria:
        xc = np.concatenate([mesh.coord[mesh.iptri[:, :3] - 1].mean(axis=1), xc])
    f = np.ones(mesh.ncell)
    for _ in range(3):
        k, a, ph = rng.uniform(-3.0, 3.0, 2), rng.uniform(0.001, 0.003), rng.uniform(0.0, 2.0 * np.pi)
        f += a * np.cos(np.pi * (xc @ k) + ph)
    return f


def _noise(case, mesh, seed):
    """Velocity noise of a state that comes from measurement (None without)."""
    if not case["noise"]:
        return None
    scale = np.array([3.0e-3] + [5.0e-4] * 5)
    return scale * np.random.default_rng([seed, 2]).standard_normal((mesh.ncell, 2, 6))


def _perturb(case, mesh, unkno, seed):
    f = _factor(mesh, seed)[:, None]
    n = mesh.ncell
    unkno[:n, 1] *= f
    unkno[:n, 2] *= f
    unkno[:n, 3] *= f * f
    w = _noise(case, mesh, seed)
    if w is not None:
        unkno[:n, 1:3] += w
    return unkno


def _pinned(a):
    t = torch.empty(a.shape, dtype=torch.float64, pin_memory=torch.cuda.is_available())
    t.numpy()[...] = a
    return t


class _State:
    pass


def prepare(case, seed):
    """The solver of the mesh (its plan) and the initial state in pinned host
    buffers; the state read back goes to pinned buffers as well."""
    m, c = _of(case)
    st = _State()
    st.case, st.cfg = case, c
    st.solver = Lag2DSolver(m, c, precision=case["precision"])
    geoel, amatr, unkno = st.solver.init_fields()
    # the area-weighted form renews its mass centres and mass matrices, so they are part of its state
    st.moving = {"geoel": geoel, "amatr": amatr} if case["nrz"] == 2 else None
    ustar = np.zeros_like(m.coord)
    st.start = [_pinned(a) for a in (_perturb(case, m, unkno, seed), m.coord, ustar)]
    st.end = [_pinned(np.zeros_like(a)) for a in (unkno, m.coord, ustar)]
    st.seed_u = np.random.default_rng(seed + 1).standard_normal((m.ncell, c.nq, c.ndegr)) \
        if case["mode"] == "adjoint_step" else None
    return st


def run(st):
    """Upload, advance, read back."""
    s, case = st.solver, st.case
    if st.moving is None:
        s.set_state_ptrs(*[t.data_ptr() for t in st.start])
    else:
        s.set_state(*[t.numpy() for t in st.start], **st.moving)
    s.itime, s.dtfix, s.tacru = 1, st.cfg.dtfix, 0.0
    if case["mode"] == "adjoint":
        J, gu, gx, gs, _ = s.adjoint(case["steps"], case["checkpoint"])
        return {"J": J, "dJ_dunkno": gu, "dJ_dcoord": gx, "dJ_dustar": gs}
    if case["mode"] == "adjoint_step":
        gu, gx, gs = s.adjoint_step(seed_unkno=st.seed_u)
        return {"grad_unkno": gu, "grad_coord": gx, "grad_ustar": gs}
    if case["mode"] == "step":
        for _ in range(case["steps"]):
            s.step()
    else:
        s.run(case["steps"])
    s.get_state_ptrs(*[t.data_ptr() for t in st.end])
    return {"unkno": st.end[0], "coord": st.end[1], "ustar": st.end[2], "dtfix": s.dtfix, "tacru": s.tacru}


def work(case):
    """State and geometry traffic of the stages, each array read and written
    once per stage, and the state over the link; the arithmetic of the scheme
    per cell and stage (P2 quads 8,000 operations, P1 3,000; a reverse stage
    three times a forward one)."""
    m, c = _of(case)
    if c.npoly == 2:
        stage, ops = stage_bytes(m.ncell, m.npoin), 8000.0 * m.ncell
    else:
        stage, ops = stage_bytes_p1(m.ncell, m.npoin), 3000.0 * m.ncell
    passes = float(case["steps"] * c.nstag)
    if case["mode"] in ("adjoint", "adjoint_step"):
        passes *= 4.0  # one forward, one reverse that reads and writes state and adjoint
    link = 2.0 * 8.0 * (m.ncell * c.nq * c.ndegr + 4 * m.npoin)
    return {"bytes": passes * stage + link, "flops": passes * ops}


# ---------------------------------------------------------------------------
# The Taylor-Green step on quads in plain torch, 64 bits: every quadrature as
# its sum over points, every corner face by itself.  The gradients are
# torch's own, with the time step size held.
# ---------------------------------------------------------------------------
_XV = [-1, 1, 1, -1, 0, 1, 0, -1, 0]
_YV = [-1, -1, 1, 1, -1, 0, 1, 0, 0]
_SUB = [[0, 4, 8, 7], [4, 1, 5, 8], [8, 5, 2, 6], [7, 8, 6, 3]]
# face of each (sub-cell, vertex, side): 1..8 the corner ends of the outer
# edges, 9..12 the inner faces, 13..16 the outer edges' mid-nodes; the sign
# is the orientation
_FACE = [[8, 1, 13, -9, -9, 12, 12, 16], [9, 13, 2, 3, 14, -10, -10, 9],
         [-11, 10, 10, 14, 4, 5, 15, -11], [16, -12, -12, 11, 11, 15, 6, 7]]
_A, _B, _C = 2.0 / 3.0, 4.0 / 3.0, 8.0 / 3.0
_WRIE = [[_A, _A, _B, _C, 1, 1, _C, _B], [_C, _B, _A, _A, _B, _C, 1, 1],
         [1, 1, _C, _B, _A, _A, _B, _C], [_B, _C, 1, 1, _C, _B, _A, _A]]
_WMAS = [[_A, _A, _B, 0, 0, 0, 0, _B], [0, _B, _A, _A, _B, 0, 0, 0],
         [0, 0, 0, _B, _A, _A, _B, 0], [_B, 0, 0, 0, 0, _B, _A, _A]]


class _Plain:
    def __init__(self, mesh, cfg, dev):
        self.c, self.dev = cfg, dev
        t = functools.partial(torch.tensor, dtype=torch.float64, device=dev)
        self.ip = torch.tensor(mesh.ipqua.astype(np.int64) - 1, device=dev)
        self.np_ = mesh.npoin
        g, gw = np.polynomial.legendre.leggauss(5)
        h, hw = np.polynomial.legendre.leggauss(6)
        x = math.sqrt(3.0 / 7.0)
        lo, low = np.array([-1.0, -x, 0.0, x, 1.0]), np.array([0.1, 49.0 / 90.0, 32.0 / 45.0, 49.0 / 90.0, 0.1])
        self.g25, self.g36, self.l25 = [self._points(*v) for v in ((g, gw), (h, hw), (lo, low))]
        self.t = t
        self._sub_tables(g, gw)
        X = t(mesh.coord)[self.ip]
        self._initial(X)
        self.mask_u = torch.zeros(mesh.npoin, dtype=torch.bool, device=dev)
        self.mask_v = torch.zeros_like(self.mask_u)
        for code, m in ((221, self.mask_v), (222, self.mask_u)):
            rows = mesh.bface[(mesh.bface[:, 2] == 22) & (mesh.bface[:, 3] == code)]
            m[torch.tensor(rows[:, [0, 1, 4]].astype(np.int64).reshape(-1) - 1, device=dev)] = True
        inner = np.ones(mesh.nquad, dtype=bool)
        inner[(mesh.esqua > mesh.ncell).any(axis=1)] = False
        self.inner = torch.tensor(inner, device=dev)

    @staticmethod
    def _points(p, w):
        r, s = np.meshgrid(p, p, indexing="ij")
        return r.ravel(), s.ravel(), np.outer(w, w).ravel()

    @staticmethod
    def _shape(r, s):
        """The 9 biquadratic shapes and their derivatives at points (P, 9)."""
        def lag(v):
            return (np.stack([0.5 * v * (v - 1), 1 - v * v, 0.5 * v * (v + 1)], -1),
                    np.stack([v - 0.5, -2 * v, v + 0.5], -1))
        (lr, dr), (ls, ds) = lag(np.asarray(r, float)), lag(np.asarray(s, float))
        a, b = [int(v) + 1 for v in _XV], [int(v) + 1 for v in _YV]
        return lr[:, a] * ls[:, b], dr[:, a] * ls[:, b], lr[:, a] * ds[:, b]

    def _jac(self, r, s, X):
        """x_r, x_s, y_r, y_s at points, each (P, cells)."""
        _, dr, ds = self._shape(r, s)
        x, y = X[..., 0].T, X[..., 1].T
        dr, ds = self.t(dr), self.t(ds)
        return dr @ x, ds @ x, dr @ y, ds @ y

    def _det(self, r, s, X):
        xr, xs, yr, ys = self._jac(r, s, X)
        return xr * ys - xs * yr

    def _sub_tables(self, g, gw):
        """Each sub-cell is itself a 9-node quad: parent nodes, parent map at
        the mid-points of its edges, serendipity centre."""
        q = [(-0.5, -1), (0.5, -1), (1, -0.5), (1, 0.5), (0.5, 1), (-0.5, 1), (-1, 0.5), (-1, -0.5),
             (0, -0.5), (0.5, 0), (0, 0.5), (-0.5, 0)]
        edge = [[0, 8, 11, 7], [1, 2, 9, 8], [9, 3, 4, 10], [11, 10, 5, 6]]
        N = self._shape([p[0] for p in q], [p[1] for p in q])[0]
        self.submap = []
        for i in range(4):
            M = np.zeros((9, 9))
            for k in range(4):
                M[k, _SUB[i][k]] = 1.0
                M[4 + k] = N[edge[i][k]]
            M[8] = -0.25 * M[:4].sum(0) + 0.5 * M[4:8].sum(0)
            self.submap.append(self.t(M))

    def _subareas(self, X):
        r, s, w = self.g25
        return [self.t(w) @ self._det(r, s, torch.einsum("ij,cjd->cid", M, X)) for M in self.submap]

    def _basis(self, r, s):
        """The 6 Taylor functions at points, each (P, cells)."""
        b1 = self.t(r)[:, None] - self.rc
        b2 = self.t(s)[:, None] - self.sc
        return [torch.ones_like(b1), b1, b2, 0.5 * b1 * b1 - self.g19, 0.5 * b2 * b2 - self.g20, b1 * b2 - self.g21]

    def _initial(self, X):
        r, s, w = self.g36
        dj = self.t(w)[:, None] * self._det(r, s, X)
        self.mass = dj.sum(0)
        R, S = self.t(r)[:, None], self.t(s)[:, None]
        self.rc, self.sc = (R * dj).sum(0) / self.mass, (S * dj).sum(0) / self.mass
        self.g19 = (0.5 * (R - self.rc) ** 2 * dj).sum(0) / self.mass
        self.g20 = (0.5 * (S - self.sc) ** 2 * dj).sum(0) / self.mass
        self.g21 = ((R - self.rc) * (S - self.sc) * dj).sum(0) / self.mass
        self.msub = self._subareas(X)
        r, s, w = self.g25
        dj = self.t(w)[:, None] * self._det(r, s, X)
        b = torch.stack(self._basis(r, s)[1:])
        M = torch.einsum("ipc,jpc,pc->cij", b, b, dj)
        self.minv, self.minv0 = torch.linalg.inv(M), 1.0 / dj.sum(0)
        N = self.t(self._shape(r, s)[0])
        x, y = math.pi * (N @ X[..., 0].T), math.pi * (N @ X[..., 1].T)
        u, v = torch.sin(x) * torch.cos(y), -torch.cos(x) * torch.sin(y)
        p = 0.25 * (torch.cos(2 * x) + torch.cos(2 * y)) + 1.0
        f = [torch.ones_like(u), u, v, p / (self.c.gamlg - 1.0) + 0.5 * (u * u + v * v)]
        U = []
        for q in range(4):
            rhs = torch.einsum("ipc,pc->ci", b, f[q] * dj)
            U.append(torch.cat([((f[q] * dj).sum(0) / self.mass)[:, None],
                                torch.einsum("cij,cj->ci", self.minv, rhs)], 1))
        self.U0 = torch.stack(U, 1)  # (cells, 4, 6)

    @staticmethod
    def _eval(U, q, b):
        return sum(U[:, q, k] * b[k] for k in range(6))

    def marked(self, U, X):
        r, s, w = self.g25
        dj = self.t(w)[:, None] * self._det(r, s, X)
        b = self._basis(r, s)
        hi = sum(U[:, 0, k] * b[k] for k in range(3, 6))
        un = self._eval(U, 0, b)
        ratio = (hi * hi * dj).sum(0) / (un * un * dj).sum(0)
        return bool((self.inner & ~(torch.log10(ratio) <= -3.0 * math.log10(4.0) - 4.0)).any())

    def _faces(self, X):
        """Face vectors of the 16 slots (half the area vectors)."""
        out = [None] * 16
        r = [-1, 1, 1, 1, 1, -1, -1, -1, 0, 1, 0, -1]
        s = [-1, -1, -1, 1, 1, 1, 1, -1, -1, 0, 1, 0]
        xr, xs, yr, ys = self._jac(r, s, X)
        for i in range(12):
            side = 0 if i in (0, 1, 8) else 1 if i in (2, 3, 9) else 2 if i in (4, 5, 10) else 3
            out[i if i < 8 else i + 4] = ((yr[i], -xr[i]), (ys[i], -xs[i]), (-yr[i], xr[i]), (-ys[i], xs[i]))[side]
        N = self.t(self._shape([0, 0.5, 0, -0.5], [-0.5, 0, 0.5, 0])[0])
        mid = torch.einsum("ij,cjd->icd", N, X)
        for i in range(4):
            d = -1.5 * X[:, 4 + i] - 0.5 * X[:, 8] + 2.0 * mid[i]
            out[8 + i] = (-d[:, 1], d[:, 0])
        return out

    def rhs(self, U, x, us):
        c, ip = self.c, self.ip
        eps, g = 1.0e-6, c.gamlg
        slp = 0.5 * (g + 1.0)
        X = x[ip]
        F = self._faces(X)
        tau0 = U[:, 0, 0]
        rho = 1.0 / tau0
        pc = torch.clamp((g - 1) * rho * (U[:, 3, 0] - 0.5 * (U[:, 1, 0] ** 2 + U[:, 2, 0] ** 2)), min=eps)
        snd = torch.sqrt(torch.clamp(g * pc / rho, min=eps))
        # sub-cell densities: initial mass over current area against the DG mean
        r, s, w = self.g25
        area = self._subareas(X)
        corr = []
        for i, (a, b) in enumerate(((-1, -1), (1, -1), (1, 1), (-1, 1))):
            rr, ss = 0.5 * (r + a), 0.5 * (s + b)
            dj = self.t(0.25 * w)[:, None] * self._det(rr, ss, X)
            tau = self._eval(U, 0, self._basis(rr, ss))
            corr.append(c.cdrho * (self.msub[i] / area[i] - (dj / tau).sum(0) / dj.sum(0)))
        bn = self._basis(np.array(_XV, float), np.array(_YV, float))
        st = [self._eval(U, q, bn) for q in range(4)]  # (9, cells)
        ke = st[3] - 0.5 * (st[1] ** 2 + st[2] ** 2)
        usn = us[ip]  # (cells, 9, 2)
        node = torch.zeros(self.np_, 5, dtype=torch.float64, device=self.dev)
        part = [[0.0] * 5 for _ in range(9)]
        tm = [[0.0, 0.0] for _ in range(9)]
        for i in range(4):
            for j in range(4):
                k = _SUB[i][j]
                p = torch.clamp((g - 1) * (1.0 / st[0][k] + corr[i]) * ke[k], min=eps)
                dux, duy = usn[:, k, 0] - st[1][k], usn[:, k, 1] - st[2][k]
                for f in range(2):
                    code, wr, wm = _FACE[i][2 * j + f], 0.25 * _WRIE[i][2 * j + f], 0.25 * _WMAS[i][2 * j + f]
                    sg = 1.0 if code > 0 else -1.0
                    ax, ay = (sg * v for v in F[abs(code) - 1])
                    dn = dux * ax + duy * ay
                    dn = torch.where(dn >= 0, dn, -dn)
                    mm = 2.0 * wr * (rho * snd * torch.sqrt(ax * ax + ay * ay) + c.cimpd * rho * slp * dn)
                    add = (mm, mm * st[1][k], mm * st[2][k], -2.0 * p * wr * ax, -2.0 * p * wr * ay)
                    part[k] = [a + b for a, b in zip(part[k], add)]
                    if wm:
                        tm[k] = [tm[k][0] + 2.0 * wm * ax, tm[k][1] + 2.0 * wm * ay]
        for k in range(9):
            node = node.index_add(0, ip[:, k], torch.stack(part[k], 1))
        un = (node[:, 1] - node[:, 3]) / node[:, 0]
        vn = (node[:, 2] - node[:, 4]) / node[:, 0]
        un = torch.where(self.mask_u, torch.zeros_like(un), un)
        vn = torch.where(self.mask_v, torch.zeros_like(vn), vn)
        R = [[0.0] * 6 for _ in range(4)]
        for k in range(8):
            uk, vk = un[ip[:, k]], vn[ip[:, k]]
            P = part[k]
            f0, f1 = P[3] + uk * P[0] - P[1], P[4] + vk * P[0] - P[2]
            val = (uk * tm[k][0] + vk * tm[k][1], f0, f1, uk * f0 + vk * f1)
            for q in range(4):
                R[q] = [R[q][i] + val[q] * bn[i][k] for i in range(6)]
        # volume integrals, 25 Gauss-Lobatto points, cofactor form
        r, s, w = self.l25
        xr, xs, yr, ys = self._jac(r, s, X)
        b = self._basis(r, s)
        u = [self._eval(U, q, b) for q in range(4)]
        W = self.t(w)[:, None]
        pr = torch.clamp((g - 1) / u[0] * (u[3] - 0.5 * (u[1] ** 2 + u[2] ** 2)), min=eps)
        one, zero = torch.ones_like(b[1]), torch.zeros_like(b[1])
        grad = [(one, zero), (zero, one), (b[1], zero), (zero, b[2]), (b[2], b[1])]
        for i, (br, bs) in enumerate(grad):
            g0, g1 = ys * br - yr * bs, -xs * br + xr * bs
            fv = g0 * u[1] + g1 * u[2]
            for q, val in enumerate((-fv, g0 * pr, g1 * pr, fv * pr)):
                R[q][i + 1] = R[q][i + 1] + (W * val).sum(0)
        # energy source
        r, s, w = self.g25
        dj = self.t(w)[:, None] * self._det(r, s, X)
        N = self.t(self._shape(r, s)[0])
        px, py = math.pi * (N @ X[..., 0].T), math.pi * (N @ X[..., 1].T)
        src = 0.25 * math.pi / (g - 1) * dj * (torch.cos(3 * px) * torch.cos(py) - torch.cos(3 * py) * torch.cos(px))
        b = self._basis(r, s)
        R[3] = [R[3][i] + (src * b[i]).sum(0) for i in range(6)]
        return torch.stack([torch.stack(v, 1) for v in R], 1), torch.stack([un, vn], 1)

    def dt(self, U, X, dvdt, itime, dt, tacru):
        c, g = self.c, self.c.gamlg
        edge = [(0, 4, 1), (1, 5, 2), (2, 6, 3), (3, 7, 0)]
        d = torch.stack([(X[:, a] - X[:, b]).norm(dim=1) + (X[:, b] - X[:, e]).norm(dim=1) for a, b, e in edge]).amin(0)
        p = torch.clamp((g - 1) / U[:, 0, 0] * (U[:, 3, 0] - 0.5 * (U[:, 1, 0] ** 2 + U[:, 2, 0] ** 2)), min=1e-6)
        snd = torch.sqrt(torch.clamp(g * p * U[:, 0, 0], min=1e-6))
        r, s, w = self.g36
        vol = (self.t(w)[:, None] * self._det(r, s, X)).sum(0)
        got = min(c.cfl * float((d / snd).min()), 0.1 * float((vol / dvdt.abs()).min()))
        if itime > 1:
            got = min(got, 1.01 * dt)
        return min(got, c.tend - tacru) if tacru + got > c.tend else got

    def step(self, U, x, us, itime, dt, tacru):
        Un, xn = U, x
        for i, alfa in enumerate((0.0, 0.75, 0.3333333333333333)):
            if self.marked(U.detach(), x.detach()[self.ip]):
                return None
            R, us = self.rhs(U, x, us)
            if i == 0:
                dt = self.dt(U.detach(), x.detach()[self.ip], R[:, 0, 0].detach(), itime, dt, tacru)
            inc = torch.cat([(self.minv0[:, None] * R[:, :, 0])[:, :, None],
                             torch.einsum("cij,cqj->cqi", self.minv, R[:, :, 1:])], 2)
            U = alfa * Un + (1.0 - alfa) * (U + dt * inc)
            x = alfa * xn + (1.0 - alfa) * (x + dt * us)
            X = x[self.ip]
            x = x.index_copy(0, self.ip[:, 8], -0.25 * X[:, :4].sum(1) + 0.5 * X[:, 4:8].sum(1))
        return U, x, us, dt, tacru + dt


def exact(case, seed):
    """The Taylor-Green runs and gradients on quads, as plain torch gives
    them.  None for the other families (limited or on triangles: a second
    restatement of the limiters and the triangle rules is not kept here) and
    where a limited cell would need one."""
    if case["family"] != "tgv":
        return None
    m, c = _of(case)
    grad = case["mode"] in ("adjoint", "adjoint_step")
    if grad and m.ncell * case["steps"] > 4 * 256 * 256:
        return None  # the tape of the window would not fit beside the state
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    if m.ncell * case["steps"] > (LARGEST if dev.type == "cuda" else 100000):
        return None
    p = _Plain(m, c, dev)
    f = p.t(_factor(m, seed))[:, None]
    U = torch.stack([p.U0[:, 0], p.U0[:, 1] * f, p.U0[:, 2] * f, p.U0[:, 3] * f * f], 1)
    w = _noise(case, m, seed)
    if w is not None:
        U[:, 1:3] += p.t(w)
    x, us = p.t(m.coord), torch.zeros(m.npoin, 2, dtype=torch.float64, device=dev)
    leaves = [v.detach().requires_grad_(grad) for v in (U, x, us)]
    state, dt, ta = tuple(leaves), c.dtfix, 0.0
    with torch.set_grad_enabled(grad):
        for it in range(1, case["steps"] + 1):
            got = p.step(*state, it, dt, ta)
            if got is None:
                return None
            state, dt, ta = got[:3], got[3], got[4]
    U, x, us = state
    if grad:
        if case["mode"] == "adjoint":
            J = 0.5 * (p.mass * (U[:, 1, 0] ** 2 + U[:, 2, 0] ** 2)).sum()
            gu, gx, gs = (v.cpu().numpy() for v in torch.autograd.grad(J, leaves))
            return {"J": float(J), "dJ_dunkno": gu, "dJ_dcoord": gx, "dJ_dustar": gs}
        w = p.t(np.random.default_rng(seed + 1).standard_normal((m.ncell, 4, 6)))
        gu, gx, gs = (v.cpu().numpy() for v in torch.autograd.grad((w * U).sum(), leaves))
        return {"grad_unkno": gu, "grad_coord": gx, "grad_ustar": gs}
    full = torch.zeros(m.nsize, 4, 6, dtype=torch.float64)
    full[:m.ncell] = U.cpu()
    return {"unkno": full, "coord": x.cpu(), "ustar": us.cpu(), "dtfix": dt, "tacru": ta}
