// The corner-face pass of the optimised FP64 stage, one thread per quad with the
// quad's four sides in a rolled loop.  Included by lag2d_fast.cu inside namespace
// lag2d::fast.
//
// The sub-cell tables are cyclic: turning the quad by a quarter maps corner v,
// its edge node and their corner faces to those of corner v + 1 with the same
// weights.  So the body is written once, for corner c = v, the edge node e to
// the next corner n, the previous edge node ep and corner p, the opposite edge
// node eo and the centre m, and runs four times with the nodes' rows of shared
// memory turned.  Per side there are four distinct face vectors:
//   C1  end of the previous side at c:  (-dy, dx) of -1.5 c + 2 ep - 0.5 p
//   C2  start of the side at c:         (dy, -dx) of -1.5 c + 2 e - 0.5 n
//   A   the side at its mid-node e:     (dy, -dx) of 0.5 (n - c)
//   B   the inner face e - m:           (-dy, dx) of -0.75 e + m - 0.25 eo
// (getfnds_lagsms_simpsonhybrid and getfnds_lagsmsif_hybrid,
// Getrhslaggauss.f90:9660-10021, 3356-3602; the weights below are the tables of
// :10534-10552 x 0.25).  The unrolled 9-node body this replaces was 50 KB of
// instructions and stalled on their fetch as much as on memory: on a mesh that
// fills one wave 20.5 -> 11.8 us a launch (97 x 61), 256 x 256 24 -> 20 us, and
// 242 us on 1024 x 1024 as before (bound by load latency at 16 warps per SM).
// Measured and not kept: one warp per node of 32 quads, nine unrolled bodies
// side by side (380 us on 1024 x 1024, instruction fetch).

__constant__ double cXc[4] = {-1.0, 1.0, 1.0, -1.0}, cYc[4] = {-1.0, -1.0, 1.0, 1.0};  // corners
__constant__ double cXe[4] = {0.0, 1.0, 0.0, -1.0}, cYe[4] = {-1.0, 0.0, 1.0, 0.0};    // edge nodes

__device__ __forceinline__ void stage8(double *dst, const double *src) {
  __pipeline_memcpy_async(dst, src, sizeof(double));
}
__device__ __forceinline__ void basis_at(const CellGeo &g, double x, double y, double *b) {
  b[0] = 1.0;
  b[1] = x - g.rc;
  b[2] = y - g.sc;
  b[3] = 0.5 * b[1] * b[1] - g.g19;
  b[4] = 0.5 * b[2] * b[2] - g.g20;
  b[5] = b[1] * b[2] - g.g21;
}

// ---------------------------------------------------------------------------
// Corner faces: the node partial sums (m, m u - sigma.n A), three rows a node:
// the node solve and the corner forces need m u and sigma.n A only as their
// difference
// ---------------------------------------------------------------------------
// rows of a thread's column: x, y, u*_prev, v*_prev of the 9 nodes, 4 corrections
constexpr int kFaceBlock = 128;
constexpr int kFaceRows = 40;

// vertex state: velocity, 1/tau and the specific internal energy
struct VState {
  double u, v, rho, ke;
};
__device__ __forceinline__ VState vertex_state(const double (*u)[6], const double *b, int mdegr) {
  double st[4];
#pragma unroll
  for (int q = 0; q < 4; q++) {
    double acc = 0.0;
#pragma unroll
    for (int k = 0; k < 6; k++)
      if (k < mdegr) acc += u[q][k] * b[k];
    st[q] = acc;
  }
  return VState{st[1], st[2], 1.0 / st[0], st[3] - 0.5 * (st[1] * st[1] + st[2] * st[2])};
}
// corner_m without its weight 2 w: rho c |a| + kappa |du.a|, or with the
// jump-direction branch (|du| >= 1e12 c; j = du / |du|) the same over |a| times |a.j|
__device__ __forceinline__ double impedance(double rhoc, double kap, double nn, double dun, bool regular, double rdu) {
  const double m = rhoc * nn + kap * dun;
  return regular ? m : m / nn * (dun * rdu);
}

__device__ void f_faces(const Dev &d, int iq_in, double *col) {
  if (iq_in >= d.nquad) return;
  const int iq = iq_in, e = iq + d.ntria;
  const size_t nq = d.nquad;
  // all loads in flight before the first use
  await_previous();
  const int done = d.sc_dev->done;
  int pn[9];
#pragma unroll
  for (int k = 0; k < 9; k++) pn[k] = d.ipq[k * nq + iq];
#pragma unroll
  for (int s = 0; s < 4; s++) stage8(col + (36 + s) * kFaceBlock, d.corr + s * nq + iq);
  double u[4][6];
  load_u(d, d.Us, e, u);
  const CellGeo G{d.rc[e], d.sc[e], d.g19[e], d.g20[e], d.g21[e]};
#pragma unroll
  for (int k = 0; k < 9; k++) {
    stage8(col + k * kFaceBlock, d.xs + pn[k]);
    stage8(col + (9 + k) * kFaceBlock, d.ys + pn[k]);
    stage8(col + (18 + k) * kFaceBlock, d.us + pn[k]);
    stage8(col + (27 + k) * kFaceBlock, d.vs + pn[k]);
  }
  __pipeline_commit();
  if (d.flag[e] == 2) {
    // the moments WENO replaced (they are not committed to the stage state)
#pragma unroll
    for (int q = 0; q < 4; q++)
#pragma unroll
      for (int k = 1; k < 6; k++) u[q][k] = d.Uw[(q * 5 + k - 1) * nq + iq];
  }
  __pipeline_wait_prior(0);
  if (done) return;
#define FX(k) col[(k) * kFaceBlock]
#define FY(k) col[(9 + (k)) * kFaceBlock]
#define FU(k) col[(18 + (k)) * kFaceBlock]
#define FV(k) col[(27 + (k)) * kFaceBlock]
#define FC(s) col[(36 + (s)) * kFaceBlock]
  const double eps = 1.0e-6, g = d.gamlg, gm = g - 1.0;
  const double rhoct = 1.0 / u[0][0];
  const double pctr = fmax(eps, gm * rhoct * (u[3][0] - 0.5 * (u[1][0] * u[1][0] + u[2][0] * u[2][0])));
  const double sdctr = sqrt(fmax(eps, g * pctr * u[0][0]));
  const double rhoc = rhoct * sdctr, kap = d.cimpd * rhoct * (0.5 * (g + 1.0)), lim2 = 1.0e24 * sdctr * sdctr;
  double b[6];
  basis_at(G, 0.0, 0.0, b);
  const VState m = vertex_state(u, b, d.mdegr);
  const double mdx = FU(8) - m.u, mdy = FV(8) - m.v, mj2 = mdx * mdx + mdy * mdy;
  const bool mreg = mj2 < lim2;
  const double mrj = mreg ? 0.0 : rsqrt(mj2), mpe = gm * m.ke;
  double M0 = 0.0, M3 = 0.0, M4 = 0.0;
  double pm = fmax(eps, (m.rho + FC(0)) * mpe);
#pragma unroll 1
  for (int v = 0; v < 4; v++) {
    const int vn = (v + 1) & 3, vp = (v + 3) & 3, vo = (v + 2) & 3;
    const double cx = FX(v), cy = FY(v), nx = FX(vn), ny = FY(vn), ex = FX(4 + v), ey = FY(4 + v);
    const double corr0 = FC(v), corr1 = FC(vn);
    {
      // corner c: C1 and C2 of sub-cell v with weight 1/6 each
      const double px = FX(vp), py = FY(vp), qx = FX(4 + vp), qy = FY(4 + vp);
      const double ax = 1.5 * cy - 2.0 * qy + 0.5 * py, ay = -1.5 * cx + 2.0 * qx - 0.5 * px;
      const double bx = -1.5 * cy + 2.0 * ey - 0.5 * ny, by = 1.5 * cx - 2.0 * ex + 0.5 * nx;
      basis_at(G, cXc[v], cYc[v], b);
      const VState s = vertex_state(u, b, d.mdegr);
      const double dx = FU(v) - s.u, dy = FV(v) - s.v, j2 = dx * dx + dy * dy;
      const bool reg = j2 < lim2;
      const double rj = reg ? 0.0 : rsqrt(j2);
      const double P0 = (1.0 / 3.0) * (impedance(rhoc, kap, sqrt(ax * ax + ay * ay), fabs(dx * ax + dy * ay), reg, rj) +
                                       impedance(rhoc, kap, sqrt(bx * bx + by * by), fabs(dx * bx + dy * by), reg, rj));
      const double pw = (-1.0 / 3.0) * fmax(eps, gm * (s.rho + corr0) * s.ke);
      double *o = d.npart + v * nq + iq;
      o[0] = P0;
      o[9 * nq] = P0 * s.u - pw * (ax + bx);
      o[18 * nq] = P0 * s.v - pw * (ay + by);
    }
    {
      // edge node e: A with weight 1/3 and -B, B with weight 2/3 in sub-cells
      // v, v + 1; centre: B with weight 1/4 out of v, into v + 1
      const double ax = 0.5 * (ny - cy), ay = 0.5 * (cx - nx);
      const double bx = 0.75 * ey - FY(8) + 0.25 * FY(4 + vo), by = FX(8) - 0.75 * ex - 0.25 * FX(4 + vo);
      const double nb = sqrt(bx * bx + by * by);
      basis_at(G, cXe[v], cYe[v], b);
      const VState s = vertex_state(u, b, d.mdegr);
      const double dx = FU(4 + v) - s.u, dy = FV(4 + v) - s.v, j2 = dx * dx + dy * dy;
      const bool reg = j2 < lim2;
      const double rj = reg ? 0.0 : rsqrt(j2);
      const double P0 =
          (4.0 / 3.0) * impedance(rhoc, kap, sqrt(ax * ax + ay * ay), fabs(dx * ax + dy * ay), reg, rj) +
          (8.0 / 3.0) * impedance(rhoc, kap, nb, fabs(dx * bx + dy * by), reg, rj);
      const double pe = gm * s.ke;
      const double p0 = fmax(eps, (s.rho + corr0) * pe), p1 = fmax(eps, (s.rho + corr1) * pe);
      const double wa = (-2.0 / 3.0) * (p0 + p1), wb = (4.0 / 3.0) * (p0 - p1);
      double *o = d.npart + (4 + v) * nq + iq;
      o[0] = P0;
      o[9 * nq] = P0 * s.u - (wa * ax + wb * bx);
      o[18 * nq] = P0 * s.v - (wa * ay + wb * by);
      M0 += impedance(rhoc, kap, nb, fabs(mdx * bx + mdy * by), mreg, mrj);
      const double pn1 = fmax(eps, (m.rho + corr1) * mpe);
      M3 += (pm - pn1) * bx;
      M4 += (pm - pn1) * by;
      pm = pn1;
    }
  }
  double *o = d.npart + 8 * nq + iq;
  o[0] = M0;
  o[9 * nq] = M0 * m.u - 0.5 * M3;
  o[18 * nq] = M0 * m.v - 0.5 * M4;
#undef FX
#undef FY
#undef FU
#undef FV
#undef FC
}

__global__ void __launch_bounds__(kFaceBlock, LAG2D_FACES_MINB) k_faces(Dev d) {
  extern __shared__ double face_stage[];
  f_faces(d, blockIdx.x * blockDim.x + threadIdx.x, face_stage + threadIdx.x);
}

// The same with four lanes per quad, lane = side: a lane loads its corner, its edge
// node and the centre and takes the neighbours' coordinates by shuffle, so a side's
// body runs once instead of four times and no shared memory is used: 11.8 -> 6 us
// a launch at 97 x 61.  128 registers, 48 bytes of spills: 162 registers and 3
// blocks an SM are 3% slower a step at 256 x 256.
__device__ __forceinline__ double lane_get(double v, int lane) { return __shfl_sync(0xffffffffu, v, lane, 4); }
__device__ __forceinline__ double lane_sum(double v) {
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  return v + __shfl_xor_sync(0xffffffffu, v, 2);
}
constexpr int kFace4Block = 128;
__global__ void __launch_bounds__(kFace4Block, LAG2D_FACES4_MINB) k_faces4(Dev d) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int v = t & 3, vn = (v + 1) & 3, vp = (v + 3) & 3, vo = (v + 2) & 3;
  const bool valid = (t >> 2) < d.nquad;
  const int iq = valid ? t >> 2 : d.nquad - 1, e = iq + d.ntria;
  const size_t nq = d.nquad;
  // all loads in flight before the first use
  const int done = d.sc_dev->done;
  const int pc = d.ipq[v * nq + iq], pe = d.ipq[(4 + v) * nq + iq], pm = d.ipq[8 * nq + iq];
  double u[4][6];
  load_u(d, d.Us, e, u);
  const CellGeo G{d.rc[e], d.sc[e], d.g19[e], d.g20[e], d.g21[e]};
  const double cx = d.xs[pc], cy = d.ys[pc], cu = d.us[pc], cv = d.vs[pc];
  const double ex = d.xs[pe], ey = d.ys[pe], eu = d.us[pe], ev = d.vs[pe];
  const double mx = d.xs[pm], my = d.ys[pm], mu = d.us[pm], mv = d.vs[pm];
  await_previous();  // WENO: corrections, flags, moments
  const double corr0 = d.corr[v * nq + iq];
  const int flag = d.flag[e];
  if (flag == 2) {
    // the moments WENO replaced (they are not committed to the stage state)
#pragma unroll
    for (int q = 0; q < 4; q++)
#pragma unroll
      for (int k = 1; k < 6; k++) u[q][k] = d.Uw[(q * 5 + k - 1) * nq + iq];
  }
  if (done) return;
  const double nx = lane_get(cx, vn), ny = lane_get(cy, vn), px = lane_get(cx, vp), py = lane_get(cy, vp);
  const double qx = lane_get(ex, vp), qy = lane_get(ey, vp), ox = lane_get(ex, vo), oy = lane_get(ey, vo);
  const double corr1 = lane_get(corr0, vn);
  const double eps = 1.0e-6, g = d.gamlg, gm = g - 1.0;
  const double rhoct = 1.0 / u[0][0];
  const double pctr = fmax(eps, gm * rhoct * (u[3][0] - 0.5 * (u[1][0] * u[1][0] + u[2][0] * u[2][0])));
  const double sdctr = sqrt(fmax(eps, g * pctr * u[0][0]));
  const double rhoc = rhoct * sdctr, kap = d.cimpd * rhoct * (0.5 * (g + 1.0)), lim2 = 1.0e24 * sdctr * sdctr;
  double b[6];
  double *o = d.npart + iq;
  {
    // corner c: C1 and C2 of sub-cell v with weight 1/6 each
    const double ax = 1.5 * cy - 2.0 * qy + 0.5 * py, ay = -1.5 * cx + 2.0 * qx - 0.5 * px;
    const double bx = -1.5 * cy + 2.0 * ey - 0.5 * ny, by = 1.5 * cx - 2.0 * ex + 0.5 * nx;
    basis_at(G, v == 1 || v == 2 ? 1.0 : -1.0, v >= 2 ? 1.0 : -1.0, b);
    const VState s = vertex_state(u, b, d.mdegr);
    const double dx = cu - s.u, dy = cv - s.v, j2 = dx * dx + dy * dy;
    const bool reg = j2 < lim2;
    const double rj = reg ? 0.0 : rsqrt(j2);
    const double P0 = (1.0 / 3.0) * (impedance(rhoc, kap, sqrt(ax * ax + ay * ay), fabs(dx * ax + dy * ay), reg, rj) +
                                     impedance(rhoc, kap, sqrt(bx * bx + by * by), fabs(dx * bx + dy * by), reg, rj));
    const double pw = (-1.0 / 3.0) * fmax(eps, gm * (s.rho + corr0) * s.ke);
    if (valid) {
      o[v * nq] = P0;
      o[(9 + v) * nq] = P0 * s.u - pw * (ax + bx);
      o[(18 + v) * nq] = P0 * s.v - pw * (ay + by);
    }
  }
  // edge node e: A with weight 1/3 and -B, B with weight 2/3 in sub-cells v, v + 1;
  // centre: B with weight 1/4 out of v, into v + 1
  const double bx = 0.75 * ey - my + 0.25 * oy, by = mx - 0.75 * ex - 0.25 * ox;
  const double nb = sqrt(bx * bx + by * by);
  {
    const double ax = 0.5 * (ny - cy), ay = 0.5 * (cx - nx);
    basis_at(G, v == 1 ? 1.0 : v == 3 ? -1.0 : 0.0, v == 2 ? 1.0 : v == 0 ? -1.0 : 0.0, b);
    const VState s = vertex_state(u, b, d.mdegr);
    const double dx = eu - s.u, dy = ev - s.v, j2 = dx * dx + dy * dy;
    const bool reg = j2 < lim2;
    const double rj = reg ? 0.0 : rsqrt(j2);
    const double P0 = (4.0 / 3.0) * impedance(rhoc, kap, sqrt(ax * ax + ay * ay), fabs(dx * ax + dy * ay), reg, rj) +
                      (8.0 / 3.0) * impedance(rhoc, kap, nb, fabs(dx * bx + dy * by), reg, rj);
    const double pe0 = gm * s.ke;
    const double p0 = fmax(eps, (s.rho + corr0) * pe0), p1 = fmax(eps, (s.rho + corr1) * pe0);
    const double wa = (-2.0 / 3.0) * (p0 + p1), wb = (4.0 / 3.0) * (p0 - p1);
    if (valid) {
      o[(4 + v) * nq] = P0;
      o[(13 + v) * nq] = P0 * s.u - (wa * ax + wb * bx);
      o[(22 + v) * nq] = P0 * s.v - (wa * ay + wb * by);
    }
  }
  basis_at(G, 0.0, 0.0, b);
  const VState m = vertex_state(u, b, d.mdegr);
  const double mdx = mu - m.u, mdy = mv - m.v, mj2 = mdx * mdx + mdy * mdy;
  const bool mreg = mj2 < lim2;
  const double mrj = mreg ? 0.0 : rsqrt(mj2), mpe = gm * m.ke;
  const double dp = fmax(eps, (m.rho + corr0) * mpe) - fmax(eps, (m.rho + corr1) * mpe);
  const double M0 = lane_sum(impedance(rhoc, kap, nb, fabs(mdx * bx + mdy * by), mreg, mrj));
  const double M3 = lane_sum(dp * bx), M4 = lane_sum(dp * by);
  if (valid && v < 3) o[(8 + 9 * v) * nq] = v == 0 ? M0 : v == 1 ? M0 * m.u - 0.5 * M3 : M0 * m.v - 0.5 * M4;
}

// The RHS pass (f_rhs3) with four lanes per quad: the face moments of the lane's
// corner and edge node, one outer Lobatto row (r = -1, -a, a, 1) and one point of
// the middle row per lane, its centre point by all four with a quarter of the
// weight; then each lane keeps one equation (sums exchanged in two steps) and
// updates it: 12.7 -> 8 us a launch at 97 x 61.  What the update needs waits in
// shared memory (in registers 420 bytes of spills); at 168 registers 5% slower a
// step at 64 x 64.
struct RowSums {
  double A0[4], A1[4], B0[4], B1[4];
};
// adds the point s with the weight w (of the row) to the sums
__device__ __forceinline__ void rhs_point(const double *xr, const double *yr, const double *xs, const double *ys,
                                          const double *ra, const double *rb, const double *rc2, double s, double ds,
                                          double w, double rtau, double gm, RowSums &S) {
  const double jxr = xr[0] + s * (xr[1] + s * xr[2]), jyr = yr[0] + s * (yr[1] + s * yr[2]);
  const double jxs = xs[0] + s * xs[1], jys = ys[0] + s * ys[1];
  double un[4];
#pragma unroll
  for (int q = 1; q < 4; q++) un[q] = ra[q] + ds * (rb[q] + rc2[q] * ds);
  const double pres = fmax(1.0e-6, gm * rtau * (un[3] - 0.5 * (un[1] * un[1] + un[2] * un[2])));
  const double al = jys * un[1] - jxs * un[2], be = jxr * un[2] - jyr * un[1];
  const double wp = w * pres, ws = w * s, wps = wp * s;
  S.A0[0] -= w * al;
  S.B0[0] -= w * be;
  S.A0[1] += wp * jys;
  S.B0[1] -= wp * jyr;
  S.A0[2] -= wp * jxs;
  S.B0[2] += wp * jxr;
  S.A0[3] += wp * al;
  S.B0[3] += wp * be;
  S.A1[0] -= ws * al;
  S.B1[0] -= ws * be;
  S.A1[1] += wps * jys;
  S.B1[1] -= wps * jyr;
  S.A1[2] -= wps * jxs;
  S.B1[2] += wps * jxr;
  S.A1[3] += wps * al;
  S.B1[3] += wps * be;
}
constexpr int kRhs4Block = 64;
__global__ void __launch_bounds__(kRhs4Block, LAG2D_RHS4_MINB) k_rhs4(Dev d, int fuse_update, double alfa) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int v = t & 3;
  const bool valid = (t >> 2) < d.nquad;
  const int iq = valid ? t >> 2 : d.nquad - 1, e = iq + d.ntria;
  const size_t nq = d.nquad, nc = d.ncell;
  // all loads in flight before the first use
  const int done = d.sc_dev->done;
  int pn[9];
#pragma unroll
  for (int k = 0; k < 9; k++) pn[k] = d.ipq[k * nq + iq];
  const int pc = d.ipq[v * nq + iq], pe = d.ipq[(4 + v) * nq + iq];
  const double c0 = d.npart[v * nq + iq], c1 = d.npart[(9 + v) * nq + iq], c2 = d.npart[(18 + v) * nq + iq];
  const double e0 = d.npart[(4 + v) * nq + iq], e1 = d.npart[(13 + v) * nq + iq], e2 = d.npart[(22 + v) * nq + iq];
  double u[4][6];
  load_u(d, d.Us, e, u);
  const CellGeo G{d.rc[e], d.sc[e], d.g19[e], d.g20[e], d.g21[e]};
  // M^-1, U^n and the source wait in shared memory, a column per quad
  __shared__ double stage[46][kRhs4Block / 4];
  double(*col)[kRhs4Block / 4] = reinterpret_cast<double(*)[kRhs4Block / 4]>(&stage[0][threadIdx.x >> 2]);
  if (fuse_update) {
#pragma unroll
    for (int i = 0; i < 4; i++) stage8(&col[4 * v + i][0], d.amatr + (4 * v + i) * nc + e);
    if (alfa != 0.0)
#pragma unroll
      for (int k = 0; k < 6; k++) stage8(&col[16 + 6 * v + k][0], d.Un + (v * 6 + k) * nc + e);
  }
  if (d.ncase == 1 && v == 3)
#pragma unroll
    for (int k = 0; k < 6; k++) stage8(&col[40 + k][0], d.src + k * nq + iq);
  __pipeline_commit();
  const int flag = d.flag[e];
  Loaded L;
  {
    const int A[9] = {0, 2, 2, 0, 1, 2, 1, 0, 1}, B[9] = {0, 0, 2, 2, 0, 1, 2, 1, 1};
#pragma unroll
    for (int k = 0; k < 9; k++) {
      L.X[A[k]][B[k]] = d.xs[pn[k]];
      L.Y[A[k]][B[k]] = d.ys[pn[k]];
    }
  }
  if (flag == 2) {
    // the moments WENO replaced (they are not committed to the stage state)
#pragma unroll
    for (int q = 0; q < 4; q++)
#pragma unroll
      for (int k = 1; k < 6; k++) u[q][k] = d.Uw[(q * 5 + k - 1) * nq + iq];
  }
  // the volume integral ahead of the wait
  double R[4][6];
#pragma unroll
  for (int q = 0; q < 4; q++)
#pragma unroll
    for (int k = 0; k < 6; k++) R[q][k] = 0.0;
  QuadMap m;
  map_coeffs(L.X, m.a);
  map_coeffs(L.Y, m.b);
  const double gm = d.gamlg - 1.0;
  double rc2[4];
#pragma unroll
  for (int q = 0; q < 4; q++) rc2[q] = 0.5 * u[q][4];
#pragma unroll 1
  for (int h = 0; h < 2; h++) {
    const int i = h == 0 ? (v < 2 ? v : v + 1) : 2;
    const double r = cL5[i], dr = r - G.rc;
    double xr[3], yr[3], xs[2], ys[2], ra[4], rb[4];
#pragma unroll
    for (int n = 0; n < 3; n++) {
      xr[n] = m.a[1][n] + (2.0 * r) * m.a[2][n];
      yr[n] = m.b[1][n] + (2.0 * r) * m.b[2][n];
    }
#pragma unroll
    for (int n = 0; n < 2; n++) {
      const double c = n + 1.0;
      xs[n] = c * (m.a[0][n + 1] + r * (m.a[1][n + 1] + r * m.a[2][n + 1]));
      ys[n] = c * (m.b[0][n + 1] + r * (m.b[1][n + 1] + r * m.b[2][n + 1]));
    }
    const double b3 = 0.5 * dr * dr - G.g19;
#pragma unroll
    for (int q = 0; q < 4; q++) {
      ra[q] = u[q][0] + u[q][1] * dr + u[q][3] * b3 - u[q][4] * G.g20 - u[q][5] * G.g21;
      rb[q] = u[q][2] + u[q][5] * dr;
    }
    RowSums S;
#pragma unroll
    for (int q = 0; q < 4; q++) S.A0[q] = S.A1[q] = S.B0[q] = S.B1[q] = 0.0;
    if (h == 0) {
      double rtau[5], tq[5], pre[5];
#pragma unroll
      for (int j = 0; j < 5; j++) {
        const double ds = l5p(j) - G.sc;
        tq[j] = ra[0] + ds * (rb[0] + rc2[0] * ds);
        pre[j] = j == 0 ? tq[0] : pre[j - 1] * tq[j];
      }
      double inv = 1.0 / pre[4];
#pragma unroll
      for (int j = 4; j > 0; j--) {
        rtau[j] = inv * pre[j - 1];
        inv = inv * tq[j];
      }
      rtau[0] = inv;
#pragma unroll
      for (int j = 0; j < 5; j++)
        rhs_point(xr, yr, xs, ys, ra, rb, rc2, l5p(j), l5p(j) - G.sc, l5w(j), rtau[j], gm, S);
    } else {
      const double s = cL5[v < 2 ? v : v + 1], ds = s - G.sc;
      const double ta = ra[0] + ds * (rb[0] + rc2[0] * ds), tb = ra[0] - G.sc * (rb[0] - rc2[0] * G.sc);
      const double inv = 1.0 / (ta * tb);
      rhs_point(xr, yr, xs, ys, ra, rb, rc2, s, ds, cLw[v < 2 ? v : v + 1], inv * tb, gm, S);
      rhs_point(xr, yr, xs, ys, ra, rb, rc2, 0.0, -G.sc, 0.25 * l5w(2), inv * ta, gm, S);
    }
    const double wi = cLw[i], wr = wi * dr;
#pragma unroll
    for (int q = 0; q < 4; q++) {
      R[q][1] += wi * S.A0[q];
      R[q][2] += wi * S.B0[q];
      R[q][3] += wr * S.A0[q];
      R[q][4] += wi * (S.B1[q] - G.sc * S.B0[q]);
      R[q][5] += wi * (S.A1[q] - G.sc * S.A0[q]) + wr * S.B0[q];
    }
  }
  await_previous();  // the node pass, in stage 1 the time step
  const double dt = d.sc_dev->dtfix;
  const double uc = d.us_new[pc], vc = d.vs_new[pc], ue = d.us_new[pe], ve = d.vs_new[pe];
  {
    // the lane's corner c and edge node e, the corners and edge nodes next to them
    const double xc = v == 1 || v == 2 ? 1.0 : -1.0, yc = v >= 2 ? 1.0 : -1.0;
    const double xe = v == 1 ? 1.0 : v == 3 ? -1.0 : 0.0, ye = v == 2 ? 1.0 : v == 0 ? -1.0 : 0.0;
    const double ax = d.xs[pc], ay = d.ys[pc], bx = d.xs[pe], by = d.ys[pe];
    const int vn = (v + 1) & 3, vp = (v + 3) & 3;
    const double nx = lane_get(ax, vn), ny = lane_get(ay, vn), px = lane_get(ax, vp), py = lane_get(ay, vp);
    const double qx = lane_get(bx, vp), qy = lane_get(by, vp);
    double tx, ty, fc[4], fe[4];
    corner_flux(px, py, qx, qy, bx, by, nx, ny, tx, ty);
    fc[0] = uc * tx + vc * ty;
    fc[1] = uc * c0 - c1;
    fc[2] = vc * c0 - c2;
    fc[3] = uc * fc[1] + vc * fc[2];
    edge_flux(ax, ay, nx, ny, tx, ty);
    fe[0] = ue * tx + ve * ty;
    fe[1] = ue * e0 - e1;
    fe[2] = ve * e0 - e2;
    fe[3] = ue * fe[1] + ve * fe[2];
    double bc[6], be[6];
    basis_at(G, xc, yc, bc);
    basis_at(G, xe, ye, be);
#pragma unroll
    for (int q = 0; q < 4; q++)
#pragma unroll
      for (int k = 0; k < 6; k++) R[q][k] += fc[q] * bc[k] + fe[q] * be[k];
  }
  // lane v keeps equation v
  double T[2][6], Rq[6];
#pragma unroll
  for (int q = 0; q < 2; q++)
#pragma unroll
    for (int k = 0; k < 6; k++) {
      const double mine = v & 2 ? R[q + 2][k] : R[q][k], other = v & 2 ? R[q][k] : R[q + 2][k];
      T[q][k] = mine + __shfl_xor_sync(0xffffffffu, other, 2);
    }
#pragma unroll
  for (int k = 0; k < 6; k++) {
    const double mine = v & 1 ? T[1][k] : T[0][k], other = v & 1 ? T[0][k] : T[1][k];
    Rq[k] = mine + __shfl_xor_sync(0xffffffffu, other, 1);
  }
  __pipeline_wait_prior(0);
  __syncwarp();
  if (!valid || done) return;
  if (d.ncase == 1 && v == 3)
#pragma unroll
    for (int k = 0; k < 6; k++) Rq[k] += col[40 + k][0];
  if (!fuse_update) {
#pragma unroll
    for (int k = 0; k < 6; k++) d.rhs[(v * 6 + k) * nc + e] = Rq[k];
    return;
  }
#pragma unroll
  for (int k = 0; k < 6; k++) Rq[k] = dt * Rq[k];
  const double oma = 1.0 - alfa;
  const int IDX[5][5] = {{0, 1, 2, 3, 4}, {1, 5, 6, 7, 8}, {2, 6, 9, 10, 11}, {3, 7, 10, 12, 13}, {4, 8, 11, 13, 14}};
#pragma unroll
  for (int k = 0; k < 6; k++) {
    double acc = 0.0;
    if (k == 0) {
      acc = col[15][0] * Rq[0];
    } else {
#pragma unroll
      for (int j = 0; j < 5; j++) acc += col[IDX[k == 0 ? 0 : k - 1][j]][0] * Rq[j + 1];
    }
    const double uk = oma * ((v < 2 ? (v == 0 ? u[0][k] : u[1][k]) : (v == 2 ? u[2][k] : u[3][k])) + acc);
    d.Uo[(v * 6 + k) * nc + e] = alfa != 0.0 ? alfa * col[16 + 6 * v + k][0] + uk : uk;  // stage 1 has alfa = 0 and reads no U^n
  }
}
