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
