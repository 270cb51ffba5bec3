// The reverse of the FP64 RHS pass, one thread per quad.  Included by lag2d_fast.cu
// inside namespace lag2d::fast.  (The FP32-mixed adjoint keeps a_rhs, whose
// sums keep their bits.)
//
// The transposes of f_rhs3 and f_tgv_src in the same terms: every equation adds
// (alpha, beta) . grad b, so along a row the adjoints of alpha and beta are linear in
// s, two operations each in place of five basis gradients (34 operations a point
// instead of 100); the Jacobians and det J hand their adjoints to the map's
// coefficients, and those to the nodes once at the end.  U and the RHS adjoint wait in
// shared memory, a column per thread.  256 x 256: 142 -> 79 us a launch; points
// unrolled 88 (more spills), at 168 registers 10% slower a reverse stage.

// nodes from the map's coefficients (transpose of map_coeffs; l[0][0]: the centre node)
__device__ __forceinline__ void map_coeffs_T(const double l[3][3], double lX[3][3]) {
  double c[3][3];
#pragma unroll
  for (int i = 0; i < 3; i++) {
    c[i][0] = 0.5 * (l[i][2] - l[i][1]);
    c[i][1] = i == 0 ? 0.0 : l[i][0] - l[i][2];
    c[i][2] = 0.5 * (l[i][2] + l[i][1]);
  }
  double o = 0.0;
#pragma unroll
  for (int j = 0; j < 3; j++) {
    const double hi = 0.5 * (c[2][j] + c[1][j]), lo = 0.5 * (c[2][j] - c[1][j]);
    const double mid = j == 1 ? 0.0 : c[0][j] - c[2][j];
    lX[2][j] += hi;
    lX[0][j] += lo;
    if (j != 1) lX[1][j] += mid;
    o += hi + lo + mid;
  }
  lX[1][1] += l[0][0] - o;
}
// transpose of map_det: adjoints of the map's coefficients from those of det J's
__device__ __forceinline__ void map_det_T(const QuadMap &m, const double lD[4][4], QuadMap &l) {
#define CT(c, p, q, i, j, k, h)                                     \
  {                                                                 \
    const double w = (c) * lD[p][q];                                \
    l.a[i][j] += w * m.b[k][h];                                     \
    l.b[k][h] += w * m.a[i][j];                                     \
    l.a[k][h] -= w * m.b[i][j];                                     \
    l.b[i][j] -= w * m.a[k][h];                                     \
  }
  CT(1.0, 0, 0, 1, 0, 0, 1)
  CT(2.0, 0, 1, 1, 0, 0, 2) CT(-1.0, 0, 1, 0, 1, 1, 1)
  CT(2.0, 0, 2, 1, 1, 0, 2) CT(-1.0, 0, 2, 0, 1, 1, 2)
  CT(-2.0, 0, 3, 0, 2, 1, 2)
  CT(1.0, 1, 0, 1, 0, 1, 1) CT(-2.0, 1, 0, 0, 1, 2, 0)
  CT(2.0, 1, 1, 1, 0, 1, 2) CT(-2.0, 1, 1, 0, 1, 2, 1) CT(4.0, 1, 1, 2, 0, 0, 2)
  CT(1.0, 1, 2, 1, 1, 1, 2) CT(-2.0, 1, 2, 0, 1, 2, 2) CT(-4.0, 1, 2, 0, 2, 2, 1)
  CT(-4.0, 1, 3, 0, 2, 2, 2)
  CT(1.0, 2, 0, 1, 0, 2, 1) CT(2.0, 2, 0, 2, 0, 1, 1)
  CT(2.0, 2, 1, 1, 0, 2, 2) CT(4.0, 2, 1, 2, 0, 1, 2) CT(-1.0, 2, 1, 1, 1, 2, 1)
  CT(3.0, 2, 2, 2, 1, 1, 2)
  CT(-2.0, 2, 3, 1, 2, 2, 2)
  CT(2.0, 3, 0, 2, 0, 2, 1)
  CT(4.0, 3, 1, 2, 0, 2, 2)
  CT(2.0, 3, 2, 2, 1, 2, 2)
#undef CT
}

// transpose of the source moments: lR3 of the energy equation -> map's coefficients
__device__ __forceinline__ void tgv_T(const QuadMap &m, const CellGeo &G, double xc, double yc, double g,
                                      const double *lR3, int stride, QuadMap &l) {
  const double PI = 3.14159265358979311599796346854;
  const double coef = PI / (g - 1.0);
  double cxc, sxc, cyc, syc, D[4][4], lD[4][4];
  sincospi(xc, &sxc, &cxc);
  sincospi(yc, &syc, &cyc);
  map_det(m, D);
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int n = 0; n < 4; n++) lD[i][n] = 0.0;
  // the adjoint of the source at a point over 1, r, s, r^2, s^2, r s
  const double l1 = lR3[stride], l2 = lR3[2 * stride], l3 = lR3[3 * stride], l4 = lR3[4 * stride], l5 = lR3[5 * stride];
  const double q0 = lR3[0] - l1 * G.rc - l2 * G.sc + l3 * (0.5 * G.rc * G.rc - G.g19) +
                    l4 * (0.5 * G.sc * G.sc - G.g20) + l5 * (G.rc * G.sc - G.g21);
  const double q1 = l1 - l3 * G.rc - l5 * G.sc, q2 = l2 - l4 * G.sc - l5 * G.rc;
#pragma unroll 1
  for (int i = 0; i < 5; i++) {
    const double r = cG5[i];
    double e[4], px[3], py[3];
    det_row(D, r, e);
#pragma unroll
    for (int n = 0; n < 3; n++) {
      px[n] = n == 0 ? r * (m.a[1][0] + r * m.a[2][0]) : m.a[0][n] + r * (m.a[1][n] + r * m.a[2][n]);
      py[n] = n == 0 ? r * (m.b[1][0] + r * m.b[2][0]) : m.b[0][n] + r * (m.b[1][n] + r * m.b[2][n]);
    }
    const double wi = coef * cW5[i], sa = wi * (q0 + r * (q1 + 0.5 * l3 * r)), sb = wi * (q2 + l5 * r), sc = wi * (0.5 * l4);
    double Mx[3] = {0, 0, 0}, My[3] = {0, 0, 0}, Ls[4] = {0, 0, 0, 0};
#pragma unroll
    for (int j = 0; j < 5; j++) {
      const double s = g5p(j);
      const double dx = px[0] + s * (px[1] + s * px[2]), dy = py[0] + s * (py[1] + s * py[2]);
      const double det = e[0] + s * (e[1] + s * (e[2] + s * e[3]));
      double cx, sx, cy, sy;
      if (fabs(dx) <= 0.15 && fabs(dy) <= 0.15) {
        double cdx, sdx, cdy, sdy;
        cossin_pi_series<7>(dx, cdx, sdx);
        cossin_pi_series<7>(dy, cdy, sdy);
        cx = cxc * cdx - sxc * sdx;
        sx = sxc * cdx + cxc * sdx;
        cy = cyc * cdy - syc * sdy;
        sy = syc * cdy + cyc * sdy;
      } else {
        sincospi(xc + dx, &sx, &cx);
        sincospi(yc + dy, &sy, &cy);
      }
      // src = c_x c_y (c_x^2 - c_y^2) det
      const double ls = g5w(j) * (sa + s * (sb + s * sc)), cx2 = cx * cx, cy2 = cy * cy, ld = ls * det;
      const double lw = ls * ((cx * cy) * (cx2 - cy2));
      const double lx = -PI * sx * (ld * (cy * (3.0 * cx2 - cy2))), ly = -PI * sy * (ld * (cx * (cx2 - 3.0 * cy2)));
      Mx[0] += lx;
      My[0] += ly;
      Ls[0] += lw;
      if (j != 2) {
        Mx[1] += lx * s;
        Mx[2] += lx * (s * s);
        My[1] += ly * s;
        My[2] += ly * (s * s);
        Ls[1] += lw * s;
        Ls[2] += lw * (s * s);
        Ls[3] += lw * (s * s * s);
      }
    }
    double rp = 1.0;
#pragma unroll
    for (int k = 0; k < 4; k++) {
#pragma unroll
      for (int n = 0; n < 4; n++) lD[k][n] += rp * Ls[n];
      if (k < 3)
#pragma unroll
        for (int n = 0; n < 3; n++) {
          l.a[k][n] += rp * Mx[n];
          l.b[k][n] += rp * My[n];
        }
      rp *= r;
    }
  }
  map_det_T(m, lD, l);
}

constexpr int kRevBlock = 64;
__global__ void __launch_bounds__(kRevBlock, 4) k_a_rhs64(Dev d, Adj a) {
  __shared__ double stage[48][kRevBlock];
  const int iq = blockIdx.x * kRevBlock + threadIdx.x;
  if (iq >= d.nquad) return;
  const int e = iq + d.ntria;
  const size_t nq = d.nquad, nc = d.ncell;
  double *col = &stage[0][threadIdx.x];
#pragma unroll 8
  for (int v = 0; v < 24; v++) {
    __pipeline_memcpy_async(col + v * kRevBlock, d.Us + v * nc + e, sizeof(double));
    __pipeline_memcpy_async(col + (24 + v) * kRevBlock, a.lR + v * nc + e, sizeof(double));
  }
  __pipeline_commit();
#define AU(q, k) col[((q) * 6 + (k)) * kRevBlock]
#define AR(q, k) col[(24 + (q) * 6 + (k)) * kRevBlock]
  const double eps = 1.0e-6, gm = d.gamlg - 1.0;
  Loaded L;
  load_cell(d, d.xs, d.ys, iq, L);
  const CellGeo G{d.rc[e], d.sc[e], d.g19[e], d.g20[e], d.g21[e]};
  double lX[3][3], lY[3][3];
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++) lX[i][j] = lY[i][j] = 0.0;
  __pipeline_wait_prior(0);
  // face integral: transpose of f = u* P0 - (P1, P2), fe = u* . f, tw = u* . t per
  // boundary node; the adjoints of the partial sums go to lP, those of u* to pbuf,
  // those of the mass-flux weights t to the nodes
  const int A[9] = {0, 2, 2, 0, 1, 2, 1, 0, 1}, B[9] = {0, 0, 2, 2, 0, 1, 2, 1, 1};
#pragma unroll
  for (int k = 0; k < 8; k++) {
    double b[6];
    node_basis2(G, k, b);
    const int pn = d.ipq[k * nq + iq];
    const double un = d.us_new[pn], vn = d.vs_new[pn];
    const double P0 = d.npart[k * nq + iq];
    const double f0 = un * P0 - d.npart[(9 + k) * nq + iq], f1 = vn * P0 - d.npart[(18 + k) * nq + iq];
    const int v = k & 3, n = (v + 1) & 3, p = (v + 3) & 3, q = 4 + p, ed = 4 + v;
    double tx, ty;
    if (k < 4)
      corner_flux(L.X[A[p]][B[p]], L.Y[A[p]][B[p]], L.X[A[q]][B[q]], L.Y[A[q]][B[q]], L.X[A[ed]][B[ed]],
                  L.Y[A[ed]][B[ed]], L.X[A[n]][B[n]], L.Y[A[n]][B[n]], tx, ty);
    else
      edge_flux(L.X[A[v]][B[v]], L.Y[A[v]][B[v]], L.X[A[n]][B[n]], L.Y[A[n]][B[n]], tx, ty);
    double ltw = 0.0, lf0 = 0.0, lf1 = 0.0, lfe = 0.0;
#pragma unroll
    for (int kk = 0; kk < 6; kk++) {
      ltw += AR(0, kk) * b[kk];
      lf0 += AR(1, kk) * b[kk];
      lf1 += AR(2, kk) * b[kk];
      lfe += AR(3, kk) * b[kk];
    }
    lf0 += lfe * un;
    lf1 += lfe * vn;
    a.lP[k * nq + iq] = lf0 * un + lf1 * vn;
    a.lP[(9 + k) * nq + iq] = -lf0;
    a.lP[(18 + k) * nq + iq] = -lf1;
    a.pbuf[(18 + k) * nq + iq] = 0.0;
    a.pbuf[(27 + k) * nq + iq] = 0.0;
    a.pbuf[(36 + k) * nq + iq] = lfe * f0 + lf0 * P0 + ltw * tx;
    a.pbuf[(45 + k) * nq + iq] = lfe * f1 + lf1 * P0 + ltw * ty;
    const double ltx = ltw * un, lty = ltw * vn;
    if (k < 4) {
      const double x2 = (2.0 * kMassCorner) * ltx, xh = (0.5 * kMassCorner) * ltx;
      const double y2 = (2.0 * kMassCorner) * lty, yh = (0.5 * kMassCorner) * lty;
      lY[A[ed]][B[ed]] += x2;
      lY[A[q]][B[q]] -= x2;
      lY[A[p]][B[p]] += xh;
      lY[A[n]][B[n]] -= xh;
      lX[A[q]][B[q]] += y2;
      lX[A[ed]][B[ed]] -= y2;
      lX[A[n]][B[n]] += yh;
      lX[A[p]][B[p]] -= yh;
    } else {
      const double xe = kMassEdge * ltx, ye = kMassEdge * lty;
      lY[A[n]][B[n]] += xe;
      lY[A[v]][B[v]] -= xe;
      lX[A[v]][B[v]] += ye;
      lX[A[n]][B[n]] -= ye;
    }
  }
#pragma unroll
  for (int v = 2; v < 6; v++) a.pbuf[(v * 9 + 8) * nq + iq] = 0.0;
#pragma unroll
  for (int v = 0; v < 3; v++) a.lP[(v * 9 + 8) * nq + iq] = 0.0;
  const double xc = L.X[1][1], yc = L.Y[1][1];
  QuadMap m, l;
  map_coeffs(L.X, m.a);
  map_coeffs(L.Y, m.b);
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++) l.a[i][j] = l.b[i][j] = 0.0;
  // volume integral
  {
    double lu[4][6];
#pragma unroll
    for (int q = 0; q < 4; q++)
#pragma unroll
      for (int k = 0; k < 6; k++) lu[q][k] = 0.0;
#pragma unroll 1
    for (int i = 0; i < 5; i++) {
      const double r = cL5[i], dr = r - G.rc, b3 = 0.5 * dr * dr - G.g19;
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
#pragma unroll
      for (int q = 0; q < 4; q++) {
        ra[q] = AU(q, 0) + AU(q, 1) * dr + AU(q, 3) * b3 - AU(q, 4) * G.g20 - AU(q, 5) * G.g21;
        rb[q] = AU(q, 2) + AU(q, 5) * dr;
      }
      // adjoints along the row: of alpha_q pa + ds pb, of beta_q qa + ds qb
      double pa[4], qa[4];
#pragma unroll
      for (int q = 0; q < 4; q++) {
        pa[q] = AR(q, 1) + dr * AR(q, 3);
        qa[q] = AR(q, 2) + dr * AR(q, 5);
      }
      double m0[4] = {0, 0, 0, 0}, m1[4] = {0, 0, 0, 0}, m2[4] = {0, 0, 0, 0};
      double Xr[3] = {0, 0, 0}, Yr[3] = {0, 0, 0}, Xs[2] = {0, 0}, Ys[2] = {0, 0};
      const double wi = cLw[i];
#pragma unroll 1
      for (int j = 0; j < 5; j++) {
        const double s = cL5[j], ds = s - G.sc, w = wi * cLw[j];
        const double jxr = xr[0] + s * (xr[1] + s * xr[2]), jyr = yr[0] + s * (yr[1] + s * yr[2]);
        const double jxs = xs[0] + s * xs[1], jys = ys[0] + s * ys[1];
        double un[4], la[4], lb[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
          un[q] = ra[q] + ds * (rb[q] + 0.5 * AU(q, 4) * ds);
          la[q] = pa[q] + ds * AR(q, 5);
          lb[q] = qa[q] + ds * AR(q, 4);
        }
        const double rho = 1.0 / un[0], kin = un[3] - 0.5 * (un[1] * un[1] + un[2] * un[2]);
        const double pe = gm * rho * kin, wp = w * fmax(eps, pe);
        const double al = jys * un[1] - jxs * un[2], be = jxr * un[2] - jyr * un[1];
        const double lal = wp * la[3] - w * la[0], lbe = wp * lb[3] - w * lb[0];
        const double lp = w * (la[1] * jys - lb[1] * jyr - la[2] * jxs + lb[2] * jxr + la[3] * al + lb[3] * be);
        const double lys = lal * un[1] + la[1] * wp, lxs = -lal * un[2] - la[2] * wp;
        const double lxr = lbe * un[2] + lb[2] * wp, lyr = -lbe * un[1] - lb[1] * wp;
        double lun[4];
        lun[1] = lal * jys - lbe * jyr;
        lun[2] = lbe * jxr - lal * jxs;
        // pressure: p = gm rho kin above the floor
        const double lk = pe > eps ? lp * gm * rho : 0.0;
        lun[3] = lk;
        lun[1] -= lk * un[1];
        lun[2] -= lk * un[2];
        lun[0] = -lk * kin * rho;
#pragma unroll
        for (int q = 0; q < 4; q++) {
          m0[q] += lun[q];
          m1[q] += lun[q] * ds;
          m2[q] += lun[q] * (ds * ds);
        }
        Xr[0] += lxr;
        Yr[0] += lyr;
        Xs[0] += lxs;
        Ys[0] += lys;
        Xr[1] += lxr * s;
        Yr[1] += lyr * s;
        Xr[2] += lxr * (s * s);
        Yr[2] += lyr * (s * s);
        Xs[1] += lxs * s;
        Ys[1] += lys * s;
      }
#pragma unroll
      for (int q = 0; q < 4; q++) {
        lu[q][0] += m0[q];
        lu[q][1] += dr * m0[q];
        lu[q][2] += m1[q];
        lu[q][3] += b3 * m0[q];
        lu[q][4] += 0.5 * m2[q] - G.g20 * m0[q];
        lu[q][5] += dr * m1[q] - G.g21 * m0[q];
      }
#pragma unroll
      for (int n = 0; n < 3; n++) {
        l.a[1][n] += Xr[n];
        l.b[1][n] += Yr[n];
        l.a[2][n] += (2.0 * r) * Xr[n];
        l.b[2][n] += (2.0 * r) * Yr[n];
      }
#pragma unroll
      for (int n = 0; n < 2; n++) {
        const double X = (n + 1.0) * Xs[n], Y = (n + 1.0) * Ys[n];
        l.a[0][n + 1] += X;
        l.b[0][n + 1] += Y;
        l.a[1][n + 1] += r * X;
        l.b[1][n + 1] += r * Y;
        l.a[2][n + 1] += (r * r) * X;
        l.b[2][n + 1] += (r * r) * Y;
      }
    }
#pragma unroll
    for (int q = 0; q < 4; q++)
#pragma unroll
      for (int k = 0; k < 6; k++) a.lU[(q * 6 + k) * nc + e] += lu[q][k];
  }
  if (d.ncase == 1) tgv_T(m, G, xc, yc, d.gamlg, &AR(3, 0), kRevBlock, l);
  map_coeffs_T(l.a, lX);
  map_coeffs_T(l.b, lY);
#pragma unroll
  for (int k = 0; k < 9; k++) {
    a.pbuf[k * nq + iq] = lX[A[k]][B[k]];
    a.pbuf[(9 + k) * nq + iq] = lY[A[k]][B[k]];
  }
#undef AU
#undef AR
}

// The reverse of the FP64 corner-face pass, four lanes per quad (lane = side, as in
// k_faces4): reads the node-sum adjoints lS at its nodes plus the RHS pass's adjoints
// of its partials (lP); adds the cell DOF adjoint into lU, writes the node
// contributions (x, y, u*_prev, v*_prev) into pbuf and the adjoints of the sub-cell
// density corrections into lcorr.  Every lane works on its two corner ends, its
// edge and its inner face; what falls to the neighbours' nodes goes over by shuffle,
// the DOF adjoints are summed so that lane q keeps equation q.  The 32 unrolled faces
// of one thread per quad took 114 us a launch on 256 x 256, this 56
// (168 registers; 2 or 4 blocks an SM 3% slower a reverse stage).
struct NodeAdj {
  double rho = 0.0, ke = 0.0, dx = 0.0, dy = 0.0;  // of 1/tau, kinetic part, u* - u
};
// p = max(eps, gm (rho + corr) ke) from its adjoint lp
__device__ __forceinline__ void pressure_T(const VState &s, double corr, double gm, double lp, NodeAdj &n, double &lcorr) {
  if (gm * (s.rho + corr) * s.ke > 1.0e-6) {
    n.rho += lp * gm * s.ke;
    lcorr += lp * gm * s.ke;
    n.ke += lp * gm * (s.rho + corr);
  }
}
constexpr int kRevFaceBlock = 128;
__global__ void __launch_bounds__(kRevFaceBlock, 3) k_a_faces4(Dev d, Adj a) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int v = t & 3, vn = (v + 1) & 3, vp = (v + 3) & 3, vo = (v + 2) & 3;
  const bool valid = (t >> 2) < d.nquad;
  const int iq = valid ? t >> 2 : d.nquad - 1, e = iq + d.ntria;
  const size_t nq = d.nquad, np = d.npoin, nc = d.ncell;
  const int pc = d.ipq[v * nq + iq], pe = d.ipq[(4 + v) * nq + iq], pm = d.ipq[8 * nq + iq];
  double u[4][6];
  load_u(d, d.Us, e, u);
  const CellGeo G{d.rc[e], d.sc[e], d.g19[e], d.g20[e], d.g21[e]};
  const double corr0 = d.corr[v * nq + iq];
  const double cx = d.xs[pc], cy = d.ys[pc], cu = d.us[pc], cv = d.vs[pc];
  const double ex = d.xs[pe], ey = d.ys[pe], eu = d.us[pe], ev = d.vs[pe];
  const double mx = d.xs[pm], my = d.ys[pm], mu = d.us[pm], mv = d.vs[pm];
  double lc[3], le[3], lm[3];
#pragma unroll
  for (int k = 0; k < 3; k++) {
    lc[k] = a.lS[k * np + pc] + a.lP[(9 * k + v) * nq + iq];
    le[k] = a.lS[k * np + pe] + a.lP[(9 * k + 4 + v) * nq + iq];
    lm[k] = a.lS[k * np + pm] + a.lP[(9 * k + 8) * nq + iq];
  }
  const double nx = lane_get(cx, vn), ny = lane_get(cy, vn), px = lane_get(cx, vp), py = lane_get(cy, vp);
  const double qx = lane_get(ex, vp), qy = lane_get(ey, vp), ox = lane_get(ex, vo), oy = lane_get(ey, vo);
  const double corr1 = lane_get(corr0, vn);
  const double eps = 1.0e-6, g = d.gamlg, gm = g - 1.0, slpdu = 0.5 * (g + 1.0);
  const double rhoct = 1.0 / u[0][0];
  const double pctr = fmax(eps, gm * rhoct * (u[3][0] - 0.5 * (u[1][0] * u[1][0] + u[2][0] * u[2][0])));
  const double sdctr = sqrt(fmax(eps, g * pctr * u[0][0]));
  const double rhoc = rhoct * sdctr, kap = d.cimpd * rhoct * slpdu, lim2 = 1.0e24 * sdctr * sdctr;
  const double c1x = 1.5 * cy - 2.0 * qy + 0.5 * py, c1y = -1.5 * cx + 2.0 * qx - 0.5 * px;
  const double c2x = -1.5 * cy + 2.0 * ey - 0.5 * ny, c2y = 1.5 * cx - 2.0 * ex + 0.5 * nx;
  const double ax = 0.5 * (ny - cy), ay = 0.5 * (cx - nx);
  const double bx = 0.75 * ey - my + 0.25 * oy, by = mx - 0.75 * ex - 0.25 * ox;
  double lrho = 0.0, lsd = 0.0, lcr0 = 0.0, lcr1 = 0.0;
  double l1x, l1y, l2x, l2y, lax, lay, lbx, lby;
  double lu[4][6];
#pragma unroll
  for (int q = 0; q < 4; q++)
#pragma unroll
    for (int k = 0; k < 6; k++) lu[q][k] = 0.0;
  // m of one face, as the corner pass takes it
  auto imp = [&](double fx, double fy, double dx, double dy) {
    const double j2 = dx * dx + dy * dy;
    const bool reg = j2 < lim2;
    return impedance(rhoc, kap, sqrt(fx * fx + fy * fy), fabs(dx * fx + dy * fy), reg, reg ? 0.0 : rsqrt(j2));
  };
  // the vertex state's adjoint into the DOFs
  auto vertex = [&](const double *b, const VState &s, const NodeAdj &n, double lsu, double lsv) {
    const double st0 = -n.rho * s.rho * s.rho;
    const double lst[4] = {st0, lsu - n.dx - n.ke * s.u, lsv - n.dy - n.ke * s.v, n.ke};
#pragma unroll
    for (int q = 0; q < 4; q++)
#pragma unroll
      for (int k = 0; k < 6; k++)
        if (k < d.mdegr) lu[q][k] += lst[q] * b[k];
  };
  double b[6];
  NodeAdj nc_, ne_, nm_;
  {
    // corner: C1 and C2 with weight 1/6 each
    basis_at(G, v == 1 || v == 2 ? 1.0 : -1.0, v >= 2 ? 1.0 : -1.0, b);
    const VState s = vertex_state(u, b, d.mdegr);
    const double dx = cu - s.u, dy = cv - s.v;
    const double P0 = (1.0 / 3.0) * (imp(c1x, c1y, dx, dy) + imp(c2x, c2y, dx, dy));
    const double pw = (-1.0 / 3.0) * fmax(eps, gm * (s.rho + corr0) * s.ke);
    const double lmm = lc[0] + lc[1] * s.u + lc[2] * s.v;
    l1x = l2x = -lc[1] * pw;
    l1y = l2y = -lc[2] * pw;
    pressure_T(s, corr0, gm, (1.0 / 3.0) * (lc[1] * (c1x + c2x) + lc[2] * (c1y + c2y)), nc_, lcr0);
    corner_m_T(rhoct, sdctr, d.cimpd, slpdu, dx, dy, c1x, c1y, 1.0 / 6.0, lmm, lrho, lsd, nc_.dx, nc_.dy, l1x, l1y);
    corner_m_T(rhoct, sdctr, d.cimpd, slpdu, dx, dy, c2x, c2y, 1.0 / 6.0, lmm, lrho, lsd, nc_.dx, nc_.dy, l2x, l2y);
    vertex(b, s, nc_, lc[1] * P0, lc[2] * P0);
  }
  {
    // edge node: A with weight 1/3, B with 2/3, in both sub-cells
    basis_at(G, v == 1 ? 1.0 : v == 3 ? -1.0 : 0.0, v == 2 ? 1.0 : v == 0 ? -1.0 : 0.0, b);
    const VState s = vertex_state(u, b, d.mdegr);
    const double dx = eu - s.u, dy = ev - s.v;
    const double P0 = (4.0 / 3.0) * imp(ax, ay, dx, dy) + (8.0 / 3.0) * imp(bx, by, dx, dy);
    const double p0 = fmax(eps, gm * (s.rho + corr0) * s.ke), p1 = fmax(eps, gm * (s.rho + corr1) * s.ke);
    const double wa = (-2.0 / 3.0) * (p0 + p1), wb = (4.0 / 3.0) * (p0 - p1);
    const double lmm = le[0] + le[1] * s.u + le[2] * s.v;
    lax = -le[1] * wa;
    lay = -le[2] * wa;
    lbx = -le[1] * wb;
    lby = -le[2] * wb;
    const double lwa = -(le[1] * ax + le[2] * ay), lwb = -(le[1] * bx + le[2] * by);
    pressure_T(s, corr0, gm, (-2.0 / 3.0) * lwa + (4.0 / 3.0) * lwb, ne_, lcr0);
    pressure_T(s, corr1, gm, (-2.0 / 3.0) * lwa - (4.0 / 3.0) * lwb, ne_, lcr1);
    corner_m_T(rhoct, sdctr, d.cimpd, slpdu, dx, dy, ax, ay, 2.0 / 3.0, lmm, lrho, lsd, ne_.dx, ne_.dy, lax, lay);
    corner_m_T(rhoct, sdctr, d.cimpd, slpdu, dx, dy, bx, by, 4.0 / 3.0, lmm, lrho, lsd, ne_.dx, ne_.dy, lbx, lby);
    vertex(b, s, ne_, le[1] * P0, le[2] * P0);
  }
  {
    // centre: the lane's share, B with weight 1/4 out of v, into v + 1
    basis_at(G, 0.0, 0.0, b);
    const VState s = vertex_state(u, b, d.mdegr);
    const double dx = mu - s.u, dy = mv - s.v;
    const double M0 = imp(bx, by, dx, dy);
    const double dp = fmax(eps, gm * (s.rho + corr0) * s.ke) - fmax(eps, gm * (s.rho + corr1) * s.ke);
    const double lmm = lm[0] + lm[1] * s.u + lm[2] * s.v, ldp = -0.5 * (lm[1] * bx + lm[2] * by);
    lbx -= 0.5 * dp * lm[1];
    lby -= 0.5 * dp * lm[2];
    pressure_T(s, corr0, gm, ldp, nm_, lcr0);
    pressure_T(s, corr1, gm, -ldp, nm_, lcr1);
    corner_m_T(rhoct, sdctr, d.cimpd, slpdu, dx, dy, bx, by, 0.5, lmm, lrho, lsd, nm_.dx, nm_.dy, lbx, lby);
    vertex(b, s, nm_, lm[1] * M0, lm[2] * M0);
  }
  centre_T(u, g, lrho, lsd, lu);  // linear in the lane's shares
  // node coordinates: the lane's corner and edge node from itself and its neighbours
  double gcx = 1.5 * (l2y - l1y) + 0.5 * lay, gcy = 1.5 * (l1x - l2x) - 0.5 * lax;
  double gex = -2.0 * l2y - 0.75 * lby, gey = 2.0 * l2x + 0.75 * lbx;
  gcx += lane_get(0.5 * l2y - 0.5 * lay, vp) + lane_get(-0.5 * l1y, vn);
  gcy += lane_get(0.5 * lax - 0.5 * l2x, vp) + lane_get(0.5 * l1x, vn);
  gex += lane_get(2.0 * l1y, vn) + lane_get(-0.25 * lby, vo);
  gey += lane_get(-2.0 * l1x, vn) + lane_get(0.25 * lbx, vo);
  const double gmx = lane_sum(lby), gmy = -lane_sum(lbx), mdx = lane_sum(nm_.dx), mdy = lane_sum(nm_.dy);
  const double lcr = lcr0 + lane_get(lcr1, vp);
  // lane v keeps equation v
  double T[2][6], lq[6];
#pragma unroll
  for (int q = 0; q < 2; q++)
#pragma unroll
    for (int k = 0; k < 6; k++) {
      const double mine = v & 2 ? lu[q + 2][k] : lu[q][k], other = v & 2 ? lu[q][k] : lu[q + 2][k];
      T[q][k] = mine + __shfl_xor_sync(0xffffffffu, other, 2);
    }
#pragma unroll
  for (int k = 0; k < 6; k++) {
    const double mine = v & 1 ? T[1][k] : T[0][k], other = v & 1 ? T[0][k] : T[1][k];
    lq[k] = mine + __shfl_xor_sync(0xffffffffu, other, 1);
  }
  if (!valid) return;
  double *pb = a.pbuf + iq;
  const double rc4[4] = {gcx, gcy, nc_.dx, nc_.dy}, re4[4] = {gex, gey, ne_.dx, ne_.dy}, rm4[4] = {gmx, gmy, mdx, mdy};
#pragma unroll
  for (int k = 0; k < 6; k++) {
    pb[(9 * k + v) * nq] = k < 4 ? rc4[k < 4 ? k : 0] : 0.0;
    pb[(9 * k + 4 + v) * nq] = k < 4 ? re4[k < 4 ? k : 0] : 0.0;
    if (v == 0) pb[(9 * k + 8) * nq] = k < 4 ? rm4[k < 4 ? k : 0] : 0.0;
    a.lU[(v * 6 + k) * nc + e] += lq[k];
  }
  a.lcorr[v * nq + iq] = lcr;
}

// The transpose of f_corner_corr, corr = cdrho (msub - masel) / area with masel = sum
// w det J / tau, from lcorr: adds into the tau DOF adjoints and the node contributions.
// One division per row of five points; both halves of a row share its sums; det J
// hands its adjoint to the map.  256 x 256: 60 -> 33 us a launch
// (128 registers, 216 bytes of spills; 4 or 6 blocks of 64 an SM 3% slower a sweep).
constexpr int kRevCorrBlock = 64;
__global__ void __launch_bounds__(kRevCorrBlock, 8) k_a_corr64(Dev d, Adj a) {
  const int iq = blockIdx.x * kRevCorrBlock + threadIdx.x;
  if (iq >= d.nquad) return;
  const int e = iq + d.ntria;
  const size_t nq = d.nquad, nc = d.ncell;
  double u[6], lm[4], la[4];
#pragma unroll
  for (int k = 0; k < 6; k++) u[k] = d.Us[k * nc + e];
#pragma unroll
  for (int k = 0; k < 4; k++) {
    lm[k] = a.lcorr[k * nq + iq];
    la[k] = -lm[k] * d.corr[k * nq + iq];
  }
  const CellGeo G{d.rc[e], d.sc[e], d.g19[e], d.g20[e], d.g21[e]};
  QuadMap m, l;
  load_map(d, iq, m);
  double D[4][4], lD[4][4], lq[6] = {0, 0, 0, 0, 0, 0};
  map_det(m, D);
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int n = 0; n < 4; n++) lD[i][n] = 0.0;
  const double b3 = 0.5 * G.rc * G.rc - G.g19, b4 = 0.5 * G.sc * G.sc - G.g20, b5 = G.rc * G.sc - G.g21;
  const double q0 = u[0] - u[1] * G.rc - u[2] * G.sc + u[3] * b3 + u[4] * b4 + u[5] * b5;
  const double q1 = u[1] - u[3] * G.rc - u[5] * G.sc, q2 = u[2] - u[4] * G.sc - u[5] * G.rc;
  const double q3 = 0.5 * u[3], t2 = 0.5 * u[4];
#pragma unroll
  for (int h = 0; h < 2; h++) {
    const double sg = h == 0 ? -1.0 : 1.0;
    const int is[2] = {h == 0 ? 0 : 1, h == 0 ? 3 : 2};  // s in [-1, 0], [0, 1]
    // the areas
    double F[4], lF[4], lms[2];
#pragma unroll
    for (int n = 0; n < 4; n++)
      F[n] = D[0][n] + (1.0 / 3.0) * D[2][n] + sg * (0.5 * D[1][n] + 0.25 * D[3][n]);
    const double ev = F[0] + (1.0 / 3.0) * F[2], od = 0.5 * F[1] + 0.25 * F[3];
    const double r0 = 1.0 / (ev - od), r1 = 1.0 / (ev + od);
    const double l0 = la[is[0]] * r0, l1 = la[is[1]] * r1;
    lms[0] = -d.cdrho * lm[is[0]] * r0;
    lms[1] = -d.cdrho * lm[is[1]] * r1;
    lF[0] = l0 + l1;
    lF[2] = (1.0 / 3.0) * lF[0];
    lF[1] = 0.5 * (l1 - l0);
    lF[3] = 0.25 * (l1 - l0);
#pragma unroll
    for (int n = 0; n < 4; n++) {
      lD[0][n] += lF[n];
      lD[1][n] += (0.5 * sg) * lF[n];
      lD[2][n] += (1.0 / 3.0) * lF[n];
      lD[3][n] += (0.25 * sg) * lF[n];
    }
#pragma unroll 1
    for (int i = 0; i < 5; i++) {
      const double r = 0.5 * cG5[i] + 0.5 * sg, wi = 0.25 * cW5[i];
      double c[4];
      det_row(D, r, c);
      const double t0 = q0 + r * (q1 + r * q3), t1 = q2 + r * u[5];
      double m0 = 0.0, m1 = 0.0, m2 = 0.0, Ls[4] = {0, 0, 0, 0};
#pragma unroll
      for (int k = 0; k < 2; k++) {
        const double lw = wi * lms[k];
        double tau[5], pre[5];
#pragma unroll
        for (int j = 0; j < 5; j++) {
          const double s = 0.5 * g5p(j) + (k == 0 ? -0.5 : 0.5);
          tau[j] = t0 + s * (t1 + s * t2);
          pre[j] = j == 0 ? tau[0] : pre[j - 1] * tau[j];
        }
        double inv = 1.0 / pre[4];
#pragma unroll
        for (int j = 4; j >= 0; j--) {
          const double s = 0.5 * g5p(j) + (k == 0 ? -0.5 : 0.5);
          const double it = j > 0 ? inv * pre[j > 0 ? j - 1 : 0] : inv;
          inv *= tau[j];
          const double det = c[0] + s * (c[1] + s * (c[2] + s * c[3]));
          const double ld = (lw * g5w(j)) * it, lt = -(ld * it) * det;
          m0 += lt;
          m1 += lt * s;
          m2 += lt * (s * s);
          Ls[0] += ld;
          Ls[1] += ld * s;
          Ls[2] += ld * (s * s);
          Ls[3] += ld * (s * s * s);
        }
      }
      lq[0] += m0;
      lq[1] += r * m0;
      lq[2] += m1;
      lq[3] += (r * r) * m0;
      lq[4] += m2;
      lq[5] += r * m1;
      double rp = 1.0;
#pragma unroll
      for (int k = 0; k < 4; k++) {
#pragma unroll
        for (int n = 0; n < 4; n++) lD[k][n] += rp * Ls[n];
        rp *= r;
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++) l.a[i][j] = l.b[i][j] = 0.0;
  map_det_T(m, lD, l);
  double lX[3][3], lY[3][3];
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++) lX[i][j] = lY[i][j] = 0.0;
  map_coeffs_T(l.a, lX);
  map_coeffs_T(l.b, lY);
  const int A[9] = {0, 2, 2, 0, 1, 2, 1, 0, 1}, B[9] = {0, 0, 2, 2, 0, 1, 2, 1, 1};
#pragma unroll
  for (int k = 0; k < 9; k++) {
    a.pbuf[k * nq + iq] += lX[A[k]][B[k]];
    a.pbuf[(9 + k) * nq + iq] += lY[A[k]][B[k]];
  }
  double *o = a.lU + e;
  o[0] += lq[0];
  o[nc] += lq[1] - G.rc * lq[0];
  o[2 * nc] += lq[2] - G.sc * lq[0];
  o[3 * nc] += b3 * lq[0] - G.rc * lq[1] + 0.5 * lq[3];
  o[4 * nc] += b4 * lq[0] - G.sc * lq[2] + 0.5 * lq[4];
  o[5 * nc] += b5 * lq[0] - G.sc * lq[1] - G.rc * lq[2] + lq[5];
}
