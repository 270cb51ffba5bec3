// The optimised RZ stage of the linear P1 path (order_exact 0; GEO 1: true volume,
// 2: area-weighted), and the time step, motion and volumes of the plane branch
// (GEO 0), whose other passes are lag2d_p1.cu's FAST forms.
// Included by lag2d_p1.cu inside namespace lag2d::p1; the reference-order kernels
// beside it stay for order_exact.
//
// On the meshes this path is run on (about 10,000 cells) every kernel is one
// wave, so a step's time is launches times the dependent chain of a thread.  A
// stage is three launches (cell, node, RHS) instead of seven to nine:
//   cell  four lanes per cell, lane = vertex: node bounds over the cells around
//         the vertex (no kernel of their own), limiter, corner coefficients;
//         area-weighted: mass centre and mass matrix with the quadrature rows
//         spread over the lanes
//   node  gather, solve, walls, and the motion once dt is known
//   RHS   one thread per cell: face and volume integral, M^-1 and the update
// Stage 1 adds the time step (finished by its last block) and the motion, which
// runs beside the RHS; volumes run beside the last RHS.
//
// Quadratures.  A straight quad's map is bilinear: x_r = e1 + e3 s, x_s = e2 +
// e3 r, det J = j0 + j1 r + j2 s.  Everything polynomial is integrated in closed
// form (the 5- and 6-point Gauss sums of the reference are exact for it): areas,
// RZ volumes and their centres, the volume-change moments.  What is left is the
// pressure at the 25 points, of which six moments (1, r, s, r^2, rs, s^2) give
// every integral with it, with one division per row of points.

// 1-D Gauss rules (ruqope), positions and weights
__device__ __forceinline__ double g5x(int i) {
  const double t[5] = {-0.9061798459386639927976269, -0.5384693101056830910363144, 0.0, 0.5384693101056830910363144,
                       0.9061798459386639927976269};
  return t[i];
}
__device__ __forceinline__ double g5wt(int i) {
  const double t[5] = {0.2369268850561890875142640, 0.4786286704993664680412915, 0.5688888888888888888888889,
                       0.4786286704993664680412915, 0.2369268850561890875142640};
  return t[i];
}
__device__ __forceinline__ double g6x(int i) {
  const double t[6] = {-0.9324695142031520278123016, -0.6612093864662645136613996, -0.2386191860831969086305017,
                       0.2386191860831969086305017, 0.6612093864662645136613996, 0.9324695142031520278123016};
  return t[i];
}
__device__ __forceinline__ double g6wt(int i) {
  const double t[6] = {0.1713244923791704, 0.3607615730481386, 0.4679139345726910, 0.4679139345726910,
                       0.3607615730481386, 0.1713244923791704};
  return t[i];
}

// the bilinear map: x_r = e1 + e3 s, x_s = e2 + e3 r, y alike with f; y at the
// origin yc, det J = j0 + j1 r + j2 s
struct Bilin {
  double e1, e2, e3, f1, f2, f3, yc, j0, j1, j2;
};
__device__ __forceinline__ Bilin bilin(const double *x, const double *y) {
  Bilin b;
  b.e1 = 0.25 * (-x[0] + x[1] + x[2] - x[3]);
  b.e2 = 0.25 * (-x[0] - x[1] + x[2] + x[3]);
  b.e3 = 0.25 * (x[0] - x[1] + x[2] - x[3]);
  b.f1 = 0.25 * (-y[0] + y[1] + y[2] - y[3]);
  b.f2 = 0.25 * (-y[0] - y[1] + y[2] + y[3]);
  b.f3 = 0.25 * (y[0] - y[1] + y[2] - y[3]);
  b.yc = 0.25 * (y[0] + y[1] + y[2] + y[3]);
  b.j0 = b.e1 * b.f2 - b.f1 * b.e2;
  b.j1 = b.e1 * b.f3 - b.f1 * b.e3;
  b.j2 = b.e3 * b.f2 - b.f3 * b.e2;
  return b;
}
// volume (RZ: per radian, weight y) of the cell
template <int GEO>
__device__ __forceinline__ double cell_volume(const Bilin &b) {
  if (GEO == 0) return 4.0 * b.j0;
  return 4.0 * b.j0 * b.yc + (4.0 / 3.0) * (b.j1 * b.f1 + b.j2 * b.f2);
}

// Face weights of corner iv's two edges (a to the previous vertex, b to the
// next): the share own that weighs the corner's own basis and the share oth that
// weighs the other end's, of the edge's area vector.  nrz = 1: the radius weights of
// the four corner faces (Getrhslagmc.f90:18534-18734); nrz = 2: (2 b_own + b_oth) / 6
// (Getrhslagrz.f90:1673-1812).
template <int GEO>
__device__ __forceinline__ void edge_weights(double ri, double rj, double &own, double &oth) {
  if (GEO == 1) { own = (1.0 / 12.0) * (3.0 * ri + rj); oth = (1.0 / 12.0) * (ri + rj); }
  else { own = 1.0 / 3.0; oth = 1.0 / 6.0; }
}

__device__ __forceinline__ double pressure(double g, double tau, double u, double v, double e, double floor_) {
  return fmax(floor_, (g - 1.0) / tau * (e - 0.5 * (u * u + v * v)));
}

// corner coefficients: rows cf[(row*4 + iv)*nquad + iq]; the node pass reads
// 0-4, the RHS 1-2 and 5-7
constexpr int CF_P0 = 0, CF_U = 1, CF_V = 2, CF_S1 = 3, CF_S2 = 4, CF_MA = 5, CF_MB = 6, CF_P = 7;

// ---------------------------------------------------------------------------
// cell: four lanes per cell
// ---------------------------------------------------------------------------
__device__ __forceinline__ double quad_min(double v) {
  v = fmin(v, __shfl_xor_sync(0xffffffffu, v, 1));
  return fmin(v, __shfl_xor_sync(0xffffffffu, v, 2));
}
__device__ __forceinline__ double quad_sum(double v) {
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  return v + __shfl_xor_sync(0xffffffffu, v, 2);
}
__device__ __forceinline__ double quad_get(double v, int lane) { return __shfl_sync(0xffffffffu, v, lane, 4); }

// nrz = 2: the mass centre of the limited density over the cell's area (5
// fixed-point passes of 36 points, Getrhslagrz.f90:4812-4994; the first, with the
// cell-average density, is the area centroid) and M^-1 of the area mass matrix
// about it over geoel(11) (25 points, :3949-4219).  tau along a row is linear, so
// a row needs one division; the rows are spread over the cell's lanes.
__device__ __forceinline__ void area_centre(const Dev1 &d, int e, int iv, bool live, const Bilin &B, double t0, double t1,
                                            double t2, double &rc, double &sc) {
  rc = B.j1 / (3.0 * B.j0);
  sc = B.j2 / (3.0 * B.j0);
  const double scale = t0 / (4.0 * B.j0);  // 1 / masel
#pragma unroll 1
  for (int pass = 1; pass < 5; pass++) {
    const double c0 = t0 - t1 * rc - t2 * sc;
    double sx = 0.0, sy = 0.0;
#pragma unroll 1
    for (int i = iv; i < 6; i += 4) {
      const double r = g6x(i), tr = c0 + t1 * r, dr = B.j0 + B.j1 * r;
      double pre[6], t[6];
#pragma unroll
      for (int j = 0; j < 6; j++) {
        t[j] = tr + t2 * g6x(j);
        pre[j] = j == 0 ? t[0] : pre[j - 1] * t[j];
      }
      double inv = 1.0 / pre[5], a0 = 0.0, a1 = 0.0;
#pragma unroll
      for (int j = 5; j >= 0; j--) {
        const double rho = j > 0 ? inv * pre[j > 0 ? j - 1 : 0] : inv;
        const double m = g6wt(j) * rho * (dr + B.j2 * g6x(j));
        a0 += m;
        a1 += m * g6x(j);
        inv *= t[j];
      }
      sx += g6wt(i) * r * a0;
      sy += g6wt(i) * a1;
    }
    rc = quad_sum(sx) * scale;
    sc = quad_sum(sy) * scale;
  }
  const double c0 = t0 - t1 * rc - t2 * sc;
  double f0 = 0.0, f1 = 0.0, f2 = 0.0, f3 = 0.0;
#pragma unroll 1
  for (int i = iv; i < 5; i += 4) {
    const double r = g5x(i), tr = c0 + t1 * r, dr = B.j0 + B.j1 * r, br = r - rc;
    double pre[5], t[5];
#pragma unroll
    for (int j = 0; j < 5; j++) {
      t[j] = tr + t2 * g5x(j);
      pre[j] = j == 0 ? t[0] : pre[j - 1] * t[j];
    }
    double inv = 1.0 / pre[4], a0 = 0.0, a1 = 0.0, a2 = 0.0;
#pragma unroll
    for (int j = 4; j >= 0; j--) {
      const double rho = j > 0 ? inv * pre[j > 0 ? j - 1 : 0] : inv;
      const double m = g5wt(j) * rho * (dr + B.j2 * g5x(j)), bs = g5x(j) - sc;
      a0 += m;
      a1 += m * bs;
      a2 += m * bs * bs;
      inv *= t[j];
    }
    f0 += g5wt(i) * a0;
    f1 += g5wt(i) * br * br * a0;
    f2 += g5wt(i) * br * a1;
    f3 += g5wt(i) * a2;
  }
  f0 = quad_sum(f0);
  f1 = quad_sum(f1);
  f2 = quad_sum(f2);
  f3 = quad_sum(f3);
  // the lanes past the end repeat the last cell, whose centre other warps may still read
  if (!live) return;
  const double rb = cell_volume<2>(B) / (4.0 * B.j0), det = (f1 * f3 - f2 * f2) * rb;
  d.amatr[iv * (size_t)d.ncell + e] = iv == 0 ? f3 / det : iv == 1 ? -f2 / det : iv == 2 ? f1 / det : 1.0 / (f0 * rb);
  if (iv == 0) d.rc[e] = rc;
  if (iv == 1) d.sc[e] = sc;
}

constexpr int kCellThreads = 128;
template <int GEO>
__global__ void __launch_bounds__(kCellThreads) k1f_cell(Dev1 d, int stage, int itime) {
  const int t = blockIdx.x * kCellThreads + threadIdx.x, iv = threadIdx.x & 3;
  const bool live = (t >> 2) < d.nquad;
  const int e = live ? t >> 2 : d.nquad - 1;  // lanes past the end repeat the last cell and store nothing
  const size_t nc = d.ncell;
  const Scalars *S = d.sc_dev;
  const int p = d.ipq[iv * nc + e];
  const int b0 = d.esuv_ptr[p], b1 = d.esuv_ptr[p + 1];
  const int cls = d.ncase != 1 ? d.wall[p] : 0;
  int ce[4];
#pragma unroll
  for (int j = 0; j < 4; j++) ce[j] = b0 + j < b1 ? d.esuv[b0 + j] : e;
  await_previous();  // the RHS pass before, in a step's first stage its exit test
  const int done = S->done, now = S->itime;
  double u[4][ND];
#pragma unroll
  for (int q = 0; q < 4; q++)
#pragma unroll
    for (int k = 0; k < ND; k++) u[q][k] = d.Us[(q * ND + k) * nc + e];
  const double pctr_s = d.pbar[e];
  double rc = d.rc[e], sc = d.sc[e];
  const double x = d.xs[p], y = d.ys[p], us0 = d.us[p], vs0 = d.vs[p];
  // the averages around the vertex; entries past the list repeat the cell itself
  double uj[4], vj[4], mx[5], mn[5];
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const double v[5] = {d.Us[ce[j]], d.Us[3 * nc + ce[j]], d.Us[6 * nc + ce[j]], d.pbar[ce[j]], d.Us[9 * nc + ce[j]]};
    uj[j] = v[1];
    vj[j] = v[2];
#pragma unroll
    for (int q = 0; q < 5; q++) {
      mx[q] = j == 0 ? v[q] : fmax(mx[q], v[q]);
      mn[q] = j == 0 ? v[q] : fmin(mn[q], v[q]);
    }
  }
  for (int i = b0 + 4; i < b1; i++) {
    const int c = d.esuv[i];
    const double v[5] = {d.Us[c], d.Us[3 * nc + c], d.Us[6 * nc + c], d.pbar[c], d.Us[9 * nc + c]};
#pragma unroll
    for (int q = 0; q < 5; q++) {
      mx[q] = fmax(mx[q], v[q]);
      mn[q] = fmin(mn[q], v[q]);
    }
  }
  if (done) return;
  const double g = d.gamlg;
  const int md = d.mdegr;
  double X[4], Y[4];
#pragma unroll
  for (int k = 0; k < 4; k++) {
    X[k] = quad_get(x, k);
    Y[k] = quad_get(y, k);
  }
  const Bilin B = bilin(X, Y);
  const double xi = (iv == 0 || iv == 3) ? -1.0 : 1.0, eta = iv < 2 ? -1.0 : 1.0;
  // unlimited vertex state
  double w[4];
#pragma unroll
  for (int q = 0; q < 4; q++)
    w[q] = u[q][0] + (md > 1 ? u[q][1] * (xi - rc) : 0.0) + (md > 2 ? u[q][2] * (eta - sc) : 0.0);
  const double tau0 = u[0][0], uc = u[1][0], vc = u[2][0], ec = u[3][0];
  const double pv_s = pressure(g, w[0], w[1], w[2], w[3], EPS_S);
  // (1) aflim(1), aflim(4) against the node bounds (Limiterlag.f90:69-188)
  const double af1 = quad_min(barthfct1(mx[0], mn[0], tau0, w[0] - tau0));
  const double af4 = quad_min(barthfct1(mx[3], mn[3], pctr_s, pv_s - pctr_s));
  // (2) the velocity limited in the principal frame of the strain rate
  // (barthlimit_sympre_quadlb, Limiterlag.f90:8242-8692)
  double m11 = 0.0, m12 = 0.0, m21 = 0.0, m22 = 0.0;
  {
    const double xr = B.e1 + B.e3 * sc, xs = B.e2 + B.e3 * rc, yr = B.f1 + B.f3 * sc, ys = B.f2 + B.f3 * rc;
    const double rj = 1.0 / (xr * ys - yr * xs);
    const double rx = ys * rj, ry = -xs * rj, sx = -yr * rj, sy = xr * rj;
    const double a = u[1][1] * rx + u[1][2] * sx, dd = u[2][1] * ry + u[2][2] * sy;
    const double c = 0.5 * ((u[1][1] * ry + u[1][2] * sy) + (u[2][1] * rx + u[2][2] * sx));
    if (fabs(c) > 1.0e-8) {
      const double tr = a + dd, rad = sqrt(0.25 * (tr * tr) - (a * dd - c * c));
      const double l1 = (0.5 * tr + rad) - dd, l2 = (0.5 * tr - rad) - dd;
      const double n1 = 1.0 / sqrt(l1 * l1 + c * c), n2 = 1.0 / sqrt(l2 * l2 + c * c);
      const double a1 = l1 * n1, c1 = c * n1, a2 = l2 * n2, c2 = c * n2;
      if (c > 0.0) { m11 = a1; m12 = c1; m21 = a2; m22 = c2; }
      else { m21 = a1; m22 = c1; m11 = a2; m12 = c2; }
    }
  }
  double fl1, fl2;
  {
    const double ur0 = uc * m11 + vc * m12, vr0 = uc * m21 + vc * m22;
    double mx1 = ur0, mx2 = vr0, mn1 = ur0, mn2 = vr0;
    auto take = [&](double a, double b) {
      const double ul = a * m11 + b * m12, vl = a * m21 + b * m22;
      mx1 = fmax(mx1, ul);
      mx2 = fmax(mx2, vl);
      mn1 = fmin(mn1, ul);
      mn2 = fmin(mn2, vl);
    };
    auto images = [&](double a, double b) {
      take(a, b);
      if (cls == 3 || cls == 10) take(a, -b);
      if (cls == 2 || cls == 10) take(-a, b);
      if (cls == 10) take(-a, -b);
    };
#pragma unroll
    for (int j = 0; j < 4; j++)
      if (b0 + j < b1) images(uj[j], vj[j]);
    for (int i = b0 + 4; i < b1; i++) images(d.Us[3 * nc + d.esuv[i]], d.Us[6 * nc + d.esuv[i]]);
    fl1 = quad_min(barthfct1(mx1, mn1, ur0, (w[1] * m11 + w[2] * m12) - ur0));
    fl2 = quad_min(barthfct1(mx2, mn2, vr0, (w[1] * m21 + w[2] * m22) - vr0));
  }
  const double fi11 = (m11 * m11) * fl1 + (m21 * m21) * fl2;
  const double fi12 = m11 * m12 * fl1 + m21 * m22 * fl2;
  const double fi22 = (m12 * m12) * fl1 + (m22 * m22) * fl2;
  // (3) aflim(5): the energy of the limited vertex state (Limiterlag.f90:290-380)
  double af5;
  {
    const double tl = tau0 + af1 * (w[0] - tau0), pl = pctr_s + af4 * (pv_s - pctr_s);
    const double e5 = pl / (g - 1.0) * tl + 0.5 * (w[1] * w[1] + w[2] * w[2]);
    af5 = quad_min(barthfct1(mx[4], mn[4], ec, e5 - ec));
  }
  if (live) {
    if (iv == 0) { d.lim[0 * nc + e] = af1; d.lim[4 * nc + e] = fi12; }
    else if (iv == 1) { d.lim[1 * nc + e] = af4; d.lim[5 * nc + e] = fi12; }
    else if (iv == 2) { d.lim[2 * nc + e] = af5; d.lim[6 * nc + e] = fi22; }
    else d.lim[3 * nc + e] = fi11;
  }
  if (GEO == 2) {
    // the stage's mass centre and mass matrix: every stage but the first of step 1
    if (stage > 1 || (itime < 0 ? now + 1 : itime) > 1) {
      const double t1 = md > 1 ? af1 * u[0][1] : 0.0, t2 = md > 2 ? af1 * u[0][2] : 0.0;
      area_centre(d, e, iv, live, B, tau0, t1, t2, rc, sc);
#pragma unroll
      for (int q = 0; q < 4; q++)
        w[q] = u[q][0] + (md > 1 ? u[q][1] * (xi - rc) : 0.0) + (md > 2 ? u[q][2] * (eta - sc) : 0.0);
    }
  }
  // (4) corner coefficients of vertex iv: edges a (from the previous vertex) and b
  const double floor_ = GEO == 1 ? 1.0e-9 : 1.0e-8;
  const double pctr = pressure(g, tau0, uc, vc, ec, floor_);
  const double snd = sqrt(fmax(floor_, g * pctr * tau0)), rho = 1.0 / tau0;
  const double pl = pctr + af4 * (pressure(g, w[0], w[1], w[2], w[3], floor_) - pctr);
  const double br = xi - rc, bs = eta - sc;
  const double ul = uc + (fi11 * u[1][1] + fi12 * u[2][1]) * br + (fi11 * u[1][2] + fi12 * u[2][2]) * bs;
  const double vl = vc + (fi12 * u[1][1] + fi22 * u[2][1]) * br + (fi12 * u[1][2] + fi22 * u[2][2]) * bs;
  const int ip = (iv + 3) & 3, in = (iv + 1) & 3;
  const double xp = quad_get(x, ip), yp = quad_get(y, ip), xn = quad_get(x, in), yn = quad_get(y, in);
  const double ax = y - yp, ay = xp - x, bx = yn - y, by = x - xn;  // outward area vectors of the edges
  const double dx = us0 - ul, dy = vs0 - vl, j2 = dx * dx + dy * dy;
  const double la = sqrt(ax * ax + ay * ay), lb = sqrt(bx * bx + by * by);
  const double da = fabs(dx * ax + dy * ay), db = fabs(dx * bx + dy * by);
  double ma = rho * snd * la, mb = rho * snd * lb;
  if (!(j2 < 1.0e24 * snd * snd)) {  // getriecoef_matrixnew's jump direction: times |n . du| / |du|
    const double rj = 1.0 / sqrt(j2);
    ma *= da / la * rj;
    mb *= db / lb * rj;
  }
  double oa, na, ob, nb_;
  edge_weights<GEO>(fabs(y), fabs(yp), oa, na);
  edge_weights<GEO>(fabs(y), fabs(yn), ob, nb_);
  if (!live) return;
  double *o = d.cf + iv * nc + e;
  o[CF_P0 * 4 * nc] = ma * (oa + na) + mb * (ob + nb_);
  o[CF_U * 4 * nc] = ul;
  o[CF_V * 4 * nc] = vl;
  o[CF_S1 * 4 * nc] = -pl * (ax * (oa + na) + bx * (ob + nb_));
  o[CF_S2 * 4 * nc] = -pl * (ay * (oa + na) + by * (ob + nb_));
  o[CF_MA * 4 * nc] = ma;
  o[CF_MB * 4 * nc] = mb;
  o[CF_P * 4 * nc] = pl;
}

// ---------------------------------------------------------------------------
// node: gather, solve, walls (and motion)
// ---------------------------------------------------------------------------
struct NodeSum {
  double m, a1, a2, s1, s2;
};
__device__ __forceinline__ void corner_add(const Dev1 &d, int c, NodeSum &n) {
  const size_t nc = d.ncell;
  const double *o = d.cf + (c & 3) * nc + (c >> 2);
  const double m = o[CF_P0 * 4 * nc];
  n.m += m;
  n.a1 += m * o[CF_U * 4 * nc];
  n.a2 += m * o[CF_V * 4 * nc];
  n.s1 += o[CF_S1 * 4 * nc];
  n.s2 += o[CF_S2 * 4 * nc];
}
template <int GEO, bool MOVE>
__global__ void __launch_bounds__(64) k1f_node(Dev1 d, double alfa) {
  const int p = blockIdx.x * 64 + threadIdx.x;
  if (p >= d.npoin) return;
  const int done = d.sc_dev->done;
  const int b = d.ncor_ptr[p], en = d.ncor_ptr[p + 1];
  double us = d.us[p], vs = d.vs[p];
  const unsigned char bc = d.bc[p];
  const double dt = MOVE ? d.sc_dev->dtfix : 0.0;
  double xn = 0.0, yn = 0.0, xs = 0.0, ys = 0.0;
  if (MOVE) {
    xn = d.xn[p];
    yn = d.yn[p];
    xs = d.xs[p];
    ys = d.ys[p];
  }
  int c[4];
#pragma unroll
  for (int j = 0; j < 4; j++) c[j] = b + j < en ? d.ncor[b + j] : 0;
  await_previous();  // the cell pass: corner coefficients
  if (done) return;
  NodeSum n{0.0, 0.0, 0.0, 0.0, 0.0};
#pragma unroll
  for (int j = 0; j < 4; j++)
    if (b + j < en) corner_add(d, c[j], n);
  for (int i = b + 4; i < en; i++) corner_add(d, d.ncor[i], n);
  // boundary forces (getbc_lagmaire2, Getrhslag.f90:11269-11491; area-weighted:
  // GetBClag.f90:57-250): the walls' area vectors (code 22), whose normal
  // velocity the force removes, and the pressure of code 21 (ncase 3)
  double bvx = 0.0, bvy = 0.0, bpx = 0.0, bpy = 0.0;
  bool wall22 = false;
  for (int i = d.bf_ptr[p]; i < d.bf_ptr[p + 1]; i++) {
    const int f = d.bf_list[i], q0 = d.bfn[f], q1 = d.bfn[d.nbfac + f], code = d.bfcode[f];
    const double x0 = d.xs[q0], y0 = d.ys[q0], x1 = d.xs[q1], y1 = d.ys[q1];
    const double nx = y1 - y0, ny = x0 - x1, len = sqrt(nx * nx + ny * ny);
    const double r0 = 1.0 - d.alfrz + d.alfrz * y0, r1 = 1.0 - d.alfrz + d.alfrz * y1;
    const double w = GEO == 2 ? 0.5 : (q0 == p ? 2.0 * r0 + r1 : 2.0 * r1 + r0) / 6.0;
    if (code / 1000 == 22) {
      wall22 = true;
      const int sub = code % 1000;
      // outward axis of the wall; ncase 1 and 2 know both sides of the unit box
      if (sub == 221) bvy += (((d.ncase == 1 || d.ncase == 2 || d.ncase == 12) && !(y0 < 1.0e-6 && y1 < 1.0e-6) &&
                               fabs(y0 - 1.0) < 1.0e-6 && fabs(y1 - 1.0) < 1.0e-6) ? w : -w) * len;
      else if (sub == 222) bvx += ((d.ncase == 1 && !(x0 < 1.0e-6 && x1 < 1.0e-6) && fabs(x0 - 1.0) < 1.0e-6 &&
                                    fabs(x1 - 1.0) < 1.0e-6) ? w : -w) * len;
    } else if (code / 1000 == 21 && d.ncase == 3) {
      bpx += 1.0e-6 * w * nx;
      bpy += 1.0e-6 * w * ny;
    }
  }
  double fx = bpx, fy = bpy;
  if (wall22) {
    const double cl = (bvx * bvx + bvy * bvy) / n.m;
    const double cr = ((n.a1 - n.s1 - bpx) * bvx + (n.a2 - n.s2 - bpy) * bvy) / n.m;
    const double k = cr / fmax(1.0e-16, cl);
    fx += k * bvx;
    fy += k * bvy;
  }
  if (!(bc & BC_KEEP)) {
    us = (n.a1 - n.s1 - fx) / n.m;
    vs = (n.a2 - n.s2 - fy) / n.m;
  }
  if (GEO == 1) {
    if (p == 0) { us = 0.0; vs = 0.0; }
    if (bc & BC_UV0) vs = 0.0;
  } else if (bc & (BC_V0 | BC_UV0)) {
    vs = 0.0;
  }
  if (bc & (BC_U0 | BC_UV0)) us = 0.0;
  d.us[p] = us;
  d.vs[p] = vs;
  if (MOVE) {
    const double oma = 1.0 - alfa;
    d.xo[p] = alfa * xn + oma * (xs + dt * us);
    d.yo[p] = alfa * yn + oma * (ys + dt * vs);
  }
}
// motion of stage 1
__global__ void __launch_bounds__(64) k1f_move(Dev1 d, double alfa) {
  const int p = blockIdx.x * 64 + threadIdx.x;
  await_previous();
  if (p >= d.npoin) return;
  const int done = d.sc_dev->done;
  const double dt = d.sc_dev->dtfix, oma = 1.0 - alfa;
  const double x = alfa * d.xn[p] + oma * (d.xs[p] + dt * d.us[p]);
  const double y = alfa * d.yn[p] + oma * (d.ys[p] + dt * d.vs[p]);
  if (done) return;
  d.xo[p] = x;
  d.yo[p] = y;
}

// ---------------------------------------------------------------------------
// dt: getdelt_lag's limits of the start-of-step cells and, in the last block, the
// step size; the step counter advances here
// ---------------------------------------------------------------------------
__device__ __forceinline__ void block_min2(double &a, double &b) {
  __shared__ double sm[2][8];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    a = fmin(a, __shfl_down_sync(0xffffffffu, a, o));
    b = fmin(b, __shfl_down_sync(0xffffffffu, b, o));
  }
  if ((threadIdx.x & 31) == 0) {
    sm[0][threadIdx.x >> 5] = a;
    sm[1][threadIdx.x >> 5] = b;
  }
  __syncthreads();
  if (threadIdx.x == 0)
    for (int w = 1; w < (int)(blockDim.x >> 5); w++) {
      a = fmin(a, sm[0][w]);
      b = fmin(b, sm[1][w]);
    }
  __syncthreads();
}
template <int GEO, bool AHEAD>
__global__ void __launch_bounds__(256) k1f_dt(Dev1 d, int ndt, int itime) {
  __shared__ int last;
  const int e = blockIdx.x * 256 + threadIdx.x;
  const size_t nc = d.ncell;
  if (!AHEAD) await_previous();
  const int el = e < d.nquad ? e : d.nquad - 1;
  int ip[4];
  double x[4], y[4], us[4], vs[4];
#pragma unroll
  for (int k = 0; k < 4; k++) {
    ip[k] = d.ipq[k * nc + el];
    x[k] = d.xn[ip[k]];
    y[k] = d.yn[ip[k]];
  }
  const double tau = d.Us[el], uc = d.Us[3 * nc + el], vc = d.Us[6 * nc + el], ec = d.Us[9 * nc + el];
  if (AHEAD) await_previous();  // the node pass: u*
  if (d.sc_dev->done) return;
  double dtcfl = 1e10, dtvol = 1e10;
  if (e < d.nquad) {
    const double eps = 1.0e-6, g = d.gamlg;
#pragma unroll
    for (int k = 0; k < 4; k++) {
      us[k] = d.us[ip[k]];
      vs[k] = d.vs[ip[k]];
    }
    const Bilin B = bilin(x, y);
    // the cell-average volume change: the face integral's moment 0 (and the
    // area-weighted form's source); in the plane branch by k1_rhs's expressions
    double dlen = 0.0, dv = 0.0;
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const int n = (k + 1) & 3;
      const double dl = sqrt((x[k] - x[n]) * (x[k] - x[n]) + (y[k] - y[n]) * (y[k] - y[n]));
      if (k == 0 || dl < dlen) dlen = dl;
    }
    if constexpr (GEO == 0) {
      double fn[4][3];
#pragma unroll
      for (int f = 0; f < 4; f++) {
        const int b = (f + 1) & 3;
        const double anx = y[b] - y[f];
        const double any = -(x[b] - x[f]);
        fn[f][0] = anx / sqrt(anx * anx + any * any);
        fn[f][1] = any / sqrt(anx * anx + any * any);
        fn[f][2] = sqrt(anx * anx + any * any);
      }
      const double c16 = 0.1666666666666666, b3 = 3.0;
#pragma unroll
      for (int iv = 0; iv < 4; iv++) {
        const int fa = (iv + 3) & 3, fb = iv;
        const double l1x = c16 * b3 * fn[fa][0] * fn[fa][2], l1y = c16 * b3 * fn[fa][1] * fn[fa][2];
        const double l2x = c16 * b3 * fn[fb][0] * fn[fb][2], l2y = c16 * b3 * fn[fb][1] * fn[fb][2];
        dv = dv + us[iv] * (l1x + l2x) + vs[iv] * (l1y + l2y);
      }
    } else {
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const int n = (k + 1) & 3;
        const double nx = y[n] - y[k], ny = x[k] - x[n];
        double o1, t1, o2, t2;
        edge_weights<GEO>(fabs(y[k]), fabs(y[n]), o1, t1);
        edge_weights<GEO>(fabs(y[n]), fabs(y[k]), o2, t2);
        dv += (o1 + t1) * (us[k] * nx + vs[k] * ny) + (o2 + t2) * (us[n] * nx + vs[n] * ny);
      }
    }
    const double vol = cell_volume<GEO>(B);
    if (GEO == 2) dv = vol / (4.0 * B.j0) * dv + vc * (4.0 * B.j0);
    const double rhoct = 1.0 / tau;
    const double pctr = fmax(eps, (g - 1.0) * rhoct * (ec - 0.5 * (uc * uc + vc * vc)));
    const double sdctr = sqrt(fmax(eps, g * pctr / rhoct));
    dtcfl = dlen / sdctr;
    dtvol = vol / fabs(dv);
  }
  block_min2(dtcfl, dtvol);
  if (threadIdx.x == 0) {
    d.dtpart[2 * blockIdx.x] = dtcfl;
    d.dtpart[2 * blockIdx.x + 1] = dtvol;
    __threadfence();
    last = atomicAdd(d.count, 1) == (int)gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  double a = 1e10, b = 1e10;
  for (int i = threadIdx.x; i < (int)gridDim.x; i += 256) {
    a = fmin(a, __ldcg(d.dtpart + 2 * i));
    b = fmin(b, __ldcg(d.dtpart + 2 * i + 1));
  }
  block_min2(a, b);
  if (threadIdx.x == 0) {
    *d.count = 0;
    Scalars *S = d.sc_dev;
    S->itime = itime < 0 ? S->itime + 1 : itime;
    dt_apply1(d, a, b, ndt);
  }
}

// ---------------------------------------------------------------------------
// RHS and update, one thread per cell
// ---------------------------------------------------------------------------
constexpr int kRhsThreads = 64;
template <int GEO>
__global__ void __launch_bounds__(kRhsThreads) k1f_rhs(Dev1 d, int fuse, double alfa, int last_stage) {
  const int e = blockIdx.x * kRhsThreads + threadIdx.x;
  const size_t nc = d.ncell;
  const int done = d.sc_dev->done, el = e < d.nquad ? e : d.nquad - 1;
  // ahead of the node pass (in stage 1 of the time step): all but the face integral
  int ip[4];
#pragma unroll
  for (int k = 0; k < 4; k++) ip[k] = d.ipq[k * nc + el];
  double u[4][ND];
#pragma unroll
  for (int q = 0; q < 4; q++)
#pragma unroll
    for (int k = 0; k < ND; k++) u[q][k] = d.Us[(q * ND + k) * nc + el];
  const double rc = d.rc[el], sc = d.sc[el];
  const double af1 = d.lim[0 * nc + el], af4 = d.lim[1 * nc + el], af5 = d.lim[2 * nc + el];
  const double v11 = d.lim[3 * nc + el], v12 = d.lim[4 * nc + el], v22 = d.lim[6 * nc + el];
  double x[4], y[4];
#pragma unroll
  for (int k = 0; k < 4; k++) {
    x[k] = d.xs[ip[k]];
    y[k] = d.ys[ip[k]];
  }
  const Bilin B = bilin(x, y);
  const double g = d.gamlg, epsd = 1.0e-6;
  const int md = d.mdegr;
  // moments of the limited pressure over the 25 points: M without, Q (nrz = 1)
  // with the radius weight
  const double pctr = pressure(g, u[0][0], u[1][0], u[2][0], u[3][0], epsd);
  double M00 = 0.0, M10 = 0.0, M01 = 0.0, M20 = 0.0, M11 = 0.0, M02 = 0.0;
  double Q00 = 0.0, Q10 = 0.0, Q01 = 0.0, Q20 = 0.0, Q11 = 0.0, Q02 = 0.0;
  double c0[4], c1[4], c2[4];
#pragma unroll
  for (int q = 0; q < 4; q++) {
    c1[q] = md > 1 ? u[q][1] : 0.0;
    c2[q] = md > 2 ? u[q][2] : 0.0;
    c0[q] = u[q][0] - c1[q] * rc - c2[q] * sc;
  }
#pragma unroll 1
  for (int i = 0; i < 5; i++) {
    const double r = g5x(i), wi = g5wt(i);
    double a[4], t[5], pre[5];
#pragma unroll
    for (int q = 0; q < 4; q++) a[q] = c0[q] + c1[q] * r;
#pragma unroll
    for (int j = 0; j < 5; j++) {
      t[j] = a[0] + c2[0] * g5x(j);
      pre[j] = j == 0 ? t[0] : pre[j - 1] * t[j];
    }
    double inv = 1.0 / pre[4], m0 = 0.0, m1 = 0.0, m2 = 0.0, q0 = 0.0, q1 = 0.0, q2 = 0.0;
    const double yr = B.yc + B.f1 * r, ysl = B.f2 + B.f3 * r;
#pragma unroll
    for (int j = 4; j >= 0; j--) {
      const double rho = j > 0 ? inv * pre[j > 0 ? j - 1 : 0] : inv;
      inv *= t[j];
      const double s = g5x(j);
      const double uu = a[1] + c2[1] * s, vv = a[2] + c2[2] * s, ee = a[3] + c2[3] * s;
      const double p = pctr + af4 * ((g - 1.0) * rho * (ee - 0.5 * (uu * uu + vv * vv)) - pctr);
      const double m = g5wt(j) * p;
      m0 += m;
      m1 += m * s;
      m2 += m * s * s;
      if (GEO == 1) {
        const double q = m * (yr + ysl * s);
        q0 += q;
        q1 += q * s;
        q2 += q * s * s;
      }
    }
    m0 *= wi; m1 *= wi; m2 *= wi;
    M00 += m0; M10 += r * m0; M20 += r * r * m0; M01 += m1; M11 += r * m1; M02 += m2;
    if (GEO == 1) {
      q0 *= wi; q1 *= wi; q2 *= wi;
      Q00 += q0; Q10 += r * q0; Q20 += r * r * q0; Q01 += q1; Q11 += r * q1; Q02 += q2;
    }
  }
  await_previous();
  if (e < d.nquad && !done) {
    double us[4], vs[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
      us[k] = d.us[ip[k]];
      vs[k] = d.vs[ip[k]];
    }
    // face integral: per corner the two edges with their own and other basis
    double R[ND][4];
#pragma unroll
    for (int k = 0; k < ND; k++)
#pragma unroll
      for (int q = 0; q < 4; q++) R[k][q] = 0.0;
    const double bm[2] = {-1.0 - rc, 1.0 - rc}, cm[2] = {-1.0 - sc, 1.0 - sc};
    auto add = [&](double r1, double r2, double tw, double f0, double f1, double fe) {
      // basis moments (1, r1, r2) already weighted into the four values
      R[1][0] += r1 * tw; R[1][1] += r1 * f0; R[1][2] += r1 * f1; R[1][3] += r1 * fe;
      R[2][0] += r2 * tw; R[2][1] += r2 * f0; R[2][2] += r2 * f1; R[2][3] += r2 * fe;
    };
#pragma unroll
    for (int iv = 0; iv < 4; iv++) {
      const int vp = (iv + 3) & 3, vn = (iv + 1) & 3;
      const double *o = d.cf + iv * nc + e;
      const double br = bm[(iv == 1 || iv == 2) ? 1 : 0], bs = cm[iv >= 2 ? 1 : 0];
      const double ul = o[CF_U * 4 * nc], vl = o[CF_V * 4 * nc];
      const double dux = us[iv] - ul, duy = vs[iv] - vl;
      const double ax = y[iv] - y[vp], ay = x[vp] - x[iv], bx = y[vn] - y[iv], by = x[iv] - x[vn];
      const double pl = o[CF_P * 4 * nc], ma = o[CF_MA * 4 * nc], mb = o[CF_MB * 4 * nc];
      // edge a ends at the previous vertex, edge b at the next one
      const double brp = bm[(vp == 1 || vp == 2) ? 1 : 0], bsp = cm[vp >= 2 ? 1 : 0];
      const double brn = bm[(vn == 1 || vn == 2) ? 1 : 0], bsn = cm[vn >= 2 ? 1 : 0];
      double oa, na, ob, nn;
      edge_weights<GEO>(fabs(y[iv]), fabs(y[vp]), oa, na);
      edge_weights<GEO>(fabs(y[iv]), fabs(y[vn]), ob, nn);
      {
        const double f0 = ma * dux - pl * ax, f1 = ma * duy - pl * ay;
        const double tw = us[iv] * ax + vs[iv] * ay, fe = us[iv] * f0 + vs[iv] * f1, w = oa + na;
        R[0][0] += w * tw; R[0][1] += w * f0; R[0][2] += w * f1; R[0][3] += w * fe;
        add(oa * br + na * brp, oa * bs + na * bsp, tw, f0, f1, fe);
      }
      {
        const double f0 = mb * dux - pl * bx, f1 = mb * duy - pl * by;
        const double tw = us[iv] * bx + vs[iv] * by, fe = us[iv] * f0 + vs[iv] * f1, w = ob + nn;
        R[0][0] += w * tw; R[0][1] += w * f0; R[0][2] += w * f1; R[0][3] += w * fe;
        add(ob * br + nn * brn, ob * bs + nn * bsn, tw, f0, f1, fe);
      }
    }
    // moments of the weight alone (closed form): 1, or y in nrz = 1
    double N00 = 4.0, N10 = 0.0, N01 = 0.0, N20 = 4.0 / 3.0, N11 = 0.0, N02 = 4.0 / 3.0;
    if (GEO == 1) {
      N00 = 4.0 * B.yc; N10 = (4.0 / 3.0) * B.f1; N01 = (4.0 / 3.0) * B.f2;
      N20 = (4.0 / 3.0) * B.yc; N11 = (4.0 / 9.0) * B.f3; N02 = N20;
    } else {
      Q00 = M00; Q10 = M10; Q01 = M01; Q20 = M20; Q11 = M11; Q02 = M02;
    }
    {
      // limited velocity a0 + a1 r + a2 s
      const double ar = v11 * u[1][1] + v12 * u[2][1], as = v11 * u[1][2] + v12 * u[2][2];
      const double cr = v12 * u[1][1] + v22 * u[2][1], cs = v12 * u[1][2] + v22 * u[2][2];
      const double a0 = u[1][0] - ar * rc - as * sc, b0 = u[2][0] - cr * rc - cs * sc;
      // k = 1: cof = (y_s, -x_s); k = 2: cof = (-y_r, x_r)
      const double h00 = B.f2 * a0 - B.e2 * b0, h10 = B.f2 * ar + B.f3 * a0 - B.e2 * cr - B.e3 * b0,
                   h01 = B.f2 * as - B.e2 * cs, h20 = B.f3 * ar - B.e3 * cr, h11 = B.f3 * as - B.e3 * cs;
      const double k00 = B.e1 * b0 - B.f1 * a0, k10 = B.e1 * cr - B.f1 * ar,
                   k01 = B.e1 * cs + B.e3 * b0 - B.f1 * as - B.f3 * a0, k11 = B.e3 * cr - B.f3 * ar,
                   k02 = B.e3 * cs - B.f3 * as;
      R[1][0] -= h00 * N00 + h10 * N10 + h01 * N01 + h20 * N20 + h11 * N11;
      R[2][0] -= k00 * N00 + k10 * N10 + k01 * N01 + k11 * N11 + k02 * N02;
      R[1][1] += B.f2 * Q00 + B.f3 * Q10;
      R[2][1] -= B.f1 * Q00 + B.f3 * Q01;
      R[1][2] -= B.e2 * Q00 + B.e3 * Q10;
      R[2][2] += B.e1 * Q00 + B.e3 * Q01;
      R[1][3] += h00 * Q00 + h10 * Q10 + h01 * Q01 + h20 * Q20 + h11 * Q11;
      R[2][3] += k00 * Q00 + k10 * Q10 + k01 * Q01 + k11 * Q11 + k02 * Q02;
    }
    {
      // moments of p det J (no radius weight): the sources
      const double d0 = B.j0 * M00 + B.j1 * M10 + B.j2 * M01;
      const double d1 = B.j0 * M10 + B.j1 * M20 + B.j2 * M11 - rc * d0;
      const double d2 = B.j0 * M01 + B.j1 * M11 + B.j2 * M02 - sc * d0;
      if (GEO == 1) {  // hoop stress (Getrhslagmc.f90:15800-16048)
        R[0][2] += d.alfrz * d0;
        R[1][2] += d.alfrz * d1;
        R[2][2] += d.alfrz * d2;
      } else {         // times geoel(11), then the sources of Getrhslagrz.f90:2818-3096
        const double rb = cell_volume<2>(B) / (4.0 * B.j0);
#pragma unroll
        for (int k = 0; k < ND; k++)
#pragma unroll
          for (int q = 0; q < 4; q++) R[k][q] *= rb;
        const double vc = u[2][0], t0 = 4.0 * B.j0;
        R[0][0] += vc * t0;
        R[1][0] += vc * ((4.0 / 3.0) * B.j1 - rc * t0);
        R[2][0] += vc * ((4.0 / 3.0) * B.j2 - sc * t0);
        R[0][3] -= vc * d0;
        R[1][3] -= vc * d1;
        R[2][3] -= vc * d2;
      }
    }
    if (!fuse) {
#pragma unroll
      for (int k = 0; k < ND; k++)
#pragma unroll
        for (int q = 0; q < 4; q++) d.rhs[(q * ND + k) * nc + e] = R[k][q];
    } else {
      // limited slopes (Getrhslagmc.f90:7283-7298) and update (Getrhslag.f90:1789-1904)
      const double dt = d.sc_dev->dtfix, oma = 1.0 - alfa;
      const double m1 = d.amatr[0 * nc + e], m2 = d.amatr[1 * nc + e], m3 = d.amatr[2 * nc + e], m0 = d.amatr[3 * nc + e];
      double avg[4];
#pragma unroll
      for (int q = 0; q < 4; q++) {
        double s1, s2;
        if (q == 0) { s1 = u[0][1] * af1; s2 = u[0][2] * af1; }
        else if (q == 1) { s1 = v11 * u[1][1] + v12 * u[2][1]; s2 = v11 * u[1][2] + v12 * u[2][2]; }
        else if (q == 2) { s1 = v12 * u[1][1] + v22 * u[2][1]; s2 = v12 * u[1][2] + v22 * u[2][2]; }
        else { s1 = u[3][1] * af5; s2 = u[3][2] * af5; }
        const double n0 = oma * (u[q][0] + m0 * (dt * R[0][q]));
        const double n1 = oma * (s1 + (m1 * (dt * R[1][q]) + m2 * (dt * R[2][q])));
        const double n2 = oma * (s2 + (m2 * (dt * R[1][q]) + m3 * (dt * R[2][q])));
        const size_t o = (size_t)q * ND * nc + e;
        // stage 1 has alfa = 0 and reads no U^n
        avg[q] = alfa != 0.0 ? alfa * d.Un[o] + n0 : n0;
        const double o1 = alfa != 0.0 ? alfa * d.Un[o + nc] + n1 : n1, o2 = alfa != 0.0 ? alfa * d.Un[o + 2 * nc] + n2 : n2;
        d.Uo[o] = avg[q];
        d.Uo[o + nc] = o1;
        d.Uo[o + 2 * nc] = o2;
      }
      d.pbar[e] = pressure(g, avg[0], avg[1], avg[2], avg[3], EPS_S);
    }
  }
  if (!last_stage || done) return;
  // the exit test, once every block has read the flag
  __syncthreads();
  if (threadIdx.x == 0 && atomicAdd(d.count + 1, 1) == (int)gridDim.x - 1) {
    d.count[1] = 0;
    Scalars *S = d.sc_dev;
    if (fabs(S->tacru - d.tend) / d.tend <= 1e-11) S->done = 1;
  }
}

// cell-average pressures of a state that an upload or the initial fields set
__global__ void k1f_pbar(Dev1 d, const double *A) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= d.ncell) return;
  const size_t nc = d.ncell;
  d.pbar[e] = pressure(d.gamlg, A[e], A[3 * nc + e], A[6 * nc + e], A[9 * nc + e], EPS_S);
}

// volumes and their centres in closed form; nrz = 2 also the area centroid and
// geoel(11).  No exit test: on unchanged nodes it repeats itself.
template <int GEO>
__global__ void k1f_geom(Dev1 d, const double *X, const double *Y) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= d.nquad) return;
  double x[4], y[4];
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const int p = d.ipq[k * (size_t)d.nquad + e];
    x[k] = X[p];
    y[k] = Y[p];
  }
  const Bilin B = bilin(x, y);
  const double vol = cell_volume<GEO>(B);
  double rcv = B.j1 / (3.0 * B.j0), scv = B.j2 / (3.0 * B.j0);
  if (GEO == 1) {
    rcv = ((4.0 / 3.0) * (B.j0 * B.f1 + B.j1 * B.yc) + (4.0 / 9.0) * B.j2 * B.f3) / vol;
    scv = ((4.0 / 3.0) * (B.j0 * B.f2 + B.j2 * B.yc) + (4.0 / 9.0) * B.j1 * B.f3) / vol;
  }
  d.vol[e] = vol;
  d.vcx[e] = rcv;
  d.vcy[e] = scv;
  if (GEO == 2) d.rbar[e] = vol / (4.0 * B.j0);
  if (!(vol > 0.0)) atomicOr(&d.sc_dev->status, ST_NONPHYS);
}
