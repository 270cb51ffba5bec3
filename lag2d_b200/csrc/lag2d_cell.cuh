// The cell integrals of the optimised FP64 stage: Persson indicator, sub-cell
// density corrections, Taylor-Green source; one thread per quad.  Included by
// lag2d_fast.cu inside namespace lag2d::fast.
//
// All three are bound by FP64 operations (60-75% of that pipe), so what counts is
// the operations a quad.  They start from the 16 coefficients of the quad's
// biquadratic map (64 operations) instead of its 28 node cross products: det J
// then takes 25 pairs of coefficients (75 operations) instead of a dense 28 x 15
// map (330).  Integrals of polynomials are taken in closed form; the Gauss sums
// that are not polynomial run over pairs of points at +-y, whose even and odd
// parts are shared.

// x(r, s) = sum a[i][j] r^i s^j relative to the centre node, y alike with b
struct QuadMap {
  double a[3][3], b[3][3];
};
__host__ __device__ __forceinline__ void map_coeffs(const double X[3][3], double a[3][3]) {
  const double o = X[1][1];
  double c[3][3];
#pragma unroll
  for (int j = 0; j < 3; j++) {
    const double lo = X[0][j] - o, hi = X[2][j] - o, mid = j == 1 ? 0.0 : X[1][j] - o;
    c[0][j] = mid;
    c[1][j] = 0.5 * (hi - lo);
    c[2][j] = 0.5 * (hi + lo) - mid;
  }
#pragma unroll
  for (int i = 0; i < 3; i++) {
    a[i][0] = c[i][1];
    a[i][1] = 0.5 * (c[i][2] - c[i][0]);
    a[i][2] = 0.5 * (c[i][2] + c[i][0]) - c[i][1];
  }
}
__host__ __device__ __forceinline__ void load_map(const Dev &d, int iq, QuadMap &m) {
  Loaded L;
  load_cell(d, d.xs, d.ys, iq, L);
  map_coeffs(L.X, m.a);
  map_coeffs(L.Y, m.b);
}
// det J = sum D[i][j] r^i s^j (D[3][3] = 0): x_r y_s - x_s y_r pairs the terms
// (i, j), (k, l) of x and y with the weight i l - j k
__host__ __device__ __forceinline__ void map_det(const QuadMap &m, double D[4][4]) {
#define CR(i, j, k, l) (m.a[i][j] * m.b[k][l] - m.a[k][l] * m.b[i][j])
  D[0][0] = CR(1, 0, 0, 1);
  D[0][1] = 2.0 * CR(1, 0, 0, 2) - CR(0, 1, 1, 1);
  D[0][2] = 2.0 * CR(1, 1, 0, 2) - CR(0, 1, 1, 2);
  D[0][3] = -2.0 * CR(0, 2, 1, 2);
  D[1][0] = CR(1, 0, 1, 1) - 2.0 * CR(0, 1, 2, 0);
  D[1][1] = 2.0 * CR(1, 0, 1, 2) - 2.0 * CR(0, 1, 2, 1) + 4.0 * CR(2, 0, 0, 2);
  D[1][2] = CR(1, 1, 1, 2) - 2.0 * CR(0, 1, 2, 2) - 4.0 * CR(0, 2, 2, 1);
  D[1][3] = -4.0 * CR(0, 2, 2, 2);
  D[2][0] = CR(1, 0, 2, 1) + 2.0 * CR(2, 0, 1, 1);
  D[2][1] = 2.0 * CR(1, 0, 2, 2) + 4.0 * CR(2, 0, 1, 2) - CR(1, 1, 2, 1);
  D[2][2] = 3.0 * CR(2, 1, 1, 2);
  D[2][3] = -2.0 * CR(1, 2, 2, 2);
  D[3][0] = 2.0 * CR(2, 0, 2, 1);
  D[3][1] = 4.0 * CR(2, 0, 2, 2);
  D[3][2] = 2.0 * CR(2, 1, 2, 2);
  D[3][3] = 0.0;
#undef CR
}
// coefficients of row r in s
__host__ __device__ __forceinline__ void det_row(const double D[4][4], double r, double e[4]) {
#pragma unroll
  for (int n = 0; n < 3; n++) e[n] = D[0][n] + r * (D[1][n] + r * (D[2][n] + r * D[3][n]));
  e[3] = D[0][3] + r * (D[1][3] + r * D[2][3]);
}

// ---------------------------------------------------------------------------
// Persson indicator (all quads): the integrals of u_P2^2 and u^2 of tau, both of
// degree 7 at most in each direction, where the reference's 5 x 5 Gauss rule is
// exact, from the moments of det J up to degree 4.  The physical mass centre and
// the frame that WENO needs are computed by WENO for its stencils, not here for
// every quad.  1024 x 1024: 66 -> 39 us a
// launch.
// ---------------------------------------------------------------------------
// integral of r^k over [-1, 1]
__host__ __device__ constexpr double mono(int k) { return k % 2 ? 0.0 : 2.0 / (k + 1); }

__host__ __device__ void f_persson(const Dev &d, int iq) {
  if (iq >= d.nquad || d.sc_dev->done) return;
  const int e = iq + d.ntria;
  double t[6];
#pragma unroll
  for (int k = 0; k < 6; k++) t[k] = d.Us[k * (size_t)d.ncell + e];
  const CellGeo g{d.rc[e], d.sc[e], d.g19[e], d.g20[e], d.g21[e]};
  QuadMap m;
  load_map(d, iq, m);
  double D[4][4];
  map_det(m, D);
  // I[a][b] = integral of r^a s^b det J, a + b <= 4
  double I[5][5];
#pragma unroll
  for (int a = 0; a < 5; a++) {
    double F[4];
#pragma unroll
    for (int n = 0; n < 4; n++)
      F[n] = a % 2 ? mono(a + 1) * D[1][n] + mono(a + 3) * D[3][n] : mono(a) * D[0][n] + mono(a + 2) * D[2][n];
#pragma unroll
    for (int b = 0; a + b < 5; b++)
      I[a][b] = b % 2 ? mono(b + 1) * F[1] + mono(b + 3) * F[3] : mono(b) * F[0] + mono(b + 2) * F[2];
  }
  // P2 part h and P1 part p over the monomials 1, r, s, r^2, s^2, r s
  double h[6], p[3], v[6];
  h[1] = -t[3] * g.rc - t[5] * g.sc;
  h[2] = -t[4] * g.sc - t[5] * g.rc;
  h[3] = 0.5 * t[3];
  h[4] = 0.5 * t[4];
  h[5] = t[5];
  h[0] = t[3] * (0.5 * g.rc * g.rc - g.g19) + t[4] * (0.5 * g.sc * g.sc - g.g20) + t[5] * (g.rc * g.sc - g.g21);
  p[0] = t[0] - t[1] * g.rc - t[2] * g.sc;
  p[1] = t[1];
  p[2] = t[2];
  const int pa[6] = {0, 1, 0, 2, 0, 1}, pb[6] = {0, 0, 1, 0, 2, 1};
#pragma unroll
  for (int i = 0; i < 6; i++) {
    v[i] = 0.0;
#pragma unroll
    for (int j = 0; j < 6; j++) v[i] += I[pa[i] + pa[j]][pb[i] + pb[j]] * h[j];
  }
  double unvar2 = 0.0;
#pragma unroll
  for (int i = 0; i < 6; i++) unvar2 += h[i] * v[i];
  double unvar1 = unvar2;
#pragma unroll
  for (int i = 0; i < 3; i++) {
    const double w = I[pa[i]][pb[i]] * p[0] + I[pa[i] + 1][pb[i]] * p[1] + I[pa[i]][pb[i] + 1] * p[2];
    unvar1 += p[i] * (2.0 * v[i] + w);
  }
  // log10(ratio) <= -3 log10(4) - 4; a negative or undefined ratio marks the quad
  const double q = unvar2 / unvar1;
  const int fl = q >= 0.0 && q <= 1.0e-4 / 64.0 ? 0 : 1;
  d.flag[e] = fl;
  if (fl) {
#ifdef __CUDA_ARCH__
    const int slot = atomicAdd(d.wcount, 1);
#else
    const int slot = (*d.wcount)++;
#endif
    d.wlist[slot] = iq;
  }
}

// ---------------------------------------------------------------------------
// Sub-cell density corrections (getrhosubg_averg / _daverg): initial mass over
// exact sub-cell area, less the DG-implied density, the sum over 5 x 5 Gauss
// points of det J / tau over that area.  The area, which the reference takes
// from the sub-cell's own 9 nodes, is the integral of det J over the sub-square.
//
// The sum is kept as one fraction: a pair of points at s0 +- y with det J = E +- O
// and tau = A +- B adds 2 (E A - O B) / (A^2 - B^2); a row's two pairs and its
// middle point are brought together first.  One division per sub-cell instead of
// one per point.  tau is scaled by the cell-average tau, so that the product of
// the 25 scaled values stays near 1.  Sub-cells 0 and 3 (r in [-1, 0]) share
// their Gauss rows, and so do 1 and 2 (r in [0, 1]).  The rows are unrolled: a
// rolled loop read the rule from local memory (131 us a launch against 86).
// 1024 x 1024: 155 -> 86 us a launch.
// ---------------------------------------------------------------------------
// one row of a sub-cell about its middle: fraction num / den of its 5 points
__host__ __device__ __forceinline__ void half_row(double e0, double e1, double e2, double e3, double t0, double t1,
                                                  double t2, double &num, double &den) {
  const double T = t1 * t1;
  double n[2], q[2];
#pragma unroll
  for (int k = 0; k < 2; k++) {
    const double y = 0.5 * (k == 0 ? g5p(4) : g5p(3)), y2 = y * y;
    const double E = e0 + y2 * e2, P = e1 + y2 * e3, A = t0 + y2 * t2;
    n[k] = E * A - y2 * (P * t1);
    q[k] = A * A - y2 * T;
  }
  const double w0 = 2.0 * g5w(4), w1 = 2.0 * g5w(3), w2 = g5w(2);
  const double qq = q[0] * q[1];
  num = (w0 * n[0] * q[1] + w1 * n[1] * q[0]) * t0 + w2 * e0 * qq;
  den = qq * t0;
}
__host__ __device__ void f_corner_corr(const Dev &d, int iq) {
  if (iq >= d.nquad || d.sc_dev->done) return;
  const int e = iq + d.ntria;
  double u[6], ms[4];
#pragma unroll
  for (int k = 0; k < 6; k++) u[k] = d.Us[k * (size_t)d.ncell + e];
#pragma unroll
  for (int k = 0; k < 4; k++) ms[k] = d.msub[k * (size_t)d.nquad + iq];
  const CellGeo G{d.rc[e], d.sc[e], d.g19[e], d.g20[e], d.g21[e]};
  QuadMap m;
  load_map(d, iq, m);
  double D[4][4];
  map_det(m, D);
  // scaled tau over the monomials 1, r, s, r^2, s^2, r s
  const double rtc = 1.0 / u[0];
  const double q3 = rtc * (0.5 * u[3]), t2 = rtc * (0.5 * u[4]), q5 = rtc * u[5];
  const double q1 = rtc * u[1] - 2.0 * q3 * G.rc - q5 * G.sc, q2 = rtc * u[2] - 2.0 * t2 * G.sc - q5 * G.rc;
  const double q0 = 1.0 - rtc * (u[1] * G.rc + u[2] * G.sc) + q3 * (G.rc * G.rc - 2.0 * G.g19) +
                    t2 * (G.sc * G.sc - 2.0 * G.g20) + q5 * (G.rc * G.sc - G.g21);
#pragma unroll
  for (int h = 0; h < 2; h++) {
    const double ofr = h == 0 ? -0.5 : 0.5;
    double N[2] = {0.0, 0.0}, Q[2] = {1.0, 1.0};  // s in [-1, 0], [0, 1]
#pragma unroll
    for (int i = 0; i < 5; i++) {
      const double r = 0.5 * g5p(i) + ofr, wi = 0.25 * g5w(i);
      double c[4];
      det_row(D, r, c);
      const double t0 = q0 + r * (q1 + r * q3), t1 = q2 + r * q5;
      // both halves about their middles s = -+1/2
      const double ea = c[0] + 0.25 * c[2], eb = 0.5 * c[1] + 0.125 * c[3], ec = c[1] + 0.75 * c[3];
      const double ta = t0 + 0.25 * t2;
#pragma unroll
      for (int k = 0; k < 2; k++) {
        const double sg = k == 0 ? -1.0 : 1.0;
        double n, q;
        half_row(ea + sg * eb, ec + sg * c[2], c[2] + (1.5 * sg) * c[3], c[3], ta + (0.5 * sg) * t1, t1 + sg * t2, t2, n,
                 q);
        N[k] = N[k] * q + (wi * n) * Q[k];
        Q[k] = Q[k] * q;
      }
    }
    // sub-areas: det J over r in [-1, 0] or [0, 1], then over s
    double F[4];
#pragma unroll
    for (int n = 0; n < 4; n++) {
      const double ev = D[0][n] + (1.0 / 3.0) * D[2][n], od = 0.5 * D[1][n] + 0.25 * D[3][n];
      F[n] = h == 0 ? ev - od : ev + od;
    }
    const double ev = F[0] + (1.0 / 3.0) * F[2], od = 0.5 * F[1] + 0.25 * F[3];
#pragma unroll
    for (int k = 0; k < 2; k++) {
      const int isg = h == 0 ? (k == 0 ? 0 : 3) : (k == 0 ? 1 : 2);
      const double area = k == 0 ? ev - od : ev + od;
      d.corr[isg * (size_t)d.nquad + iq] = d.cdrho * ((ms[isg] * Q[k] - rtc * N[k]) / (Q[k] * area));
    }
  }
}

// ---------------------------------------------------------------------------
// Taylor-Green energy source of the stage (rhsdomnsrcdg_lag_curvquad,
// Getrhslag.f90:4070-4251): it depends on the stage's nodes and the reference
// geometry only; the RHS pass adds the 6 moments (d.src, [6][nquad]).  A kernel
// of its own: inside the corner or RHS kernels its registers and code cost those
// kernels more than its own launch.
//
// Moments el[k] = sum_g src(x_g) b_k(g) det J_g w_g over the 5 x 5 Gauss points,
// src = cos 3 pi x cos pi y - cos 3 pi y cos pi x = 4 c_x c_y (c_x^2 - c_y^2).
// cos(pi x) about the centre node x_c is a polynomial in d = x - x_c, from
// NSER terms each of the series of cos(pi d) and sin(pi d) (cossin_pi_series),
// when every node of the cell lies within delta of the centre node in x and y
// (the quadratic map then keeps |d| <= 1.5625 delta at the Gauss points): delta
// <= 0.09 for 7 terms, 0.004 for 4, 0.0006 for 3, each with the first omitted
// term below 1e-17; otherwise (NSER = 0) cospi at each point.  1024 x 1024
// (NSER = 3): 130 -> 82 us a launch.
// ---------------------------------------------------------------------------
// cos(pi (x_c + d)): for NSER = 3 and 4 from the 2 NSER coefficients in d, for 7,
// whose 28 would not stay in registers, from cos and sin of x_c and the series
template <int NSER>
constexpr int kCos = NSER == 3 || NSER == 4 ? 2 * NSER : NSER == 7 ? 2 : 1;
template <int NSER>
__host__ __device__ __forceinline__ void cos_coeffs(double xc, double *k) {
  if (NSER == 0) {
    k[0] = xc;
    return;
  }
  double c, s;
#ifdef __CUDA_ARCH__
  sincospi(xc, &s, &c);
#else
  c = cos(3.14159265358979311599796346854 * xc);
  s = sin(3.14159265358979311599796346854 * xc);
#endif
  double f = 1.0;  // pi^n / n!
#pragma unroll
  for (int n = 0; n < kCos<NSER>; n++) {
    if (n > 0 && NSER != 7) f *= 3.14159265358979311599796346854 / n;
    k[n] = f * (n % 4 == 0 ? c : n % 4 == 1 ? -s : n % 4 == 2 ? -c : s);
  }
}
template <int NSER>
__host__ __device__ __forceinline__ double cos_at(const double *k, double d) {
  if (NSER == 0) {
#ifdef __CUDA_ARCH__
    return cospi(k[0] + d);
#else
    return cos(3.14159265358979311599796346854 * (k[0] + d));
#endif
  }
  if (NSER == 7) {
    double c, s;
    cossin_pi_series<7>(d, c, s);
    return k[0] * c + k[kCos<NSER> - 1] * s;
  }
  double p = k[kCos<NSER> - 1];
#pragma unroll
  for (int n = kCos<NSER> - 2; n >= 0; n--) p = k[n] + d * p;
  return p;
}
template <int NSER>
__host__ __device__ __forceinline__ void tgv_moments(const QuadMap &m, const double D[4][4], double xc, double yc,
                                                     double M[6]) {
  double kx[kCos<NSER>], ky[kCos<NSER>];
  cos_coeffs<NSER>(xc, kx);
  cos_coeffs<NSER>(yc, ky);
  // raw moments over 1, r, s, r^2, s^2, r s
#pragma unroll
  for (int k = 0; k < 6; k++) M[k] = 0.0;
#pragma unroll
  for (int i = 0; i < 5; i++) {
    const double r = g5p(i), wi = g5w(i);
    double e[4], px[3], py[3];
    det_row(D, r, e);
#pragma unroll
    for (int n = 0; n < 3; n++) {
      px[n] = n == 0 ? r * (m.a[1][0] + r * m.a[2][0]) : m.a[0][n] + r * (m.a[1][n] + r * m.a[2][n]);
      py[n] = n == 0 ? r * (m.b[1][0] + r * m.b[2][0]) : m.b[0][n] + r * (m.b[1][n] + r * m.b[2][n]);
    }
    double m0, m1 = 0.0, m2 = 0.0;
    {
      const double cx = cos_at<NSER>(kx, px[0]), cy = cos_at<NSER>(ky, py[0]);
      m0 = g5w(2) * ((cx * cy) * (cx * cx - cy * cy) * e[0]);
    }
#pragma unroll
    for (int j = 3; j < 5; j++) {
      const double y = g5p(j), y2 = y * y, w = g5w(j);
      const double xe = px[0] + y2 * px[2], ye = py[0] + y2 * py[2];
      const double ee = e[0] + y2 * e[2], eo = e[1] + y2 * e[3];
      double f[2];
#pragma unroll
      for (int k = 0; k < 2; k++) {
        const double s = k == 0 ? -y : y;
        const double cx = cos_at<NSER>(kx, xe + s * px[1]), cy = cos_at<NSER>(ky, ye + s * py[1]);
        f[k] = (cx * cy) * (cx * cx - cy * cy) * (ee + s * eo);
      }
      const double sum = f[1] + f[0], dif = f[1] - f[0];
      m0 += w * sum;
      m1 += (w * y) * dif;
      m2 += (w * y2) * sum;
    }
    m0 *= wi;
    m1 *= wi;
    M[0] += m0;
    M[1] += r * m0;
    M[2] += m1;
    M[3] += (r * r) * m0;
    M[4] += wi * m2;
    M[5] += r * m1;
  }
}
__host__ __device__ void f_tgv_src(const Dev &d, int iq) {
  if (iq >= d.nquad || d.sc_dev->done) return;
  const int e = iq + d.ntria;
  Loaded L;
  load_cell(d, d.xs, d.ys, iq, L);
  const CellGeo G{d.rc[e], d.sc[e], d.g19[e], d.g20[e], d.g21[e]};
  const double xc = L.X[1][1], yc = L.Y[1][1];
  double delta = 0.0;
#pragma unroll
  for (int a = 0; a < 3; a++)
#pragma unroll
    for (int b = 0; b < 3; b++) delta = fmax(delta, fmax(fabs(L.X[a][b] - xc), fabs(L.Y[a][b] - yc)));
  QuadMap m;
  map_coeffs(L.X, m.a);
  map_coeffs(L.Y, m.b);
  double D[4][4], M[6];
  map_det(m, D);
  if (delta <= 0.0006) tgv_moments<3>(m, D, xc, yc, M);
  else if (delta <= 0.004) tgv_moments<4>(m, D, xc, yc, M);
  else if (delta <= 0.09) tgv_moments<7>(m, D, xc, yc, M);
  else tgv_moments<0>(m, D, xc, yc, M);
  // b = (1, r - rc, s - sc, (r - rc)^2/2 - g19, (s - sc)^2/2 - g20, (r - rc)(s - sc) - g21)
  const double coef = 3.14159265358979311599796346854 / (d.gamlg - 1.0);
  double *o = d.src + iq;
  const size_t nq = d.nquad;
  o[0] = coef * M[0];
  o[nq] = coef * (M[1] - G.rc * M[0]);
  o[2 * nq] = coef * (M[2] - G.sc * M[0]);
  o[3 * nq] = coef * (0.5 * M[3] - G.rc * M[1] + (0.5 * G.rc * G.rc - G.g19) * M[0]);
  o[4 * nq] = coef * (0.5 * M[4] - G.sc * M[2] + (0.5 * G.sc * G.sc - G.g20) * M[0]);
  o[5 * nq] = coef * (M[5] - G.rc * M[2] - G.sc * M[1] + (G.rc * G.sc - G.g21) * M[0]);
}
