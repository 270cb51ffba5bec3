// Triangle passes of the optimised step (order_exact 0): the corner
// coefficients with their node sums, and the RHS with its update, FP64, one
// thread per triangle.
//
// Same arithmetic as the reference-order kernels of lag2d_kernels.cu
// (b_tri_corner, b_tri_rhs) up to rounding.  Those keep the reference's loops
// over indexed arrays (normals, vertex states, node sums), which live in local
// memory, and its ~150 divisions and square roots; a triangle's pass is one
// dependent chain, so on meshes of one or a few waves of blocks that chain is the
// kernel's time.  Here everything is unrolled over compile-time tables into
// registers, the face vectors are not normalised (m = rho c |w an| and sigma.n A
// w = -p w an need no unit normal: 15 square roots, no division), the harmonic
// tau mean is one fraction, the RHS takes the face integral from the 30 node sums
// instead of the 120 corner coefficients, and the source's cosines come from
// cospi and the triple-angle formula.  Hybrid 128 x 128 (16,384 triangles, one
// wave): corner 62 -> 20 us, RHS 49 -> 19 us a launch.
#include <cuda_runtime.h>
#include <math.h>

#include "lag2d_device.cuh"

namespace lag2d {
namespace tri {

// sub-triangle vertices (0-based nodes), face slots (1-based, sign =
// orientation) and face weights (getriem_triasubg3, Getrhslaggauss.f90:12264-12302)
constexpr int kNode[4][3] = {{0, 3, 5}, {3, 4, 5}, {3, 1, 4}, {5, 4, 2}};
constexpr int kFace[4][6] = {{6, 1, 10, -7, -13, 12}, {7, 14, 8, 15, 9, 13}, {-14, 10, 2, 3, 11, -8}, {12, -9, -15, 11, 4, 5}};
constexpr double kA = 1.0 / 6.0, kB = 1.0 / 3.0, kC = 2.0 / 3.0;
constexpr double kW[4][6] = {{kA, kA, kB, kC, kC, kB}, {kC, kC, kC, kC, kC, kC}, {kC, kB, kA, kA, kB, kC}, {kB, kC, kC, kB, kA, kA}};
// 7-point rule of rutope (dgflo2d.f90:2232-2254)
constexpr double kG0 = 0.333333333333333, kG1 = 0.059715871789770, kG2 = 0.470142064105115, kG3 = 0.797426985353087,
                 kG4 = 0.101286507323456;
__device__ __forceinline__ double gr(int i) { constexpr double t[7] = {kG0, kG1, kG2, kG2, kG3, kG4, kG4}; return t[i]; }
__device__ __forceinline__ double gs(int i) { constexpr double t[7] = {kG0, kG2, kG1, kG2, kG4, kG3, kG4}; return t[i]; }
__device__ __forceinline__ double gw(int i) {
  constexpr double t[7] = {0.225000000000000, 0.132394152788506, 0.132394152788506, 0.132394152788506,
                           0.125939180544827, 0.125939180544827, 0.125939180544827};
  return t[i];
}
// reference coordinates of the nodes; vertex j of sub-triangle s
__device__ __forceinline__ double xv(int k) { constexpr double t[6] = {0.0, 1.0, 0.0, 0.5, 0.5, 0.0}; return t[k]; }
__device__ __forceinline__ double yv(int k) { constexpr double t[6] = {0.0, 0.0, 1.0, 0.0, 0.5, 0.5}; return t[k]; }
__device__ __forceinline__ int node(int s, int j) {
  constexpr int t[12] = {0, 3, 5, 3, 4, 5, 3, 1, 4, 5, 4, 2};
  return t[3 * s + j];
}

// 6-node shapes and derivatives (k a compile-time index after unrolling)
__device__ __forceinline__ constexpr double shp(int k, double r, double s) {
  const double t = 1.0 - r - s;
  return k == 0 ? t * (2.0 * t - 1.0) : k == 1 ? r * (2.0 * r - 1.0) : k == 2 ? s * (2.0 * s - 1.0)
       : k == 3 ? 4.0 * r * t : k == 4 ? 4.0 * r * s : 4.0 * s * t;
}
__device__ __forceinline__ constexpr double dshr(int k, double r, double s) {
  const double t = 1.0 - r - s;
  return k == 0 ? 1.0 - 4.0 * t : k == 1 ? 4.0 * r - 1.0 : k == 2 ? 0.0
       : k == 3 ? 4.0 * (1.0 - 2.0 * r - s) : k == 4 ? 4.0 * s : -4.0 * s;
}
__device__ __forceinline__ constexpr double dshs(int k, double r, double s) {
  const double t = 1.0 - r - s;
  return k == 0 ? 1.0 - 4.0 * t : k == 1 ? 0.0 : k == 2 ? 4.0 * s - 1.0
       : k == 3 ? -4.0 * r : k == 4 ? 4.0 * r : 4.0 * (1.0 - r - 2.0 * s);
}
// sum_k c_k x_k without the terms whose coefficient is 0 at compile time
#define TRI_SUM(coef, x)                          \
  [&] {                                           \
    double a_ = 0.0;                              \
    _Pragma("unroll") for (int k = 0; k < 6; k++) { \
      const double c_ = coef;                     \
      if (c_ != 0.0) a_ += c_ * x[k];             \
    }                                             \
    return a_;                                    \
  }()

struct Tri {
  double x[6], y[6];
  double rc, sc, g19, g20, g21;
};
__device__ __forceinline__ void basis(const Tri &T, double r, double s, double *b) {
  b[0] = 1.0;
  b[1] = 2.0 * (r - T.rc);
  b[2] = 2.0 * (s - T.sc);
  b[3] = 0.5 * b[1] * b[1] - T.g19;
  b[4] = 0.5 * b[2] * b[2] - T.g20;
  b[5] = b[1] * b[2] - T.g21;
}

// face vector (unit normal times area) of slot 1..15 (normals_tria): 1-6 the
// corner ends of the edges, 10-12 the edges' mid-nodes, 7-9 and 13-15 the two
// ends of the inner faces
template <int SLOT>
__device__ __forceinline__ void face(const Tri &T, double &vx, double &vy) {
  constexpr int i = SLOT - 1;
  if constexpr ((i >= 6 && i < 9) || i >= 12) {
    constexpr int f = i < 9 ? i - 6 : i - 12;
    constexpr double r = i < 9 ? -1.0 : 1.0;
    constexpr int a = f == 0 ? 3 : f == 1 ? 4 : 5, b = f == 0 ? 5 : f == 1 ? 3 : 4;
    constexpr double pr = f == 1 ? 0.5 : 0.25, ps = f == 2 ? 0.5 : 0.25;
    const double xm = TRI_SUM(shp(k, pr, ps), T.x), ym = TRI_SUM(shp(k, pr, ps), T.y);
    const double dx = (r - 0.5) * T.x[a] + (r + 0.5) * T.x[b] - 2.0 * r * xm;
    const double dy = (r - 0.5) * T.y[a] + (r + 0.5) * T.y[b] - 2.0 * r * ym;
    vx = -2.0 * dy;
    vy = 2.0 * dx;
  } else {
    constexpr int g = i < 6 ? i : i - 3;
    constexpr double pr[9] = {0, 1, 1, 0, 0, 0, 0.5, 0.5, 0}, ps[9] = {0, 0, 0, 1, 1, 0, 0, 0.5, 0.5};
    constexpr double r = pr[g], s = ps[g];
    constexpr int side = (g == 0 || g == 1 || g == 6) ? 0 : (g == 2 || g == 3 || g == 7) ? 1 : 2;
    double xr = 0.0, yr = 0.0, xs = 0.0, ys = 0.0;
    if constexpr (side != 2) { xr = TRI_SUM(dshr(k, r, s), T.x); yr = TRI_SUM(dshr(k, r, s), T.y); }
    if constexpr (side != 0) { xs = TRI_SUM(dshs(k, r, s), T.x); ys = TRI_SUM(dshs(k, r, s), T.y); }
    if constexpr (side == 0) { vx = yr; vy = -xr; }
    else if constexpr (side == 1) { vx = ys - yr; vy = xr - xs; }
    else { vx = -ys; vy = xs; }
  }
}
template <int C>
__device__ __forceinline__ void signed_face(const Tri &T, double &vx, double &vy) {
  face<(C > 0 ? C : -C)>(T, vx, vy);
  if (C < 0) { vx = -vx; vy = -vy; }
}

struct Corner {
  double rhoc, lim2;               // rho c; (1e12 c)^2
  double sub[4];                   // sub-cell density correction
  double st[6][4];                 // vertex state: 1/tau, u, v, e_int
  double dx[6], dy[6];             // u*_prev - u_vertex
};
// corner face F (0, 1) of vertex V of sub-triangle S: adds (m, m u, m v, sigma.n A)
template <int S, int V, int F>
__device__ __forceinline__ void corner(const Dev &d, const Tri &T, const Corner &C, int it, double P[6][5]) {
  constexpr int iv = kNode[S][V], code = kFace[S][2 * V + F];
  constexpr double w = kW[S][2 * V + F];
  double vx, vy;
  signed_face<code>(T, vx, vy);
  const double len = sqrt(vx * vx + vy * vy);
  double m = C.rhoc * w * len;
  const double j2 = C.dx[iv] * C.dx[iv] + C.dy[iv] * C.dy[iv];
  // the jump-direction branch: times |n . j|, j = du / |du|
  if (!(j2 < C.lim2)) m *= fabs(vx * C.dx[iv] + vy * C.dy[iv]) / (len * sqrt(j2));
  const double p = fmax(1.0e-15, (d.gamlg - 1.0) * (C.st[iv][0] + C.sub[S]) * C.st[iv][3]);
  const double c[5] = {m, m * C.st[iv][1], m * C.st[iv][2], -p * w * vx, -p * w * vy};
#pragma unroll
  for (int v = 0; v < 5; v++) P[iv][v] += c[v];
  if (d.tcf) {  // recorded for the adjoint
    const size_t nt = d.ntria;
#pragma unroll
    for (int v = 0; v < 5; v++) d.tcf[(v * 24 + F + 2 * (V + 3 * S)) * nt + it] = c[v];
  }
}

__device__ __forceinline__ void load(const Dev &d, int it, int pn[6], Tri &T) {
  const size_t nt = d.ntria;
#pragma unroll
  for (int k = 0; k < 6; k++) pn[k] = d.ipt[k * nt + it];
  T.rc = d.rc[it];
  T.sc = d.sc[it];
  T.g19 = d.g19[it];
  T.g20 = d.g20[it];
  T.g21 = d.g21[it];
#pragma unroll
  for (int k = 0; k < 6; k++) {
    T.x[k] = d.xs[pn[k]];
    T.y[k] = d.ys[pn[k]];
  }
}

// density correction of sub-triangle S (getrhosubgt_average2): initial mass over
// current volume, less the harmonic tau mean.  sum w det / tau is kept as one
// fraction; tau is scaled by the cell average so that the product stays near 1.
template <int S>
__device__ __forceinline__ double sub_density(const Dev &d, const Tri &T, const double *u, double msub) {
  // mid-edge points of the sub-triangle's own 6-node map, on the parent map
  constexpr double qr[9] = {0.25, 0.75, 0.75, 0.25, 0.0, 0.0, 0.25, 0.5, 0.25};
  constexpr double qs[9] = {0.0, 0.0, 0.25, 0.75, 0.75, 0.25, 0.25, 0.25, 0.5};
  constexpr int mid[4][3] = {{0, 6, 5}, {7, 8, 6}, {1, 2, 7}, {8, 3, 4}};
  double x[6], y[6];
#pragma unroll
  for (int j = 0; j < 3; j++) {
    const int n = node(S, j);
    x[j] = T.x[n];
    y[j] = T.y[n];
    const double r = qr[mid[S][j]], s = qs[mid[S][j]];
    x[3 + j] = TRI_SUM(shp(k, r, s), T.x);
    y[3 + j] = TRI_SUM(shp(k, r, s), T.y);
  }
  const double rt = 1.0 / u[0];
  double vol = 0.0, num = 0.0, den = 1.0;
#pragma unroll
  for (int g = 0; g < 7; g++) {
    const double r = gr(g), s = gs(g), t = 1.0 - r - s;
    const double xr = TRI_SUM(dshr(k, r, s), x), xs = TRI_SUM(dshs(k, r, s), x);
    const double yr = TRI_SUM(dshr(k, r, s), y), ys = TRI_SUM(dshs(k, r, s), y);
    const double dj = (0.5 * gw(g)) * (xr * ys - yr * xs);
    double b[6], tau = 0.0;
    basis(T, t * xv(node(S, 0)) + r * xv(node(S, 1)) + s * xv(node(S, 2)),
          t * yv(node(S, 0)) + r * yv(node(S, 1)) + s * yv(node(S, 2)), b);
#pragma unroll
    for (int k = 0; k < 6; k++)
      if (k < d.mdegr) tau += u[k] * b[k];
    tau *= rt;
    vol += dj;
    num = num * tau + dj * den;
    den *= tau;
  }
  return (msub - rt * num / den) / vol;
}

template <int NR>
__global__ void __launch_bounds__(64) k_corner(Dev d) {
  const int it = blockIdx.x * blockDim.x + threadIdx.x;
  if (it >= d.ntria) return;
  const int done = d.sc_dev->done;
  const size_t nc = d.ncell, nt = d.ntria;
  Tri T;
  int pn[6];
  double u[4][6], ms[4];
#pragma unroll
  for (int q = 0; q < 4; q++)
#pragma unroll
    for (int k = 0; k < 6; k++) u[q][k] = d.Us[(q * 6 + k) * nc + it];
#pragma unroll
  for (int s = 0; s < 4; s++) ms[s] = d.tmsub[s * nt + it];
  load(d, it, pn, T);
  Corner C;
#pragma unroll
  for (int k = 0; k < 6; k++) {
    C.dx[k] = d.us[pn[k]];
    C.dy[k] = d.vs[pn[k]];
  }
  if (done) return;
  const double eps = 1.0e-15, g = d.gamlg;
  const double rhoct = 1.0 / u[0][0];
  const double pctr = fmax(eps, (g - 1.0) * rhoct * (u[3][0] - 0.5 * (u[1][0] * u[1][0] + u[2][0] * u[2][0])));
  const double c = sqrt(fmax(eps, g * pctr * u[0][0]));
  C.rhoc = rhoct * c;
  C.lim2 = 1.0e24 * c * c;
  C.sub[0] = sub_density<0>(d, T, u[0], ms[0]);
  C.sub[1] = sub_density<1>(d, T, u[0], ms[1]);
  C.sub[2] = sub_density<2>(d, T, u[0], ms[2]);
  C.sub[3] = sub_density<3>(d, T, u[0], ms[3]);
#pragma unroll
  for (int v = 0; v < 6; v++) {
    double b[6], st[4];
    basis(T, xv(v), yv(v), b);
#pragma unroll
    for (int q = 0; q < 4; q++) {
      st[q] = 0.0;
#pragma unroll
      for (int k = 0; k < 6; k++)
        if (k < d.mdegr) st[q] += u[q][k] * b[k];
    }
    C.st[v][0] = 1.0 / st[0];
    C.st[v][1] = st[1];
    C.st[v][2] = st[2];
    C.st[v][3] = st[3] - 0.5 * (st[1] * st[1] + st[2] * st[2]);
    C.dx[v] -= st[1];
    C.dy[v] -= st[2];
  }
  double P[6][5];
#pragma unroll
  for (int k = 0; k < 6; k++)
#pragma unroll
    for (int v = 0; v < 5; v++) P[k][v] = 0.0;
#define TRI_SUB(S)                                                        \
  corner<S, 0, 0>(d, T, C, it, P); corner<S, 0, 1>(d, T, C, it, P);       \
  corner<S, 1, 0>(d, T, C, it, P); corner<S, 1, 1>(d, T, C, it, P);       \
  corner<S, 2, 0>(d, T, C, it, P); corner<S, 2, 1>(d, T, C, it, P);
  TRI_SUB(0) TRI_SUB(1) TRI_SUB(2) TRI_SUB(3)
#undef TRI_SUB
#pragma unroll
  for (int k = 0; k < 6; k++)
#pragma unroll
    for (int v = 0; v < NR; v++)
      d.tpart[(v * 6 + k) * nt + it] = NR == 3 && v > 0 ? P[k][v] - P[k][v + 2] : P[k][v];
}

// sum of the weights with which slot N (1..15) enters the mass flux of node V
__host__ __device__ constexpr double mass_weight(int V, int N) {
  double c = 0.0;
  for (int s = 0; s < 4; s++)
    for (int j = 0; j < 6; j++)
      if (kNode[s][j / 2] == V && (kFace[s][j] == N || kFace[s][j] == -N)) c += kFace[s][j] > 0 ? kW[s][j] : -kW[s][j];
  return c;
}
template <int V, int N>
__device__ __forceinline__ void mass_vec(const Tri &T, double &tx, double &ty) {
  constexpr double c = mass_weight(V, N);
  if constexpr (c > 1e-12 || c < -1e-12) {
    double vx, vy;
    face<N>(T, vx, vy);
    tx += c * vx;
    ty += c * vy;
  }
  if constexpr (N < 15) mass_vec<V, N + 1>(T, tx, ty);
}
// face integral at node V: the corner forces are affine in the node's velocity,
// sum_f F_f = u* P0 - (P1, P2), plus (P3, P4) where sigma.n A has its own rows
template <int V, int NR>
__device__ __forceinline__ void face_node(const Tri &T, double us, double vs, const double P[NR], double R[4][6]) {
  double tx = 0.0, ty = 0.0, b[6];
  mass_vec<V, 1>(T, tx, ty);
  basis(T, xv(V), yv(V), b);
  double f0 = us * P[0] - P[1], f1 = vs * P[0] - P[2];
  if (NR == 5) {
    f0 = P[NR - 2] + f0;
    f1 = P[NR - 1] + f1;
  }
  const double tw = us * tx + vs * ty, fe = us * f0 + vs * f1;
#pragma unroll
  for (int k = 0; k < 6; k++) {
    R[0][k] += tw * b[k];
    R[1][k] += f0 * b[k];
    R[2][k] += f1 * b[k];
    R[3][k] += fe * b[k];
  }
}

template <int NR>
__global__ void __launch_bounds__(64) k_rhs(Dev d, const double *usn, const double *vsn, int fuse, double alfa) {
  const int it = blockIdx.x * blockDim.x + threadIdx.x;
  if (it >= d.ntria) return;
  const int done = d.sc_dev->done;
  const size_t nc = d.ncell, nt = d.ntria;
  const double g = d.gamlg;
  Tri T;
  int pn[6];
  double u[4][6], P[6][NR], us[6], vs[6];
#pragma unroll
  for (int q = 0; q < 4; q++)
#pragma unroll
    for (int k = 0; k < 6; k++) u[q][k] = d.Us[(q * 6 + k) * nc + it];
#pragma unroll
  for (int k = 0; k < 6; k++)
#pragma unroll
    for (int v = 0; v < NR; v++) P[k][v] = d.tpart[(v * 6 + k) * nt + it];
  load(d, it, pn, T);
#pragma unroll
  for (int k = 0; k < 6; k++) {
    us[k] = usn[pn[k]];
    vs[k] = vsn[pn[k]];
  }
  if (done) return;
  double R[4][6];
#pragma unroll
  for (int q = 0; q < 4; q++)
#pragma unroll
    for (int k = 0; k < 6; k++) R[q][k] = 0.0;
  face_node<0, NR>(T, us[0], vs[0], P[0], R);
  face_node<1, NR>(T, us[1], vs[1], P[1], R);
  face_node<2, NR>(T, us[2], vs[2], P[2], R);
  face_node<3, NR>(T, us[3], vs[3], P[3], R);
  face_node<4, NR>(T, us[4], vs[4], P[4], R);
  face_node<5, NR>(T, us[5], vs[5], P[5], R);
  // volume integral (cofactor form, 7-point rule) and, on Taylor-Green, the
  // energy source on the same points
  const double csrc = d.ncase == 1 ? 0.25 * 3.14159265358979311599796346854 / (g - 1.0) : 0.0;
#pragma unroll
  for (int i = 0; i < 7; i++) {
    const double r = gr(i), s = gs(i), w = 0.5 * gw(i);
    const double xr = TRI_SUM(dshr(k, r, s), T.x), xs = TRI_SUM(dshs(k, r, s), T.x);
    const double yr = TRI_SUM(dshr(k, r, s), T.y), ys = TRI_SUM(dshs(k, r, s), T.y);
    double b[6], un[4];
    basis(T, r, s, b);
#pragma unroll
    for (int q = 0; q < 4; q++) {
      un[q] = 0.0;
#pragma unroll
      for (int k = 0; k < 6; k++)
        if (k < d.mdegr) un[q] += u[q][k] * b[k];
    }
    const double pres = (g - 1.0) / un[0] * (un[3] - 0.5 * (un[1] * un[1] + un[2] * un[2]));
    // basis gradients (2,0), (0,2), (2 b1,0), (0,2 b2), (2 b2, 2 b1)
    const double w2 = 2.0 * w, wp = w2 * pres;
    const double a = ys * un[1] - xs * un[2], c = xr * un[2] - yr * un[1];
    const double grad[5][2] = {{1.0, 0.0}, {0.0, 1.0}, {b[1], 0.0}, {0.0, b[2]}, {b[2], b[1]}};
#pragma unroll
    for (int k = 0; k < 5; k++) {
      const double br = grad[k][0], bs = grad[k][1];
      double fv, g0, g1;
      if (k == 0 || k == 2) { fv = br * a; g0 = br * ys; g1 = -br * xs; }
      else if (k == 1 || k == 3) { fv = bs * c; g0 = -bs * yr; g1 = bs * xr; }
      else { fv = br * a + bs * c; g0 = br * ys - bs * yr; g1 = bs * xr - br * xs; }
      R[0][k + 1] -= w2 * fv;
      R[1][k + 1] += wp * g0;
      R[2][k + 1] += wp * g1;
      R[3][k + 1] += wp * fv;
    }
    if (d.ncase == 1) {
      const double xg = TRI_SUM(shp(k, r, s), T.x), yg = TRI_SUM(shp(k, r, s), T.y);
      const double cx = cospi(xg), cy = cospi(yg);
      const double c3x = cx * (4.0 * cx * cx - 3.0), c3y = cy * (4.0 * cy * cy - 3.0);
      const double src = csrc * (c3x * cy - c3y * cx) * (w * (xr * ys - yr * xs));
#pragma unroll
      for (int k = 0; k < 6; k++) R[3][k] += src * b[k];
    }
  }
  if (!fuse) {
#pragma unroll
    for (int q = 0; q < 4; q++)
#pragma unroll
      for (int k = 0; k < 6; k++) d.rhs[(q * 6 + k) * nc + it] = R[q][k];
    return;
  }
  const double dt = d.sc_dev->dtfix, oma = 1.0 - alfa;
  double am[16];
#pragma unroll
  for (int i = 0; i < 16; i++) am[i] = d.amatr[i * nc + it];
  constexpr int IDX[5][5] = {{0, 1, 2, 3, 4}, {1, 5, 6, 7, 8}, {2, 6, 9, 10, 11}, {3, 7, 10, 12, 13}, {4, 8, 11, 13, 14}};
#pragma unroll
  for (int q = 0; q < 4; q++) {
#pragma unroll
    for (int k = 0; k < 6; k++) R[q][k] *= dt;
    const size_t base = (size_t)(q * 6) * nc + it;
#pragma unroll
    for (int i = 0; i < 6; i++) {
      double acc = 0.0;
      if (i == 0) acc = am[15] * R[q][0];
      else
#pragma unroll
        for (int j = 0; j < 5; j++) acc += am[IDX[i > 0 ? i - 1 : 0][j]] * R[q][j + 1];
      d.Uo[base + i * nc] = alfa * d.Un[base + i * nc] + oma * (u[q][i] + acc);
    }
  }
}

}  // namespace tri

void launch_fast_tri_corner(const Dev &d, cudaStream_t st) {
  if (!d.ntria) return;
  if (d.nrow == 3) tri::k_corner<3><<<(d.ntria + 63) / 64, 64, 0, st>>>(d);
  else tri::k_corner<5><<<(d.ntria + 63) / 64, 64, 0, st>>>(d);
}
void launch_fast_tri_rhs(const Dev &d, cudaStream_t st, const double *usn, const double *vsn, int fuse, double alfa) {
  if (!d.ntria) return;
  if (d.nrow == 3) tri::k_rhs<3><<<(d.ntria + 63) / 64, 64, 0, st>>>(d, usn, vsn, fuse, alfa);
  else tri::k_rhs<5><<<(d.ntria + 63) / 64, 64, 0, st>>>(d, usn, vsn, fuse, alfa);
}

}  // namespace lag2d
