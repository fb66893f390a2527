// Vertex-tuple energies in translation-free coordinates.
//
// An energy of A vertices that does not change under a translation depends
// on M = A - 1 vectors y_p = sum_a Q[a][p] x_a only, with Q's columns
// orthonormal and orthogonal to (1, ..., 1).  Then the gradient with respect
// to vertex a is sum_p Q[a][p] dE/dy_p, the 3A x 3A Hessian is
// H = (Q (x) I) K (Q (x) I)^T with K = d2E/dy2 (3M x 3M), and because Q (x) I
// has orthonormal columns the nonzero eigenvalues of H are those of K:
//   proj(H) = (Q (x) I) proj(K) (Q (x) I)^T
// exactly.  So the derivatives, the PSD test and the negative modes run on
// 45 packed entries for four vertices instead of 78 (21 for 45 with three),
// which is what bounds these kernels: FP64 work and registers a thread.
//
// The energies here are functions of a few invariants of the y_p (the plane
// distance y0 . n / |n| with n = y1 x y2 for point-triangle and edge-edge
// pairs, the hinge angle, the metric of a membrane), so K is written in
// closed form: the invariants' gradients (rank-one terms) and their sparse
// second derivatives.
#pragma once

#include "ys_ad.cuh"
#include "ys_common.cuh"

namespace ys {

struct D3v {
  double x, y, z;
};
__device__ __forceinline__ D3v operator+(D3v a, D3v b) { return {a.x + b.x, a.y + b.y, a.z + b.z}; }
__device__ __forceinline__ D3v operator-(D3v a, D3v b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ D3v operator*(double s, D3v a) { return {s * a.x, s * a.y, s * a.z}; }
__device__ __forceinline__ double dot(D3v a, D3v b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ D3v cross(D3v a, D3v b) {
  return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}
__device__ __forceinline__ double at(const D3v& a, int i) { return i == 0 ? a.x : (i == 1 ? a.y : a.z); }
__device__ __forceinline__ D3v d3v(const double (&p)[3]) { return {p[0], p[1], p[2]}; }

// [w]x: the matrix of v -> w x v.
__device__ __forceinline__ double skew(const D3v& w, int r, int c) {
  if (r == c) return 0.0;
  const int k = 3 - r - c;
  return ((r + 1) % 3 == c) ? -at(w, k) : at(w, k);
}

// Value, gradient and Hessian (packed upper) over the M vectors y.
template <int A>
struct Reduced {
  static constexpr int M = A - 1, N = 3 * M, H = N * (N + 1) / 2;
  double v;
  double g[N];
  double k[H];
};

// Entry pairs (i, j) of block (p, q), p <= q, restricted to i <= j.
template <int N, class F>
__device__ __forceinline__ void add_block(double (&k)[N * (N + 1) / 2], int p, int q, F&& f) {
#pragma unroll
  for (int r = 0; r < 3; ++r)
#pragma unroll
    for (int c = 0; c < 3; ++c)
      if (3 * p + r <= 3 * q + c) k[utri<N>(3 * p + r, 3 * q + c)] += f(r, c);
}

// Orthonormal reduction of 2, 3 and 4 vertices (Q[a][p]).
// Four vertices as two pairs (edge-edge): half the sums and differences.
struct QPairs {
  __host__ __device__ static constexpr double q(int a, int p) {
    return p == 0 ? (a < 2 ? 0.5 : -0.5) : p == 1 ? (a % 2 == 0 ? 0.5 : -0.5) : (a == 0 || a == 3 ? 0.5 : -0.5);
  }
};
constexpr double kSqrt1_2 = 0.70710678118654752440;   // 1 / sqrt(2)
constexpr double kSqrt3_2 = 1.22474487139158904910;   // sqrt(3 / 2)
constexpr double kSqrt2_3 = 0.81649658092772603273;   // sqrt(2 / 3)
constexpr double kSqrt1_6 = 0.40824829046386301637;   // 1 / sqrt(6)
constexpr double kSqrt3_4 = 0.86602540378443864676;   // sqrt(3) / 2
constexpr double kSqrt1_12 = 0.28867513459481288225;  // 1 / (2 sqrt(3))
// Vertex 0 against the triangle 1, 2, 3.
struct QPointTriangle {
  __host__ __device__ static constexpr double q(int a, int p) {
    return p == 0 ? (a == 0 ? kSqrt3_4 : -kSqrt1_12)
                  : p == 1 ? (a == 1 ? kSqrt1_2 : a == 2 ? -kSqrt1_2 : 0.0)
                           : (a == 0 ? 0.0 : a == 3 ? -kSqrt2_3 : kSqrt1_6);
  }
};
// Hinge: edge 0-1, wings 2 and 3.
struct QHinge {
  __host__ __device__ static constexpr double q(int a, int p) {
    return p == 0 ? (a < 2 ? -0.5 : 0.5)
                  : p == 1 ? (a == 0 ? -kSqrt1_2 : a == 1 ? kSqrt1_2 : 0.0)
                           : (a == 2 ? -kSqrt1_2 : a == 3 ? kSqrt1_2 : 0.0);
  }
};
// Vertex 0 against the edge 1-2.
struct QThree {
  __host__ __device__ static constexpr double q(int a, int p) {
    return p == 0 ? (a == 0 ? kSqrt2_3 : -kSqrt1_6) : (a == 1 ? kSqrt1_2 : a == 2 ? -kSqrt1_2 : 0.0);
  }
};
struct QTwo {
  __host__ __device__ static constexpr double q(int a, int) { return a == 0 ? kSqrt1_2 : -kSqrt1_2; }
};

// Derivatives of the log-barrier kappa u^2 L^2 (see barrier_of) at d.
__device__ __forceinline__ double barrier_value(double d, double dhat, double kappa, double& df, double& d2f) {
  const double u = d - dhat, L = log(d / dhat), ix = 1.0 / d;
  df = kappa * (2.0 * u * L * L + 2.0 * u * u * L * ix);
  d2f = kappa * (2.0 * L * L + 8.0 * u * L * ix + 2.0 * u * u * ix * ix - 2.0 * u * u * L * ix * ix);
  return kappa * u * u * L * L;
}

// E = b(d), d = sigma (y0 . n)^2 / |n|^2 with n = y1 x y2: the squared
// distance of a point from a triangle's plane (sigma 4/3 with QPointTriangle)
// and of two lines (sigma 1 with QPairs).
__device__ __forceinline__ void plane_barrier(const D3v (&y)[3], double sigma, double dhat, double kappa,
                                              Reduced<4>& e) {
  const D3v n = cross(y[1], y[2]);
  const double u = dot(y[0], n), s = dot(n, n), is = 1.0 / s;
  const double d = sigma * u * u * is;
  double f1, f2;
  e.v = barrier_value(d, dhat, kappa, f1, f2);
  const double du = 2.0 * sigma * u * is, ds = -d * is;
  const double Eu = f1 * du, Es = f1 * ds;
  const double Euu = f2 * du * du + f1 * (2.0 * sigma * is);
  const double Eus = f2 * du * ds - f1 * du * is;
  const double Ess = f2 * ds * ds + f1 * (2.0 * d * is * is);
  const D3v gu[3] = {n, cross(y[2], y[0]), cross(y[0], y[1])};
  const D3v gs[3] = {{0.0, 0.0, 0.0}, 2.0 * cross(y[2], n), 2.0 * cross(n, y[1])};
#pragma unroll
  for (int p = 0; p < 3; ++p) {
    const D3v g = p == 0 ? Eu * gu[0] : Eu * gu[p] + Es * gs[p];
    e.g[3 * p] = g.x;
    e.g[3 * p + 1] = g.y;
    e.g[3 * p + 2] = g.z;
  }
  // rank-one terms: (Euu gu + Eus gs) gu^T + (Eus gu + Ess gs) gs^T
  D3v a[3], b[3];
#pragma unroll
  for (int p = 0; p < 3; ++p) {
    a[p] = p == 0 ? Euu * gu[0] : Euu * gu[p] + Eus * gs[p];
    b[p] = p == 0 ? Eus * gu[0] : Eus * gu[p] + Ess * gs[p];
  }
#pragma unroll
  for (int i = 0; i < 9; ++i)
#pragma unroll
    for (int j = i; j < 9; ++j) {
      double t = at(a[i / 3], i % 3) * at(gu[j / 3], j % 3);
      if (j >= 3) t += at(b[i / 3], i % 3) * at(gs[j / 3], j % 3);
      e.k[utri<9>(i, j)] = t;
    }
  // second derivatives of u (trilinear): skew blocks
  const D3v w01 = (-Eu) * y[2], w02 = Eu * y[1], w12 = (-Eu) * y[0];
  add_block<9>(e.k, 0, 1, [&](int r, int c) { return skew(w01, r, c); });
  add_block<9>(e.k, 0, 2, [&](int r, int c) { return skew(w02, r, c); });
  // and of s = |y1|^2 |y2|^2 - (y1 . y2)^2
  const double s11 = 2.0 * Es * dot(y[2], y[2]), s22 = 2.0 * Es * dot(y[1], y[1]), s12 = -2.0 * Es * dot(y[1], y[2]);
  const D3v e1 = (2.0 * Es) * y[1], e2 = (2.0 * Es) * y[2];
  add_block<9>(e.k, 1, 1, [&](int r, int c) { return (r == c ? s11 : 0.0) - at(e2, r) * at(y[2], c); });
  add_block<9>(e.k, 2, 2, [&](int r, int c) { return (r == c ? s22 : 0.0) - at(e1, r) * at(y[1], c); });
  add_block<9>(e.k, 1, 2, [&](int r, int c) {
    return (r == c ? s12 : skew(w12, r, c)) + 2.0 * at(e1, r) * at(y[2], c) - at(e2, r) * at(y[1], c);
  });
}

// E = b(d), d = 3/2 |y0 x y1|^2 / |y1|^2: a point against an edge's line.
__device__ __forceinline__ void line_barrier(const D3v (&y)[2], double dhat, double kappa, Reduced<3>& e) {
  const D3v n = cross(y[0], y[1]);
  const double s = dot(n, n), q = dot(y[1], y[1]), iq = 1.0 / q;
  const double d = 1.5 * s * iq;
  double f1, f2;
  e.v = barrier_value(d, dhat, kappa, f1, f2);
  const double ds = 1.5 * iq, dq = -d * iq;
  const double Es = f1 * ds, Eq = f1 * dq;
  const double Ess = f2 * ds * ds, Esq = f2 * ds * dq - f1 * ds * iq, Eqq = f2 * dq * dq + f1 * (2.0 * d * iq * iq);
  const D3v gs[2] = {2.0 * cross(y[1], n), 2.0 * cross(n, y[0])};
  const D3v gq = 2.0 * y[1];
#pragma unroll
  for (int p = 0; p < 2; ++p) {
    const D3v g = p == 0 ? Es * gs[0] : Es * gs[1] + Eq * gq;
    e.g[3 * p] = g.x;
    e.g[3 * p + 1] = g.y;
    e.g[3 * p + 2] = g.z;
  }
  const D3v a[2] = {Ess * gs[0], Ess * gs[1] + Esq * gq}, b[2] = {Esq * gs[0], Esq * gs[1] + Eqq * gq};
#pragma unroll
  for (int i = 0; i < 6; ++i)
#pragma unroll
    for (int j = i; j < 6; ++j) {
      double t = at(a[i / 3], i % 3) * at(gs[j / 3], j % 3);
      if (j >= 3) t += at(b[i / 3], i % 3) * at(gq, j % 3);
      e.k[utri<6>(i, j)] = t;
    }
  const double s00 = 2.0 * Es * dot(y[1], y[1]), s11 = 2.0 * Es * dot(y[0], y[0]) + 2.0 * Eq;
  const double s01 = -2.0 * Es * dot(y[0], y[1]);
  const D3v e0 = (2.0 * Es) * y[0], e1 = (2.0 * Es) * y[1];
  add_block<6>(e.k, 0, 0, [&](int r, int c) { return (r == c ? s00 : 0.0) - at(e1, r) * at(y[1], c); });
  add_block<6>(e.k, 1, 1, [&](int r, int c) { return (r == c ? s11 : 0.0) - at(e0, r) * at(y[0], c); });
  add_block<6>(e.k, 0, 1, [&](int r, int c) {
    return (r == c ? s01 : 0.0) + 2.0 * at(e0, r) * at(y[1], c) - at(e1, r) * at(y[0], c);
  });
}

// E = b(2 |y0|^2): two points.
__device__ __forceinline__ void point_barrier(const D3v& y, double dhat, double kappa, Reduced<2>& e) {
  double f1, f2;
  e.v = barrier_value(2.0 * dot(y, y), dhat, kappa, f1, f2);
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    e.g[i] = 4.0 * f1 * at(y, i);
#pragma unroll
    for (int j = i; j < 3; ++j) e.k[utri<3>(i, j)] = 16.0 * f2 * at(y, i) * at(y, j) + (i == j ? 4.0 * f1 : 0.0);
  }
}

// E = w (theta - theta0)^2 of a hinge.  With e the edge and a, b the wings
// seen from the edge's midpoint, theta is the angle of b minus that of a
// about e (up to a constant): d theta/da = -|e| na / |na|^2 with na = e x a,
// d theta/db = |e| nb / |nb|^2, and d theta/de = -(ca ga + cb gb) with ca, cb
// the wings' coordinates along e.  y = (y0, y1, y2) by QHinge gives
// e = sqrt2 y1, a = y0 - y2 / sqrt2, b = y0 + y2 / sqrt2.
__device__ __forceinline__ void hinge_energy(const D3v (&y)[3], double w, double dtheta, Reduced<4>& out) {
  const D3v e = 1.41421356237309504880 * y[1];
  const D3v h = kSqrt1_2 * y[2];
  const D3v a = y[0] - h, b = y[0] + h;
  const D3v na = cross(e, a), nb = cross(e, b);
  const double le2 = dot(e, e), le = sqrt(le2), ile2 = 1.0 / le2;
  const double ia = 1.0 / dot(na, na), ib = 1.0 / dot(nb, nb);
  const double ca = dot(a, e) * ile2, cb = dot(b, e) * ile2;
  const D3v ga = (-le * ia) * na, gb = (le * ib) * nb;
  const D3v ge = (-ca) * ga - cb * gb;
  out.v = w * dtheta * dtheta;
  const double c1 = 2.0 * w * dtheta, c2 = 2.0 * w;
  const D3v gy[3] = {ga + gb, 1.41421356237309504880 * ge, kSqrt1_2 * (gb - ga)};
#pragma unroll
  for (int i = 0; i < 9; ++i) {
    out.g[i] = c1 * at(gy[i / 3], i % 3);
#pragma unroll
    for (int j = i; j < 9; ++j) out.k[utri<9>(i, j)] = c2 * at(gy[i / 3], i % 3) * at(gy[j / 3], j % 3);
  }
  // second derivatives of theta (times c1): H_aa, H_bb symmetric, H_ab = 0,
  // H_ae, H_be, H_ee
  const D3v ra = (c1 * le * ia * ia) * cross(na, e), rb = (-c1 * le * ib * ib) * cross(nb, e);
  const D3v qa = (c1 * le * ia) * a, qb = (-c1 * le * ib) * b;  // skew parts of H_ae, H_be
  const double ea = -c1 * ia / le, eb = c1 * ib / le;
  const D3v ta = (-2.0 * c1 * le * ia * ia) * cross(na, a), tb = (2.0 * c1 * le * ib * ib) * cross(nb, b);
  const D3v va = ea * e + ta, vb = eb * e + tb;  // H_ae = na va^T + [qa]x
  const D3v ua = (c1 * ile2) * (a - (2.0 * ca) * e), ub = (c1 * ile2) * (b - (2.0 * cb) * e);
  auto haa = [&](int r, int c) { return at(na, r) * at(ra, c) + at(ra, r) * at(na, c); };
  auto hbb = [&](int r, int c) { return at(nb, r) * at(rb, c) + at(rb, r) * at(nb, c); };
  auto hae = [&](int r, int c) { return at(na, r) * at(va, c) + skew(qa, r, c); };
  auto hbe = [&](int r, int c) { return at(nb, r) * at(vb, c) + skew(qb, r, c); };
  auto hee = [&](int r, int c) {
    return -(at(ga, r) * at(ua, c) + ca * hae(r, c) + at(gb, r) * at(ub, c) + cb * hbe(r, c));
  };
#pragma unroll
  for (int r = 0; r < 3; ++r)
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const double A = haa(r, c), B = hbb(r, c);
      if (r <= c) {
        out.k[utri<9>(r, c)] += A + B;
        out.k[utri<9>(6 + r, 6 + c)] += 0.5 * (A + B);
        out.k[utri<9>(3 + r, 3 + c)] += hee(r, c) + hee(c, r);  // 2 H_ee, symmetrised
      }
      out.k[utri<9>(r, 6 + c)] += kSqrt1_2 * (B - A);
      const double x = hae(r, c), z = hbe(r, c);
      out.k[utri<9>(r, 3 + c)] += 1.41421356237309504880 * (x + z);
      out.k[utri<9>(3 + c, 6 + r)] += z - x;
    }
}

// Membrane energy of the metric A = f0.f0, B = f1.f1, C = f0.f1 with
// f_j = sum_p m[p][j] y_p: first derivatives pa, pb, pc and second ones
// paa, pbb, pab, pcc of the energy.
__device__ __forceinline__ void metric_energy(const D3v& f0, const D3v& f1, const double (&m)[2][2], double pa,
                                              double pb, double pc, double paa, double pbb, double pab, double pcc,
                                              Reduced<3>& e) {
  D3v gA[2], gB[2], gC[2];
#pragma unroll
  for (int p = 0; p < 2; ++p) {
    gA[p] = (2.0 * m[p][0]) * f0;
    gB[p] = (2.0 * m[p][1]) * f1;
    gC[p] = m[p][0] * f1 + m[p][1] * f0;
    const D3v g = pa * gA[p] + pb * gB[p] + pc * gC[p];
    e.g[3 * p] = g.x;
    e.g[3 * p + 1] = g.y;
    e.g[3 * p + 2] = g.z;
  }
#pragma unroll
  for (int p = 0; p < 2; ++p) {
    const D3v u = paa * gA[p] + pab * gB[p], v = pab * gA[p] + pbb * gB[p], t = pcc * gC[p];
#pragma unroll
    for (int q = p; q < 2; ++q) {
      const double iso = 2.0 * pa * m[p][0] * m[q][0] + 2.0 * pb * m[p][1] * m[q][1] +
                         pc * (m[p][0] * m[q][1] + m[p][1] * m[q][0]);
#pragma unroll
      for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int c = 0; c < 3; ++c)
          if (3 * p + r <= 3 * q + c)
            e.k[utri<6>(3 * p + r, 3 * q + c)] = at(u, r) * at(gA[q], c) + at(v, r) * at(gB[q], c) +
                                                 at(t, r) * at(gC[q], c) + (r == c ? iso : 0.0);
    }
  }
}

// Largest |diagonal entry| of the vertex-space Hessian (Q (x) I) K (Q (x) I)^T
// and 1: the scale of the PSD test's tolerance (psd_test_packed).
template <class Q, int A>
__device__ __forceinline__ double vertex_scale(const double (&k)[Reduced<A>::H]) {
  constexpr int M = A - 1, N = 3 * M;
  double scale = 1.0;
#pragma unroll
  for (int a = 0; a < A; ++a)
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      double d = 0.0;
#pragma unroll
      for (int p = 0; p < M; ++p)
#pragma unroll
        for (int q = 0; q < M; ++q)
          if (Q::q(a, p) != 0.0 && Q::q(a, q) != 0.0) d += (Q::q(a, p) * Q::q(a, q)) * k[sym<N>(3 * p + c, 3 * q + c)];
      scale = fmax(scale, fabs(d));
    }
  return scale;
}

// Blocks of the vertex-space Hessian, a row at a time: row(a) forms
// Y_q = sum_p Q[a][p] K_pq from packed K (entry i at k[i * stride], in the
// shared stash), block(b) is sum_q Q[b][q] Y_q.
template <class Q, int A>
struct VertexRows {
  static constexpr int M = A - 1, N = 3 * M;
  const double* k;
  int stride;
  double y[M][3][3];
  __device__ __forceinline__ void row(int a) {
#pragma unroll
    for (int q = 0; q < M; ++q)
#pragma unroll
      for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          double d = 0.0;
#pragma unroll
          for (int p = 0; p < M; ++p)
            if (Q::q(a, p) != 0.0) d += Q::q(a, p) * k[sym<N>(3 * p + r, 3 * q + c) * stride];
          y[q][r][c] = d;
        }
  }
  __device__ __forceinline__ void block(int, int b, double (&blk)[3][3]) const {
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        double d = 0.0;
#pragma unroll
        for (int q = 0; q < M; ++q)
          if (Q::q(b, q) != 0.0) d += Q::q(b, q) * y[q][r][c];
        blk[r][c] = d;
      }
  }
};

// Packed lower triangle of the vertex-space Hessian's first ROWS vertices.
template <class Q, int A, int ROWS>
__device__ __forceinline__ void vertex_lower(const double* k, int stride, double* s) {
  VertexRows<Q, A> v{k, stride};
#pragma unroll
  for (int i = 0; i < ROWS; ++i) {
    v.row(i);
#pragma unroll
    for (int j = 0; j <= i; ++j) {
      double blk[3][3];
      v.block(i, j, blk);
#pragma unroll
      for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int c = 0; c < 3; ++c)
          if (3 * j + c <= 3 * i + r) s[tri(3 * i + r, 3 * j + c)] = blk[r][c];
    }
  }
}

// Shared-memory doubles a thread needs for write_block_records.
constexpr int kRecordRow = 9;

// Records of a local Hessian of A arguments of size 3 given by its blocks
// (v.row(a), then v.block(a, b, out) for the blocks of row a):
// target arguments (code >= 2) merged when they repeat, blocks transposed
// when the row DoF exceeds the column DoF (hessianKernelNoProject.pyx:94-264),
// in the slot order of the coordinates.  Called by whole warps, lanes without
// an element with live == false.  A record is 72 contiguous bytes at its own
// place: a lane storing its own record touches 32 lines an instruction.  With
// SHARED the warp passes its 32 records through shared memory (`rows`, the
// block's kRecordRow doubles a thread) and stores them in runs of 9 lanes, 4-5
// lines an instruction: the SNH evaluation, bound by its stores, 0.96 ->
// 0.56 ms at 1.5M tets.  The projection kernels run 8 warps an SM and are bound
// by latency, where the detour costs more than it gives: they store directly.
template <int A, bool SHARED, class Rows>
__device__ __forceinline__ void write_block_records(bool live, const uint32_t (&code)[A], uint32_t occ0,
                                                    const uint32_t* __restrict__ record, double* __restrict__ out,
                                                    double* rows, Rows&& v) {
  constexpr unsigned kAll = 0xffffffffu;
  constexpr uint32_t kNone = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  double* const warp_rows = rows + (threadIdx.x & ~31u) * kRecordRow;
  bool dup = false;
#pragma unroll
  for (int a = 0; a < A; ++a)
#pragma unroll
    for (int b = a + 1; b < A; ++b) dup |= (code[a] >= 2 && code[a] == code[b]);
  // Common case: every target argument is its own group (compile-time indices).
  uint32_t next = occ0;
#pragma unroll
  for (int ai = 0; ai < A; ++ai) {
    v.row(ai);
#pragma unroll
    for (int bi = ai; bi < A; ++bi) {
      const bool w = live && !dup && code[ai] >= 2 && code[bi] >= 2;
      if constexpr (!SHARED) {
        if (!w) continue;
        double blk[3][3];
        v.block(ai, bi, blk);
        double* dst = out + record[next++];
        const bool upper = code[ai] < code[bi];
#pragma unroll
        for (int k = 0; k < 3; ++k)
#pragma unroll
          for (int l = 0; l < 3; ++l) dst[3 * k + l] = upper ? blk[k][l] : blk[l][k];
        continue;
      }
      if (!__any_sync(kAll, w)) continue;
      uint32_t off = kNone;
      __syncwarp();
      if (w) {
        off = record[next++];
        double blk[3][3];
        v.block(ai, bi, blk);
        const bool upper = code[ai] < code[bi];
#pragma unroll
        for (int k = 0; k < 3; ++k)
#pragma unroll
          for (int l = 0; l < 3; ++l) warp_rows[kRecordRow * lane + 3 * k + l] = upper ? blk[k][l] : blk[l][k];
      }
      __syncwarp();
#pragma unroll
      for (int i = 0; i < kRecordRow; ++i) {
        const int e = 32 * i + lane, r = e / kRecordRow;
        const uint32_t o = __shfl_sync(kAll, off, r);
        if (o != kNone) out[o + (uint32_t)(e - kRecordRow * r)] = warp_rows[e];
      }
    }
  }
  if (!live || !dup) return;
  int first[A];
  int nfirst = 0;
  int group[A];
#pragma unroll
  for (int a = 0; a < A; ++a) {
    group[a] = -1;
    if (code[a] < 2) continue;
    int gsel = -1;
    for (int q = 0; q < nfirst; ++q)
      if (code[first[q]] == code[a]) gsel = q;
    if (gsel < 0) { first[nfirst] = a; gsel = nfirst++; }
    group[a] = gsel;
  }
  uint32_t occ = occ0;
  for (int gi = 0; gi < nfirst; ++gi) {
    for (int gj = gi; gj < nfirst; ++gj) {
      double acc[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
#pragma unroll
      for (int a = 0; a < A; ++a) {
        if (group[a] != gi) continue;
        v.row(a);
#pragma unroll
        for (int b = 0; b < A; ++b) {
          if (group[b] != gj) continue;
          double blk[3][3];
          v.block(a, b, blk);
#pragma unroll
          for (int k = 0; k < 3; ++k)
#pragma unroll
            for (int l = 0; l < 3; ++l) acc[k][l] += blk[k][l];
        }
      }
      double* dst = out + record[occ];
      const bool upper = code[first[gi]] < code[first[gj]];
#pragma unroll
      for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int l = 0; l < 3; ++l) dst[3 * k + l] = upper ? acc[k][l] : acc[l][k];
      ++occ;
    }
  }
}

}  // namespace ys
