// Jacobi rotations of the MLS fit (mls.cu): IEEE arithmetic in the order of the
// CPU restatement, bit for bit, where this is compiled without contraction.
#pragma once

#include "common.cuh"

namespace pacman_b200 {

// Packed upper-triangle position of (i, j) in an M x M symmetric matrix.
__host__ __device__ constexpr int sym_at(int i, int j, int M) {
  return i <= j ? i * M - i * (i - 1) / 2 + (j - i) : j * M - j * (j - 1) / 2 + (i - j);
}

// A thread's column of a [K][128] array in shared memory.
struct MlsColumn {
  double *p;
  __device__ __forceinline__ double &operator[](int i) const { return p[128 * i]; }
};

// RN(sqrt(x)) for x in [1, 1e40]: two Goldschmidt steps for g ~ sqrt(x), h ~
// 1 / (2 sqrt(x)), then RN(g + (x - g g) h) (Markstein, IBM J. Res. Dev. 34(1),
// 1990).  Both steps leave h within 2^-52 relatively (roundings only).  With a
// 53-bit integer M and x scaled to an integer X, the root lies (X - (M + 1/2)^2)
// / (2 M) from the midpoint M + 1/2, X - (M + 1/2)^2 = j - 1/4 with an integer
// j, and the error of the correction can only matter for |j| <= 7: those X are
// the few solutions of M^2 + M + j = 0 modulo the spacing of X, and the tests go
// through all of them.
// The divisions beside it are the compiler's: Markstein's theorem needs a
// correctly rounded reciprocal, which costs more than they do (500,000 targets,
// whole call: 7.7 ms with this root and the compiler's division, 8.8 with its
// root too, 9.2 with a division that refines the reciprocal once more).
__device__ __forceinline__ double root_mid(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  double g = x * y, h = 0.5 * y;
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const double e = __fma_rn(-g, h, 0.5);
    g = __fma_rn(g, e, g);
    h = __fma_rn(h, e, h);
  }
  return __fma_rn(__fma_rn(-g, g, x), h, g);
}

// The rotation annihilating A(P, Q), applied to A, u and v.
template <int M, int P, int Q>
__device__ __forceinline__ void mls_rotate(double *a, MlsColumn u, MlsColumn v) {
  constexpr int pq = sym_at(P, Q, M), pp = sym_at(P, P, M), qq = sym_at(Q, Q, M);
  const double apq = a[pq];
  if (apq == 0.0) return;
  const double app = a[pp], aqq = a[qq];
  const double g = 100.0 * fabs(apq);
  if (fabs(app) + g == fabs(app) && fabs(aqq) + g == fabs(aqq)) {
    a[pq] = 0.0;  // below the rounding of both diagonal entries
    return;
  }
  const double h = aqq - app;
  double t;
  if (fabs(h) + g == fabs(h)) {
    t = apq / h;
  } else {
    const double theta = 0.5 * h / apq;  // at most 1e18: |h| + 100 |apq| > |h|
    t = 1.0 / (fabs(theta) + root_mid(1.0 + theta * theta));
    if (theta < 0.0) t = -t;
  }
  const double c = 1.0 / root_mid(1.0 + t * t);
  const double s = t * c;
  const double tau = s / (1.0 + c);
  a[pp] = app - t * apq;
  a[qq] = aqq + t * apq;
  a[pq] = 0.0;
#pragma unroll
  for (int r = 0; r < M; ++r) {
    if (r == P || r == Q) continue;
    const int rp = sym_at(r, P, M), rq = sym_at(r, Q, M);
    const double arp = a[rp], arq = a[rq];
    a[rp] = arp - s * (arq + tau * arp);
    a[rq] = arq + s * (arp - tau * arq);
  }
  const double up = u[P], uq = u[Q];
  u[P] = up - s * (uq + tau * up);
  u[Q] = uq + s * (up - tau * uq);
  const double vp = v[P], vq = v[Q];
  v[P] = vp - s * (vq + tau * vp);
  v[Q] = vq + s * (vp - tau * vq);
}

}  // namespace pacman_b200
