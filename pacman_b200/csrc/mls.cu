// Moving least squares transfer of the B200 engine (PACMAN::MLS_interpolate,
// src/mls_interface.cpp; src/mls/interpolator.hpp:49-77).  The reference
// hands the whole computation to ArborX 2.1's
// Interpolation::MovingLeastSquares with its defaults: for each target the K
// nearest sources (K = size of the quadratic basis: 3, 6, 10 in 1D, 2D, 3D),
// radius 1.1 x the farthest neighbour's distance, Wendland C0 weights
// (1 - d / radius)^2, the moment matrix A = sum_j w_j p_j p_j^T of the
// monomials of degree <= 2 of (source - target), and the value
// e_0^T A^+ (sum_j w_j f_j p_j) with A^+ the pseudo-inverse of the symmetric A.
// Here the monomials are those of (source - target) / radius: the same value
// wherever A is invertible, without the radius^4 spread of A's eigenvalues.
//
// Two kernels, one thread per target each, targets in the order of their grid
// cells:
//  * k_mls_search: the K nearest on the uniform source grid (search.cuh), kept
//    sorted by (squared distance, source index) in registers, so ties go to
//    the lowest index and the neighbour set and order are exactly the CPU
//    oracle's.
//  * k_mls_fit: A (packed upper triangle, K(K+1)/2 doubles) in registers and b;
//    a cyclic Jacobi eigen-decomposition A = V L V^T (Rutishauser's rotation
//    formulas) whose rotations are applied to u = V^T e_0 and v = V^T b, so
//    neither V nor A^+ is formed; value = sum over |l_k| > 1e-13 max|l| of
//    u_k v_k / l_k.
// 500,000 refined sources -> 500,000 uniform targets: 1.6 + 6.1 ms, against 32.8
// ms for one kernel in the caller's target order, whose search (always 5^3
// cells or more, a warp's targets scattered over the cloud) kept 12 of 32
// lanes busy at 8 warps per SM.  The search runs at twice the warps now; the
// fit is bound by the latency of each rotation's divisions and square roots
// at 8 warps per SM (255 registers; 168 spill and give the same time).
// This file is compiled without floating-point contraction (-fmad=false):
// each product and sum is rounded on its own, in the same order as the
// oracle's restatement, so the values agree bit for bit.
#include <algorithm>
#include <cfloat>
#include <climits>
#include <cmath>

#include "jacobi.cuh"
#include "plan.hpp"
#include "search.cuh"

namespace pacman_b200 {

namespace {

constexpr int kMlsSweeps = 64;

template <int DIM>
struct Mls {
  static constexpr int K = DIM == 1 ? 3 : (DIM == 2 ? 6 : 10);
  static constexpr int NP = K * (K + 1) / 2;
};

template <int DIM>
__device__ __forceinline__ void mls_basis(const double *x, double *p) {
  p[0] = 1.0;
  if (DIM == 1) {
    p[1] = x[0];
    p[2] = x[0] * x[0];
  } else if (DIM == 2) {
    p[1] = x[0];
    p[2] = x[1];
    p[3] = x[0] * x[0];
    p[4] = x[0] * x[1];
    p[5] = x[1] * x[1];
  } else {
    p[1] = x[0];
    p[2] = x[1];
    p[3] = x[2];
    p[4] = x[0] * x[0];
    p[5] = x[0] * x[1];
    p[6] = x[0] * x[2];
    p[7] = x[1] * x[1];
    p[8] = x[1] * x[2];
    p[9] = x[2] * x[2];
  }
}

// One cyclic sweep over the pairs (P, Q), P < Q, row by row.
template <int M, int P, int Q>
__device__ __forceinline__ void mls_sweep(double *a, MlsColumn u, MlsColumn v) {
  if constexpr (P < M - 1) {
    mls_rotate<M, P, Q>(a, u, v);
    if constexpr (Q + 1 < M)
      mls_sweep<M, P, Q + 1>(a, u, v);
    else if constexpr (P + 2 < M)
      mls_sweep<M, P + 1, P + 2>(a, u, v);
  }
}

// The K nearest sources of every target, ascending by (squared distance,
// source id): ids to nbr[k * M + t], INT_MAX where there are fewer.  Targets in
// cell order, so that a warp's threads scan the same cells.
template <int DIM>
__global__ void __launch_bounds__(128)
    k_mls_search(int64_t t0, int64_t M, GridView g, const double4 *__restrict__ sorted, double h,
                 int *__restrict__ nbr) {
  constexpr int K = Mls<DIM>::K;
  const double4 *tgt = sorted + g.start[g.ncells + 1] + t0;
  for (int64_t t = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; t < M;
       t += int64_t(gridDim.x) * blockDim.x) {
    const double4 y = tgt[t];
    double bd[K];
    int bi[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
      bd[k] = DBL_MAX;
      bi[k] = INT_MAX;
    }
    // A target with a NaN coordinate has no neighbours: its value is zero.
    if (!has_nan(y))
      scan_shells<DIM>(
          g, sorted, h, y,
          [&](const double4 &x) {
            const int id = int(x.w);
            const double d2 = sqdist3(y.x, y.y, y.z, x.x, x.y, x.z);
            if (!(d2 < bd[K - 1] || (d2 == bd[K - 1] && id < bi[K - 1]))) return;
            bd[K - 1] = d2;
            bi[K - 1] = id;
#pragma unroll
            for (int k = K - 1; k > 0; --k) {
              if (bd[k] < bd[k - 1] || (bd[k] == bd[k - 1] && bi[k] < bi[k - 1])) {
                const double td = bd[k];
                bd[k] = bd[k - 1];
                bd[k - 1] = td;
                const int ti = bi[k];
                bi[k] = bi[k - 1];
                bi[k - 1] = ti;
              }
            }
          },
          [&] { return bi[K - 1] == INT_MAX ? INFINITY : bd[K - 1]; });
#pragma unroll
    for (int k = 0; k < K; ++k) nbr[int64_t(k) * M + t] = bi[k];
  }
}

// The fit of every target from its neighbours.  The moment matrix stays in
// registers; u and v, touched at two entries by a rotation, are in shared
// memory.
template <int DIM>
__global__ void __launch_bounds__(128, 2)
    k_mls_fit(int64_t t0, int64_t M, GridView g, const double4 *__restrict__ sorted,
              const int *__restrict__ nbr, const double4 *__restrict__ src,
              const double *__restrict__ vals, int64_t n, double *__restrict__ out) {
  constexpr int K = Mls<DIM>::K;
  constexpr int NP = Mls<DIM>::NP;
  __shared__ double us[K][128], vs[K][128];
  const MlsColumn u{&us[0][threadIdx.x]}, b{&vs[0][threadIdx.x]};
  const double4 *tgt = sorted + g.start[g.ncells + 1] + t0;
  const int kk = n < K ? int(n) : K;
  for (int64_t t = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; t < M;
       t += int64_t(gridDim.x) * blockDim.x) {
    const double4 y = tgt[t];
    // Weights, moment matrix and right-hand side.  With finite coordinates
    // the first kk entries are filled; the id test keeps a NaN coordinate
    // (never a neighbour) from indexing past the sources.
    int bi[K];
    bool use[K];
    double dist[K];
    double rad = 10.0 * DBL_EPSILON;
#pragma unroll
    for (int j = 0; j < K; ++j) {
      bi[j] = nbr[int64_t(j) * M + t];
      use[j] = j < kk && bi[j] != INT_MAX;
      dist[j] = 0.0;
      if (use[j]) {
        const double4 x = src[bi[j]];
        dist[j] = sqrt(sqdist3(y.x, y.y, y.z, x.x, x.y, x.z));
        rad = fmax(rad, dist[j]);
      }
    }
    const double radius = 1.1 * rad;
    const double yc[3] = {y.x, y.y, y.z};
    double a[NP];
#pragma unroll
    for (int i = 0; i < NP; ++i) a[i] = 0.0;
#pragma unroll
    for (int i = 0; i < K; ++i) {
      b[i] = 0.0;
      u[i] = i == 0 ? 1.0 : 0.0;
    }
#pragma unroll
    for (int j = 0; j < K; ++j) {
      if (use[j]) {
        const double4 s4 = src[bi[j]];
        const double sc[3] = {s4.x, s4.y, s4.z};
        double x[3], p[K];
#pragma unroll
        for (int d = 0; d < 3; ++d) x[d] = d < DIM ? (sc[d] - yc[d]) / radius : 0.0;
        mls_basis<DIM>(x, p);
        const double rho = dist[j] / radius;
        const double w = (1.0 - rho) * (1.0 - rho);
        const double wf = w * vals[bi[j]];
#pragma unroll
        for (int r = 0; r < K; ++r) {
          const double wr = w * p[r];
#pragma unroll
          for (int c = r; c < K; ++c) a[sym_at(r, c, K)] = a[sym_at(r, c, K)] + wr * p[c];
          b[r] = b[r] + wf * p[r];
        }
      }
    }
    // e_0^T A^+ b by cyclic Jacobi, at most kMlsSweeps sweeps.
    for (int sw = 0; sw < kMlsSweeps; ++sw) {
      bool off = false;
#pragma unroll
      for (int p = 0; p < K; ++p)
#pragma unroll
        for (int q = p + 1; q < K; ++q) off |= a[sym_at(p, q, K)] != 0.0;
      if (!off) break;
      mls_sweep<K, 0, 1>(a, u, b);
    }
    double lmax = 0.0;
#pragma unroll
    for (int k = 0; k < K; ++k) lmax = fmax(lmax, fabs(a[sym_at(k, k, K)]));
    const double cut = 1e-13 * lmax;
    double val = 0.0;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const double l = a[sym_at(k, k, K)];
      if (fabs(l) > cut) val = val + (u[k] * b[k]) / l;
    }
    out[int(y.w)] = kk > 0 ? val : 0.0;
  }
}

template <int DIM>
void launch_mls(const PointSearch &ps, int64_t m, const double *vals_dev, int64_t n,
                double *out_dev, cudaStream_t st) {
  constexpr int K = Mls<DIM>::K;
  // Neighbour ids of up to 4M targets at a time.
  const int64_t chunk = std::min<int64_t>(m, int64_t(1) << 22);
  DevMem nbr;
  nbr.alloc(sizeof(int) * size_t(K) * size_t(chunk), st);
  const double h = 1.0 / ps.grid.inv_h;
  for (int64_t t0 = 0; t0 < m; t0 += chunk) {
    const int64_t M = std::min(chunk, m - t0);
    const int blocks = int(std::max<int64_t>(1, (M + 127) / 128));
    k_mls_search<DIM><<<blocks, 128, 0, st>>>(t0, M, ps.grid, ps.sorted, h, nbr.as<int>());
    k_mls_fit<DIM><<<blocks, 128, 0, st>>>(t0, M, ps.grid, ps.sorted, nbr.as<int>(),
                                           ps.src4.as<double4>(), vals_dev, n, out_dev);
    note_launch(2);
  }
  PB_CUDA(cudaGetLastError());
}

}  // namespace

void mls_interpolate(int dim, const double *src_dev, int64_t n, const double *vals_dev,
                     const double *tgt_dev, int64_t m, double *out_dev, cudaStream_t st) {
  if (m == 0) return;
  if (n == 0) {  // no source: the zero fill of SetupTransferClass (transfer.hxx:100-110)
    PB_CUDA(cudaMemsetAsync(out_dev, 0, sizeof(double) * size_t(m), st));
    return;
  }
  for (int64_t t0 = 0; t0 < m; t0 += kSearchTargets) {
    const int64_t M = std::min(m - t0, kSearchTargets);
    PointSearch ps;
    // Cells 1.5 times as wide as for one source each: the ten nearest of a
    // uniform cloud then mostly lie in the 3^3 cells around the target.
    build_point_search(ps, dim, src_dev, n, tgt_dev + t0 * dim, M, 1.5, st);
    if (dim == 1) launch_mls<1>(ps, M, vals_dev, n, out_dev + t0, st);
    else if (dim == 2) launch_mls<2>(ps, M, vals_dev, n, out_dev + t0, st);
    else launch_mls<3>(ps, M, vals_dev, n, out_dev + t0, st);
  }
  PB_CUDA(host_sync(st));
}

}  // namespace pacman_b200
