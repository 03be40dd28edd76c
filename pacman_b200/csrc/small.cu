// Register-resident solver for the small patches (n <= 96) of the B200
// RBF-PUM transfer: both precisions of the forward transfer and the adjoint.
//
// Per patch (src/rbf_pum/solver/solver.hpp:180-286): A = phi(|x_i - x_j|),
// the polynomial block (serial_ops.hpp:108-139), alpha = A^{-1}(b - Q beta)
// by unpivoted LU (the elimination order of the reference, here on the
// symmetric positive definite A) and local = E alpha + V beta.
//
// k_small_moments and k_small_fit do the polynomial block of every listed
// patch beforehand: a warp sums one patch's moments, then a thread per patch
// does the condition test and the least squares.
//
// k_small_lu is one block of N / 32 warps per patch with one matrix row per
// thread, in registers.  Pivot p: every thread holds a[i][p]; the column was
// published to shared memory (a[p][j] = a[j][p] by symmetry), so row i needs
// only its own multiplier a[i][p] / a[p][p] and broadcast reads of the
// column.  Column p + 1 is updated and published before the rest of the row,
// so that the barrier's and the reciprocal's latency overlaps the remaining
// multiply-adds, and the right-hand sides ride along.  The pivot loop is
// unrolled by kBlk columns; a finished group of columns (multipliers below
// the diagonal, U on and above it) goes to shared memory and the row shifts
// down by kBlk registers, which keeps the code small and every register index
// static.  U x = y is then solved row-locally with shuffles inside each warp.
//
// What bounds it: latency and issue, not the FP64 pipe.  A pivot is a chain
// of about 300 cycles (column read, reciprocal, multiplier, update, publish,
// barrier) and a row takes 2 N registers, so 8 to 16 warps share an SM; the
// FP64 pipe is 34% busy and an instruction issues in 42% of the cycles (ncu,
// class 48, 4 fields).  Size classes in steps of 8 keep the registers and the
// unused columns few.  500,000 uniform points, Wendland C4, 4 fields (54,500
// patches): all small-patch launches 2.1 ms, against 8.6 ms for a 256-thread
// team per patch on the padded 64 x 64 block with the explicit L^{-1}; 200,000
// points, C6, 1 field, FP64: 0.77 ms against 4.5 ms for the shared-memory LU.
// The class of 65 to 96 sources is three warps at 255 registers, two blocks
// per SM: 44 us for one patch against 142 for the shared-memory LU (a 2D
// transfer between meshes of 3,000 and 4,000 points 0.62 -> 0.49 ms; 48 mixed
// transfers of 1,000 to 30,000 points 13.5 -> 11.9 ms).
// The classes of a list share nothing: each starts in the room that the last
// blocks of the one before leave (programmatic launches).  Gradients of 150,000
// points 3.35 -> 3.17 ms, the 2D transfer 0.46 -> 0.425.
#include <type_traits>

#include "patch.cuh"

namespace pacman_b200 {

namespace {

constexpr int kMomWarps = 4;            // patches per block of k_small_moments
constexpr int kMomLd = kSmallWide + 1;  // column stride: odd, one bank per column

// Moments of the patch's centred monomials (poly.cuh: red layout up to the
// coordinate ranges), a warp per patch and a lane per value: every value is a
// sum over the points of a product of two of the columns 1, q_x, q_y, q_z,
// b_f, in point order.
__global__ void __launch_bounds__(kMomWarps * 32)
    k_small_moments(PatchArgs a, const int *__restrict__ plist, int np, int Fm) {
  __shared__ double tab[kMomWarps][4 + kMaxF][kMomLd];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int e = blockIdx.x * kMomWarps + warp;
  if (e >= np) return;
  const int k = plist[e];
  const int64_t s0 = a.soff[k];
  const int n = int(a.soff[k + 1] - s0);
  const double4 c = a.centers[k];
  double(*col)[kMomLd] = tab[warp];
  for (int i = lane; i < n; i += 32) {
    const int id = a.sidx[s0 + i];
    const double4 p = a.src[id];
    col[0][i] = 1.0;
    col[1][i] = p.x - c.x;
    col[2][i] = p.y - c.y;
    col[3][i] = p.z - c.z;
    for (int f = 0; f < Fm; ++f) col[4 + f][i] = a.vals[int64_t(id) * a.F + f];
  }
  __syncwarp();
  const int nred = 10 + 4 * Fm;
  for (int id = lane; id < nred; id += 32) {
    int u = id, v = 0;
    if (id >= 10) {
      u = (id - 10) & 3;
      v = 4 + ((id - 10) >> 2);
    } else if (id >= 4) {
      u = id < 7 ? 1 : (id < 9 ? 2 : 3);
      v = id < 7 ? id - 3 : (id < 9 ? id - 5 : 3);
    }
    const double *cu = col[u], *cv = col[v];
    double s = 0.0;
#pragma unroll 4
    for (int i = 0; i < n; ++i) s = __fma_rn(cu[i], cv[i], s);
    a.pred[int64_t(e) * kRedVals + id] = s;
  }
}

// Polynomial block of a patch per thread: the condition test and the least
// squares are serial chains of a few thousand dependent FP64 operations, so a
// warp works on 32 patches side by side.  adj: beta receives the 4 x 4 factor
// R, act its terms S and their count.
__global__ void __launch_bounds__(32)
    k_small_fit(PatchArgs a, const int *__restrict__ plist, int np, int adj) {
  const int e = blockIdx.x * 32 + threadIdx.x;
  if (e >= np) return;
  const int k = plist[e];
  const double4 c = a.centers[k];
  const double shift[3] = {c.x, c.y, c.z};
  double *beta = a.pbeta + int64_t(e) * 4 * kMaxF;
  int *act = a.pact + int64_t(e) * 8;
  const int Fm = adj ? 0 : a.F;
  double red[kRedVals];
  for (int v = 0; v < 10 + 4 * Fm; ++v) red[v] = a.pred[int64_t(e) * kRedVals + v];
  // Coordinate ranges: only a failed condition test reads them.
  auto ranges = [&](double *mn, double *mx) {
    for (int d = 0; d < 3; ++d) {
      mn[d] = INFINITY;
      mx[d] = -INFINITY;
    }
    for (int64_t i = a.soff[k]; i < a.soff[k + 1]; ++i) {
      const double4 p = a.src[a.sidx[i]];
      mn[0] = fmin(mn[0], p.x);
      mn[1] = fmin(mn[1], p.y);
      mn[2] = fmin(mn[2], p.z);
      mx[0] = fmax(mx[0], p.x);
      mx[1] = fmax(mx[1], p.y);
      mx[2] = fmax(mx[2], p.z);
    }
  };
  int S[4] = {0, 0, 0, 0}, pv;
  double R[4][4];
  const int dropped = poly_axes(red, a.dim, shift, ranges, S, pv, R);
  if (adj) {
    for (int i = 0; i < 4; ++i) {
      act[i] = S[i];
      for (int j = 0; j < 4; ++j) beta[4 * i + j] = R[i][j];
    }
    act[4] = pv;
  } else {
    poly_fit(red, a.F, shift, S, pv, R, beta, act);
    if (a.alpha_out != nullptr) {
      double *bo = a.beta_out + int64_t(k) * 4 * kMaxF;
      for (int v = 0; v < 4 * kMaxF; ++v) bo[v] = v < 4 * a.F ? beta[v] : 0.0;
      for (int d = 0; d < 3; ++d) a.act_out[int64_t(k) * 3 + d] = act[d];
    }
  }
  a.status[k] = dropped ? kStatusDropped : 0;
}

template <int N, int KF, bool ADJ>
struct SmallCfg {
  static constexpr int kT = (N + 31) / 32 * 32;  // threads
  static constexpr int kLd = N + 2;              // row stride: 16-byte rows, spread over the banks
  static constexpr int kBlk = 16;                // pivots per unrolled group
  static constexpr size_t kSmem = size_t(N) * kLd * sizeof(double);
  // Resident blocks per SM the registers are shared out for.  A row takes 2 N
  // registers; four, three or two warps per scheduler leave 128, 168 or 255.
  static constexpr int kMinBlocks = N <= 32   ? 16
                                    : N <= 40 ? 8
                                    : N <= 48 ? 5
                                    : N <= 56 ? (KF == 1 || !ADJ ? 5 : 4)
                                    : N <= 64 ? 4
                                              : 2;
};

template <int N, int KF, bool ADJ>
__global__ void __launch_bounds__(SmallCfg<N, KF, ADJ>::kT, SmallCfg<N, KF, ADJ>::kMinBlocks)
    k_small_lu(PatchArgs a, const int *__restrict__ plist) {
  // A class launched behind this one may start once all blocks here have.
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  using C = SmallCfg<N, KF, ADJ>;
  constexpr int T = C::kT, LD = C::kLd, BLK = C::kBlk;
  extern __shared__ __align__(16) double As[];  // N x LD
  __shared__ __align__(16) double col[2][T + BLK];
  __shared__ double xs[T], ys[T], zs[T];
  __shared__ double rp[2][KF];
  __shared__ double al[KF][T];
  __shared__ int flag_s;
  const int e = blockIdx.x;
  const int i = threadIdx.x, lane = i & 31, warp = i >> 5;
  const int k = plist[e];
  const int64_t s0 = a.soff[k];
  const int n = int(a.soff[k + 1] - s0);
  const int64_t t0 = a.toff[k];
  const int m = int(a.toff[k + 1] - t0);
  const int F = a.F;
  const double *beta = a.pbeta + int64_t(e) * 4 * kMaxF;
  const int *act = a.pact + int64_t(e) * 8;
  const bool load = a.fac_mode == 2;
  if (i == 0) flag_s = 0;

  // Gather the patch (TeamFillB, team_ops.hpp:113-121) and form the residual
  // b - Q beta (serial_ops.hpp:149-185).
  double r[KF];
#pragma unroll
  for (int f = 0; f < KF; ++f) r[f] = 0.0;
  double4 x = make_double4(0.0, 0.0, 0.0, 0.0);
  if (i < n) {
    const int id = a.sidx[s0 + i];
    x = a.src[id];
    if (!ADJ) {
      const double pc[3] = {x.x, x.y, x.z};
#pragma unroll
      for (int f = 0; f < KF; ++f)
        if (f < F) {
          double t = beta[4 * f];
#pragma unroll
          for (int j = 0; j < 3; ++j) {
            const int ax = act[j];
            if (ax >= 0) t = __fma_rn(ax == 0 ? pc[0] : (ax == 1 ? pc[1] : pc[2]), beta[4 * f + 1 + j], t);
          }
          r[f] = a.vals[int64_t(id) * F + f] - t;
        }
    }
  }
  xs[i] = x.x;
  ys[i] = x.y;
  zs[i] = x.z;
  __syncthreads();

  // Adjoint: thread i sums value vq = 4 field + monomial over every kParts-th
  // point, from part i / (4 KF).
  constexpr int kParts = T / (4 * KF);
  __shared__ double vpart[ADJ ? T : 1];
  const int vq = i % (4 * KF), vf = vq >> 2, vax = vq & 3;
  if (ADJ) {
    // Right-hand sides E^T h, E_ij = phi(|y_i - x_j|), and the parts of V'^T h:
    // T targets at a time are staged in As, a target per thread (read one after
    // another from memory by all, they cost a third of the block's time: all
    // adjoint launches for 150,000 uniform points and 4 fields 1.09 -> 0.75 ms).
    static_assert((3 + KF) * T <= N * LD, "staged targets");
    const double4 c = a.centers[k];
    const double cc = vax == 1 ? c.x : (vax == 2 ? c.y : c.z);
    double v = 0.0;
    with_basis(a.basis, [&](auto B) {
      for (int tb = 0; tb < m; tb += T) {
        const int cnt = m - tb < T ? m - tb : T;
        if (i < cnt) {
          const double4 y = a.tgt[a.tidx[t0 + tb + i]];
          As[i] = y.x;
          As[T + i] = y.y;
          As[2 * T + i] = y.z;
#pragma unroll
          for (int f = 0; f < KF; ++f)
            As[(3 + f) * T + i] = f < F ? a.h[(t0 + tb + i) * F + f] : 0.0;
        }
        __syncthreads();
        for (int t = 0; t < cnt; ++t) {
          const double ph = phi_at<B>(
              sqdist3(As[t], As[T + t], As[2 * T + t], x.x, x.y, x.z), a.rinv);
#pragma unroll
          for (int f = 0; f < KF; ++f) r[f] = __fma_rn(ph, As[(3 + f) * T + t], r[f]);
        }
        const double *yc = As + (vax > 0 ? vax - 1 : 0) * T;
        for (int t = i / (4 * KF); t < cnt; t += kParts)
          v += (vax == 0 ? 1.0 : yc[t] - cc) * As[(3 + vf) * T + t];
        __syncthreads();
      }
    });
    vpart[i] = v;
    if (i >= n) {
#pragma unroll
      for (int f = 0; f < KF; ++f) r[f] = 0.0;
    }
  }

  bool bad = false;
  if (!load) {
    // Assembly (TeamFillA, team_ops.hpp:35-52): thread i evaluates the pairs
    // (i, i + d mod n), d <= n / 2, which covers every pair of the symmetric
    // matrix with equal work per thread.
    if (i < n) {
      with_basis(a.basis, [&](auto B) {
        int j = i;
        for (int d = 0; d <= n / 2; ++d) {
          const double v = phi_at<B>(sqdist3(x.x, x.y, x.z, xs[j], ys[j], zs[j]), a.rinv);
          As[i * LD + j] = v;
          As[j * LD + i] = v;
          if (++j == n) j = 0;
        }
      });
    }
    __syncthreads();
    double row[N];
#pragma unroll
    for (int j = 0; j < N; j += 2) {
      double2 v = make_double2(0.0, 0.0);
      if (i < n && j < n) v = *reinterpret_cast<const double2 *>(&As[i * LD + j]);
      row[j] = v.x;
      row[j + 1] = j + 1 < n ? v.y : 0.0;
    }
    col[0][i] = row[0];
    if (i == 0) {
#pragma unroll
      for (int f = 0; f < KF; ++f) rp[0][f] = r[f];
    }
#pragma unroll 1
    for (int pb = 0; pb < n; pb += BLK) {
#pragma unroll
      for (int q = 0; q < BLK; ++q) {
        const int p = pb + q;
        if (p < n) {
          __syncthreads();
          const double *cp = &col[q & 1][pb];  // this column from row pb on
          const double d = cp[q];
          bad |= !(d > 0.0);
          double mi = quot(row[q], d, recip(d));
          if (i <= p) mi = 0.0;
          else row[q] = mi;
          if (q + 1 < N) {
            row[q + 1] = __fma_rn(-mi, cp[q + 1], row[q + 1]);
            col[(q + 1) & 1][i] = row[q + 1];
          }
#pragma unroll
          for (int f = 0; f < KF; ++f) r[f] = __fma_rn(-mi, rp[q & 1][f], r[f]);
          if (i == p + 1) {
#pragma unroll
            for (int f = 0; f < KF; ++f) rp[(q + 1) & 1][f] = r[f];
          }
          // The rest of the row, in groups of eight columns up to n.
#pragma unroll
          for (int g = 0; g < N / 8; ++g) {
            if (8 * g + 7 >= q + 2 && pb + 8 * g < n) {
#pragma unroll
              for (int j = 8 * g; j < 8 * g + 8; ++j)
                if (j >= q + 2) row[j] = __fma_rn(-mi, cp[j], row[j]);
            }
          }
        }
      }
      if (i < N) {
#pragma unroll
        for (int q = 0; q < BLK; q += 2)
          if (N % BLK == 0 || pb + q < N)
            *reinterpret_cast<double2 *>(&As[i * LD + pb + q]) = make_double2(row[q], row[q + 1]);
      }
      if constexpr (N > BLK) {
#pragma unroll
        for (int j = 0; j + BLK < N; ++j) row[j] = row[j + BLK];
      }
    }
    __syncthreads();
    if (a.fac_mode == 1) {
      double *facp = a.fac + size_t(e) * N * N;
      for (int v = i; v < N * N / 2; v += T) {
        const int rr = v / (N / 2), cc = 2 * (v % (N / 2));
        if (rr < n && cc < n)
          *reinterpret_cast<double2 *>(facp + rr * N + cc) =
              *reinterpret_cast<const double2 *>(&As[rr * LD + cc]);
      }
    }
  } else {
    // Kept factors of an earlier execute; the forward substitution, which
    // the elimination does on the way, is done from them.
    const double *facp = a.fac + size_t(e) * N * N;
    for (int v = i; v < N * N / 2; v += T) {
      const int rr = v / (N / 2), cc = 2 * (v % (N / 2));
      if (rr < n && cc < n)
        *reinterpret_cast<double2 *>(&As[rr * LD + cc]) =
            *reinterpret_cast<const double2 *>(facp + rr * N + cc);
    }
    __syncthreads();
    // L y = r: each warp its own rows from the first, what later warps need of
    // them through shared memory.
    const double *ar = As + (i < n ? i : 0) * LD;
    for (int w = 0; w < T / 32; ++w) {
      const int j0 = 32 * w, j1 = n < j0 + 32 ? n : j0 + 32;
      if (warp == w) {
        for (int p = j0; p < j1; ++p) {
          const double l = (i > p && i < n) ? ar[p] : 0.0;
#pragma unroll
          for (int f = 0; f < KF; ++f)
            r[f] = __fma_rn(-l, __shfl_sync(0xffffffffu, r[f], p - j0), r[f]);
        }
#pragma unroll
        for (int f = 0; f < KF; ++f) al[f][i] = r[f];
      }
      __syncthreads();
      if (warp > w && i < n) {
        for (int p = j0; p < j1; ++p) {
          const double l = ar[p];
#pragma unroll
          for (int f = 0; f < KF; ++f) r[f] = __fma_rn(-l, al[f][p], r[f]);
        }
      }
    }
  }

  // U alpha = y: each warp its own rows from the last, what earlier warps need
  // of them through shared memory.
  {
    const double *ar = As + (i < n ? i : 0) * LD;
    const double dg = i < n ? ar[i] : 1.0;
    const double inv = recip(dg);
    for (int w = T / 32 - 1; w >= 0; --w) {
      const int j0 = 32 * w, j1 = n < j0 + 32 ? n : j0 + 32;
      if (warp == w) {
        for (int j = j1 - 1; j >= j0; --j) {
          const double u = (i < j) ? ar[j] : 0.0;
#pragma unroll
          for (int f = 0; f < KF; ++f) {
            const double xj = __shfl_sync(0xffffffffu, quot(r[f], dg, inv), j - j0);
            if (i == j) r[f] = xj;
            else r[f] = __fma_rn(-u, xj, r[f]);
          }
        }
#pragma unroll
        for (int f = 0; f < KF; ++f) al[f][i] = r[f];
      }
      __syncthreads();
      if (warp < w) {
        for (int j = j0; j < j1; ++j) {
          const double u = ar[j];
#pragma unroll
          for (int f = 0; f < KF; ++f) r[f] = __fma_rn(-u, al[f][j], r[f]);
        }
      }
    }
  }

  bool nonfinite = false;
  if (ADJ) {
    // g = z - Q' G'^{-1} (Q'^T z - V'^T h), centred monomials q' = [1, x - c].
    __shared__ double corr[4 * KF];
    __shared__ double upart[T];
    const double4 c = a.centers[k];
    {
      const double cc = vax == 1 ? c.x : (vax == 2 ? c.y : c.z);
      const double *xc = vax == 1 ? xs : (vax == 2 ? ys : zs);
      double u = 0.0;
      for (int j = i / (4 * KF); j < n; j += kParts)
        u += (vax == 0 ? 1.0 : xc[j] - cc) * al[vf][j];
      upart[i] = u;
    }
    __syncthreads();
    if (i < 4 * KF) {
      double u = 0.0, v = 0.0;
      for (int q = i; q < kParts * 4 * KF; q += 4 * KF) {
        u += upart[q];
        v += vpart[q];
      }
      corr[i] = u - v;
    }
    __syncthreads();
    if (i < F) {
      double R[4][4], rhs[4] = {0, 0, 0, 0}, sol[4] = {0, 0, 0, 0};
      const int pv = act[4];
      for (int q = 0; q < 4; ++q)
        for (int j = 0; j < 4; ++j) R[q][j] = beta[4 * q + j];
      for (int q = 0; q < pv; ++q) rhs[q] = corr[4 * i + act[q]];
      gram_solve(R, pv, rhs, sol);
      for (int q = 0; q < 4; ++q) corr[4 * i + q] = 0.0;
      for (int q = 0; q < pv; ++q) corr[4 * i + act[q]] = sol[q];
    }
    __syncthreads();
    if (i < n) {
      const double q[3] = {x.x - c.x, x.y - c.y, x.z - c.z};
#pragma unroll
      for (int f = 0; f < KF; ++f)
        if (f < F) {
          double g = al[f][i];
          g -= corr[4 * f];
#pragma unroll
          for (int d = 0; d < 3; ++d) g -= q[d] * corr[4 * f + 1 + d];
          nonfinite |= !isfinite(g);
          a.g_out[(s0 + i) * F + f] = g;
        }
    }
  } else {
    if (a.alpha_out != nullptr && i < n) {
#pragma unroll
      for (int f = 0; f < KF; ++f)
        if (f < F) a.alpha_out[(s0 + i) * F + f] = al[f][i];
    }
    // local = E alpha + V beta (solver.hpp:270-273), a thread per target, two
    // sources at a time with a sum each.
    with_basis(a.basis, [&](auto B) {
      for (int t = i; t < m; t += T) {
        const double4 y = a.tgt[a.tidx[t0 + t]];
        double acc[KF], odd[KF];
#pragma unroll
        for (int f = 0; f < KF; ++f) acc[f] = odd[f] = 0.0;
        auto at = [&](int j, double *sum) {
          const double ph = phi_at<B>(sqdist3(y.x, y.y, y.z, xs[j], ys[j], zs[j]), a.rinv);
#pragma unroll
          for (int f = 0; f < KF; ++f) sum[f] = __fma_rn(ph, al[f][j], sum[f]);
        };
        int j = 0;
        for (; j + 1 < n; j += 2) {
          at(j, acc);
          at(j + 1, odd);
        }
        if (j < n) at(j, acc);
#pragma unroll
        for (int f = 0; f < KF; ++f) acc[f] += odd[f];
        const double yc[3] = {y.x, y.y, y.z};
#pragma unroll
        for (int f = 0; f < KF; ++f)
          if (f < F) {
            double vb = beta[4 * f];
#pragma unroll
            for (int j = 0; j < 3; ++j) {
              const int ax = act[j];
              if (ax >= 0) vb = __fma_rn(ax == 0 ? yc[0] : (ax == 1 ? yc[1] : yc[2]), beta[4 * f + 1 + j], vb);
            }
            const double out = acc[f] + vb;
            nonfinite |= !isfinite(out);
            a.local[(t0 + t) * F + f] = out;
          }
      }
    });
  }
  if (nonfinite) atomicOr(&flag_s, kStatusNonFinite);
  if (bad && i == 0) atomicOr(&flag_s, kStatusBreakdown);
  __syncthreads();
  if (i == 0 && flag_s) a.status[k] |= flag_s;
  // What follows this launch waits for it alone, so it ends no sooner than the
  // class before it (block 0 waits; at once where nothing runs ahead).
  if (e == 0) asm volatile("griddepcontrol.wait;" ::: "memory");
}

template <int N, bool ADJ>
void launch_n(const PatchArgs &a, const int *plist, int np, bool behind, cudaStream_t st) {
  using C = SmallCfg<N, 1, ADJ>;
  auto go = [&](auto kernel) {
    if (C::kSmem > 40 * 1024)
      PB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   int(C::kSmem)));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(np);
    cfg.blockDim = dim3(C::kT);
    cfg.dynamicSmemBytes = C::kSmem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = behind ? 1 : 0;
    PB_CUDA(cudaLaunchKernelEx(&cfg, kernel, a, plist));
  };
  if (a.F == 1) go(k_small_lu<N, 1, ADJ>);
  else if (a.F <= 4) go(k_small_lu<N, 4, ADJ>);
  else go(k_small_lu<N, 8, ADJ>);
  note_launch();
  PB_CUDA(cudaGetLastError());
}

}  // namespace

int small_class(int n) { return n <= 32 ? 32 : (n <= 64 ? (n + 7) / 8 * 8 : kSmallWide); }

void launch_small_poly(const PatchArgs &a, const int *plist, int np, bool adj, cudaStream_t st) {
  if (np == 0) return;
  k_small_moments<<<(np + kMomWarps - 1) / kMomWarps, kMomWarps * 32, 0, st>>>(
      a, plist, np, adj ? 0 : a.F);
  k_small_fit<<<(np + 31) / 32, 32, 0, st>>>(a, plist, np, adj ? 1 : 0);
  note_launch(2);
  PB_CUDA(cudaGetLastError());
}

void launch_small_lu(const PatchArgs &a, const int *plist, int np, int N, bool adj, bool behind,
                     cudaStream_t st) {
  if (np == 0) return;
  auto go = [&](auto A) {
    constexpr bool kAdjoint = decltype(A)::value;
    switch (N) {
    case 32: launch_n<32, kAdjoint>(a, plist, np, behind, st); break;
    case 40: launch_n<40, kAdjoint>(a, plist, np, behind, st); break;
    case 48: launch_n<48, kAdjoint>(a, plist, np, behind, st); break;
    case 56: launch_n<56, kAdjoint>(a, plist, np, behind, st); break;
    case 64: launch_n<64, kAdjoint>(a, plist, np, behind, st); break;
    default: launch_n<kSmallWide, kAdjoint>(a, plist, np, behind, st); break;
    }
  };
  if (adj) go(std::true_type{});
  else go(std::false_type{});
}

}  // namespace pacman_b200
