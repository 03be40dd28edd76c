// Left-looking blocked Cholesky for the large patches of the B200 RBF-PUM
// transfer (both precisions and the adjoint).
//
// The reference factors each patch matrix with an unpivoted LU in one GPU
// thread (src/rbf_pum/solver/solver.hpp:422-490, KokkosBatched
// SerialLU<Unblocked>).  A is symmetric positive definite, so here it is
// factored as L L^T in 64 x 64 tiles, all large patches in lockstep, one tile
// column j per step:
//   C[i, j] = A[i, j] - sum_{p<j} L[i, p] L[j, p]^T for every i > j, then
//   L[i, j] U_j = C solved against the diagonal tile's factor (U_j = L_jj^T,
//   made one step earlier) and the forward substitution r_i -= L[i, j] y_j.
// The column update runs on the int8 tensor cores as split-integer products
// (k_col_step_ws, with k_diag_next factoring the next diagonal tile after
// each step) or, for the columns before PACMAN_B200_INT8_FROM and without
// int8 slices, on the FP64 tensor cores (k_col_step, whose CTA of row tile
// j + 1 also forms and factors the next diagonal tile).  k_diag_chol does
// the diagonal tile of step 0.  Afterwards k_chol_back solves L^T alpha = y
// (with the kept tile inverses X_s = L_ss^-1) and k_chol_eval evaluates
// local = E alpha + V beta (solver.hpp:270-273).
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "blocked.cuh"

namespace pacman_b200 {

constexpr int kKC = 32;                 // K chunk of the column update (doubles)
constexpr int kKLD = kKC + 4;           // shared row stride of a chunk: conflict-free fragments
constexpr int kStages = 2;              // cp.async pipeline depth (2 CTAs per SM)
constexpr int kColRows = 2 * TB;        // rows of one column-update CTA (two tiles)
constexpr int kColThreads = 256;
constexpr int kColStage = (kColRows + TB) * kKLD;  // doubles per pipeline stage
constexpr size_t kColSmem = size_t(kStages) * kColStage * sizeof(double);
constexpr size_t kDiagSmem = (size_t(2) * TB * LDS + 6 * TB) * sizeof(double);

// acc += A B^T over one K chunk: A rows wr.., B rows wc.. (both K-contiguous).
__device__ __forceinline__ void mma_chunk_nt(const double *__restrict__ sA,
                                             const double *__restrict__ sB,
                                             double (&acc)[4][4][2], int wr, int wc, int lane) {
  const int g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int k0 = 0; k0 < kKC; k0 += 4) {
    double a[4], b[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) a[i] = sA[(wr + 8 * i + g) * kKLD + k0 + t];
#pragma unroll
    for (int jj = 0; jj < 4; ++jj) b[jj] = sB[(wc + 8 * jj + g) * kKLD + k0 + t];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int jj = 0; jj < 4; ++jj) dmma(acc[i][jj][0], acc[i][jj][1], a[i], b[jj]);
  }
}

__device__ __forceinline__ void acc_neg(double (&acc)[4][4][2]) {
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int jj = 0; jj < 4; ++jj) acc[i][jj][0] = -acc[i][jj][0], acc[i][jj][1] = -acc[i][jj][1];
}

// Rows [ti TB, ti TB + nrows) x columns [tj TB, tj TB + TB) of a slot's
// Wendland matrix A (TeamFillA, team_ops.hpp:35-52; identity past n) into sT
// (row stride LDS), by the threads t, t + nt, ...: the step kernels evaluate
// their tiles instead of reading an assembled copy.  The row and column points
// are staged in pts (3 (nrows + TB) doubles) first; sync() must be a barrier
// over the nt threads.
template <class Sync>
__device__ __forceinline__ void gen_tile(const BigArgs &a, const BigSlot &sl, int ti, int tj,
                                         int nrows, double *sT, double *pts, int t, int nt,
                                         Sync sync, bool load_cols = true) {
  const int64_t s0 = a.soff[sl.k];
  double *rx = pts, *ry = rx + nrows, *rz = ry + nrows;
  double *cx = rz + nrows, *cy = cx + TB, *cz = cy + TB;
  // With load_cols false the column points are still in pts from a previous
  // tile of the same slot and column tile.
  for (int e = t; e < (load_cols ? nrows + TB : nrows); e += nt) {
    const int gi = e < nrows ? ti * TB + e : tj * TB + (e - nrows);
    double4 p = make_double4(0.0, 0.0, 0.0, 0.0);
    if (gi < sl.n) p = a.src[a.sidx[s0 + gi]];
    if (e < nrows) {
      rx[e] = p.x;
      ry[e] = p.y;
      rz[e] = p.z;
    } else {
      cx[e - nrows] = p.x;
      cy[e - nrows] = p.y;
      cz[e - nrows] = p.z;
    }
  }
  sync();
  for (int e = t; e < nrows * TB; e += nt) {
    const int r = e >> 6, c = e & 63;
    const int gi = ti * TB + r, gj = tj * TB + c;
    double v;
    if (gi < sl.n && gj < sl.n)
      v = wendland<double>(a.basis, __dsqrt_rn(sqdist3(rx[r], ry[r], rz[r], cx[c], cy[c], cz[c])),
                           a.rinv);
    else
      v = (gi == gj) ? 1.0 : 0.0;
    sT[r * LDS + c] = v;
  }
}

__device__ __forceinline__ void sync_all() { __syncthreads(); }

// Cholesky of the 16 x 16 block D[kb.., kb..] (lower part, row stride ld,
// overwritten by L) by one warp in registers: lane i + 16 h holds columns
// 8 h .. 8 h + 7 of row kb + i; column c's entries reach the other lanes by
// shuffles.  A column-by-column right-looking Cholesky of the block: 1 / L_cc
// = rsqrt(d_cc) (one operation on the chain of pivots instead of a square
// root and a reciprocal), L_cc = sqrt(d_cc) and L_ic = d_ic / L_cc from it,
// each with one residual correction (plain products with 1 / L_cc gave local
// values 20-50% further from the 64-bit reference on the shell patches), d_ij
// -= L_ic L_jc; dis[kb + c] = 1 / L_cc.  Written without branches (selects; lane
// c keeps 1 / L_cc and stores it after the loop) so that the sixteen unrolled
// steps form one block the compiler can schedule across: FP64 operations
// and shuffles each take ~25 cycles to complete on this GPU, and a step is a
// chain of five of them.  Returns true on a pivot that is not > 0.
__device__ __noinline__ bool warp_chol16(double *D, int ld, int kb, double *dis, int lane) {
  const int i = lane & 15, h = lane >> 4;
  double a[8];
#pragma unroll
  for (int t = 0; t < 8; ++t) a[t] = 8 * h + t <= i ? D[(kb + i) * ld + kb + 8 * h + t] : 0.0;
  double myrs = 0.0;
  bool ok = true;
#pragma unroll
  for (int c = 0; c < 16; ++c) {
    const int hc = c >> 3, tc = c & 7;
    const double piv = __shfl_sync(0xffffffffu, a[tc], c + 16 * hc);
    ok = ok && piv > 0.0;
    const double rs = rsqrt(piv);
    const double g = piv * rs;
    const double lcc = __fma_rn(__fma_rn(-g, g, piv), 0.5 * rs, g);
    const double sc = quot(a[tc], lcc, rs);
    const bool mine = h == hc;
    a[tc] = mine ? (i == c ? lcc : (i > c ? sc : a[tc])) : a[tc];
    myrs = lane == c ? rs : myrs;
    const double oth = __shfl_xor_sync(0xffffffffu, a[tc], 16);
    const double lic = mine ? a[tc] : oth;  // L[i][c]
#pragma unroll
    for (int jj = c + 1; jj < 16; ++jj) {
      const double ljc = __shfl_sync(0xffffffffu, a[tc], jj + 16 * hc);  // L[jj][c]
      const bool upd = h == (jj >> 3) && i >= jj;
      const double nv = __fma_rn(-lic, ljc, a[jj & 7]);
      a[jj & 7] = upd ? nv : a[jj & 7];
    }
  }
  if (lane < 16) dis[kb + lane] = myrs;
#pragma unroll
  for (int t = 0; t < 8; ++t)
    if (8 * h + t <= i) D[(kb + i) * ld + kb + 8 * h + t] = a[t];
  __syncwarp();
  return !ok;
}

// T = L_bb^-1 of the 16 x 16 lower-triangular block at D[kb..][kb..] (row
// stride ld) by one warp in registers, lane j (and j + 16) computing column j
// of T down the column (T_jj = 1 / L_jj from dis, T_ij = -(sum_{j<=k<i} L_ik
// T_kj) / L_ii), unrolled and without branches; stored transposed:
// ui[j kUiLd + i] = T_ij, i.e. ui holds (L_bb^T)^-1 = U_bb^-1.
__device__ __noinline__ void warp_trinv16(const double *D, int ld, int kb, const double *dis,
                                          double *ui, int lane) {
  const int j = lane & 15;
  double t[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    double s = 0.0;
#pragma unroll
    for (int k = 0; k < i; ++k) {
      const double v = __fma_rn(D[(kb + i) * ld + kb + k], t[k], s);
      s = k >= j ? v : s;
    }
    const double di = dis[kb + i];
    t[i] = i < j ? 0.0 : (i == j ? di : -s * di);
  }
  if (lane < 16) {
#pragma unroll
    for (int i = 0; i < 16; ++i) ui[j * kUiLd + i] = t[i];
  }
  __syncwarp();
}

// The diagonal tile of a step, 256 threads (8 warps): the Cholesky factor
// L_c of the 64 x 64 tile D (lower part, in shared memory at g with row stride
// ld, overwritten), X = L_c^{-1} (to gi, row stride TB), y = X r for the first
// F columns of the residual tile (rg, row stride rld, overwritten) and, with
// gu, U = L_c^T (row stride uld; zeros below its diagonal) for the triangular
// solves of the tiles below.  Blocked right-looking Cholesky in 16 x 16
// blocks: warp 0 factors the diagonal block (16 column steps synchronised
// within the warp), the eight warps solve the panel below it by substitution
// and update the trailing blocks on the FP64 tensor cores, three barriers per
// block.  X comes from the row solves X^T U = I: warp_rows_trsm8_tc, or with ui
// (scratch for U's diagonal blocks' inverses) warp_rows_solve8.  Us (TB x LDS) is shared scratch for U,
// dis (TB) for 1 / diag(L_c), ys (TB x kMaxF) for r.  Returns true on a
// non-positive pivot (status 4 for the caller).
template <class Sync, bool kBlockInv>
__device__ bool diag_tile_t(const double *g_in, int ld, double *rg, int rld, int F, double *gi,
                            double *Us, double *dis, double (*ys)[kMaxF], int tid, Sync sync,
                            double *gu = nullptr, int uld = 0, double *ui = nullptr,
                            bool ys_loaded = false) {
  double *D = const_cast<double *>(g_in);
  const int lane = tid & 31, warp = tid >> 5;
  const int gq = lane >> 2, tq = lane & 3;
  const int col16 = lane & 15, half = lane & 16, rsel = lane >> 4;
  bool bad = false;
  if (!ys_loaded)
    for (int e = tid; e < TB * kMaxF; e += 256) {
      const int r = e / kMaxF, f = e % kMaxF;
      ys[r][f] = f < F ? __ldcg(rg + int64_t(r) * rld + f) : 0.0;
    }
  // (a) the first diagonal block, warp 0 (warp_chol16).
  if (warp == 0) bad |= warp_chol16(D, ld, 0, dis, lane);
  sync();
  for (int kb = 0; kb + 16 < TB; kb += 16) {
    // (b) the panel below: rows kb + 16 .. 63 solve x L_kk^T = d.
    const int r0 = kb + 16 + 8 * warp;
    if (r0 < TB) {
      double acc[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) acc[q] = D[(r0 + rsel + 2 * q) * ld + kb + col16];
#pragma unroll 4
      for (int c = 0; c < 16; ++c) {
        const double d = dis[kb + c], lcc = D[(kb + c) * ld + kb + c];
        const double l = D[(kb + col16) * ld + kb + c];  // L_kk[col16][c], used for col16 > c
        const bool own = col16 == c, below = col16 > c;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const double x = quot(__shfl_sync(0xffffffffu, acc[q], half | c), lcc, d);
          acc[q] = own ? x : (below ? __fma_rn(-x, l, acc[q]) : acc[q]);
        }
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) D[(r0 + rsel + 2 * q) * ld + kb + col16] = acc[q];
    }
    sync();
    // (c) trailing blocks: D[i, j] -= P_i P_j^T (P: the panel columns), 8 x 8
    // output tiles (ti, tj) with kb + 16 <= 8 tj <= 8 ti.  Warp 0 updates
    // the next diagonal block's three tiles first and factors that block
    // (look-ahead) while warps 1..7 update the rest: the chain of diagonal
    // blocks does not wait for the whole trailing update.
    const int base = (kb + 16) / 8, nt = 8 - base;
    auto tile = [&](int ti, int tj) {
      double c0 = D[(8 * ti + gq) * ld + 8 * tj + 2 * tq];
      double c1 = D[(8 * ti + gq) * ld + 8 * tj + 2 * tq + 1];
#pragma unroll
      for (int k0 = 0; k0 < 16; k0 += 4) {
        const double av = -D[(8 * ti + gq) * ld + kb + k0 + tq];
        const double bv = D[(8 * tj + gq) * ld + kb + k0 + tq];
        dmma(c0, c1, av, bv);
      }
      D[(8 * ti + gq) * ld + 8 * tj + 2 * tq] = c0;
      D[(8 * ti + gq) * ld + 8 * tj + 2 * tq + 1] = c1;
    };
    if (warp == 0) {
      tile(base, base);
      tile(base + 1, base);
      tile(base + 1, base + 1);
      __syncwarp();
      bad |= warp_chol16(D, ld, kb + 16, dis, lane);
    } else {
      for (int u = warp - 1; u < nt * nt; u += 7) {
        const int ti = base + u / nt, tj = base + u % nt;
        if (tj > ti || (ti < base + 2 && tj < base + 2)) continue;
        tile(ti, tj);
      }
    }
    sync();
  }
  // U = L_c^T with zeros below its diagonal; 1 / diag for the row solves.
  for (int e = tid; e < TB * TB; e += 256) {
    const int p = e >> 6, i = e & 63;
    const double u = i >= p ? D[i * ld + p] : 0.0;
    Us[p * LDS + i] = u;
    if (gu) gu[int64_t(p) * uld + i] = u;
  }
  // With ui: the inverses of U's four 16 x 16 diagonal blocks, one warp each,
  // for the block-inverse row solves of X below.
  if (kBlockInv && warp < 4) warp_trinv16(D, ld, 16 * warp, dis, ui + 16 * warp * kUiLd, lane);
  sync();
  // X^T from X^T U = I: rows of the identity solved in place of D.
  for (int e = tid; e < TB * TB; e += 256) D[(e >> 6) * ld + (e & 63)] = (e >> 6) == (e & 63);
  sync();
  if (kBlockInv) {
    double x[8][2];
    warp_rows_solve8<true>(D + 8 * warp * ld, Us, ui, lane, x);
  } else {
    warp_rows_trsm8_tc(D + 8 * warp * ld, Us, dis, lane);
  }
  sync();
  // X (row-major, gi) and y = X r.
  for (int e = tid; e < TB * TB; e += 256) {
    const int r = e >> 6, c = e & 63;
    gi[r * TB + c] = D[c * ld + r];
  }
  for (int e = tid; e < TB * F; e += 256) {
    const int r = e / F, f = e % F;
    double s = 0.0;
    for (int k = 0; k <= r; ++k) s = __fma_rn(D[k * ld + r], ys[k][f], s);
    rg[int64_t(r) * rld + f] = s;
  }
  // Every thread learns about a breakdown (warp 0 saw the pivots).
  __shared__ int bad_any;
  if (tid == 0) bad_any = 0;
  sync();
  if (bad) bad_any = 1;
  sync();
  return bad_any != 0;
}

__device__ __forceinline__ bool diag_tile(const double *g, int ld, double *rg, int rld, int F,
                                          double *gi, double *Xs, double *dis,
                                          double (*ys)[kMaxF], double *gu, int uld) {
  auto sync = [] { __syncthreads(); };
  return diag_tile_t<decltype(sync), false>(g, ld, rg, rld, F, gi, Xs, dis, ys, int(threadIdx.x),
                                            sync, gu, uld);
}

// The diagonal tile of step 0 of every slot.
__global__ void __launch_bounds__(256, 4) k_diag_chol(BigArgs a, const BigSlot *__restrict__ slots,
                                                      int j) {
  extern __shared__ double sm[];
  __shared__ double dis[TB];
  __shared__ double ys[TB][kMaxF];
  const BigSlot sl = slots[blockIdx.x];
  const int ld = sl.ld;
  double *gt = sm + TB * LDS;  // the evaluated tile A[j, j]
  double *pts = sm + 2 * TB * LDS;
  gen_tile(a, sl, j, j, TB, gt, pts, threadIdx.x, blockDim.x, sync_all);
  __syncthreads();
  double *rg = a.W + sl.base + int64_t(j) * TB * ld + int64_t(sl.T) * TB;
  const bool bad =
      diag_tile(gt, LDS, rg, ld, a.F, a.inv + sl.inv + int64_t(j) * TB * TB, sm, dis, ys,
                a.W + sl.base + int64_t(j) * TB * ld + int64_t(j) * TB, ld);
  if (threadIdx.x == 0 && bad) atomicOr(&a.status[sl.k], 4);
}

// The next diagonal tile after an int8 step j, one CTA per slot with
// T > j + 1 (the first cnt slots): D = D' - L[j+1, j] L[j+1, j]^T, with D'
// (the tile minus the products of columns p < j) written by the step's
// diagonal item to dpart and L[j+1, j] by its row item j + 1; then
// diag_tile_t with block-inverse row solves (X_{j+1}, U_{j+1}, y_{j+1}).  A
// separate launch rather than a hand-over inside the step: the factorisation
// of a 64 x 64 tile is a chain of 64 pivots that keeps one warp busy for tens
// of microseconds, and here two CTAs per SM overlap their chains while the
// step kernel's CTAs go on with their items.
constexpr size_t kDiagNextSmem =
    (size_t(2) * TB * LDS + size_t(4) * 16 * kUiLd + TB + TB * kMaxF) * sizeof(double);
__global__ void __launch_bounds__(256, 2) k_diag_next(BigArgs a, const BigSlot *__restrict__ slots,
                                                      int j) {
  extern __shared__ __align__(16) double smn[];
  double *D = smn;                  // D' and then D (TB x LDS)
  double *Ls = D + TB * LDS;        // L[j+1, j], then U scratch
  double *ui = Ls + TB * LDS;       // U's 16 x 16 diagonal block inverses
  double *dis = ui + 4 * 16 * kUiLd;
  double(*ys)[kMaxF] = reinterpret_cast<double(*)[kMaxF]>(dis + TB);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // The next step's launch may start now (its epilogue waits for this grid).
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
  const BigSlot sl = slots[blockIdx.x];
  const int ld = sl.ld;
  double *W = a.W + sl.base;
  const double *dp = a.dpart + int64_t(sl.q) * TB * TB;
  const double *lg = W + int64_t(j + 1) * TB * ld + int64_t(j) * TB;
  for (int idx = tid; idx < TB * TB / 2; idx += 256) {
    const int r = idx >> 5, c2 = idx & 31;
    cp_async16(D + r * LDS + 2 * c2, dp + r * TB + 2 * c2);
    cp_async16(Ls + r * LDS + 2 * c2, lg + int64_t(r) * ld + 2 * c2);
  }
  // r_{j+1} (the first F columns of the residual tile), for y = X r.
  double *rg = W + int64_t(j + 1) * TB * ld + int64_t(sl.T) * TB;
  for (int e = tid; e < TB * a.F; e += 256)
    cp_async8(&ys[e / a.F][e % a.F], rg + int64_t(e / a.F) * ld + e % a.F);
  cp_async_commit();
  cp_async_wait<0>();
  __syncthreads();
  {
    const int wr = (warp >> 1) * 32, wc = (warp & 1) * 32;
    double acc[4][4][2];
    if (warp < 4) {
      acc_load(acc, D, LDS, wr, wc, lane);
      mma64<false, true>(Ls, Ls, acc, -1.0, wr, wc, lane);
    }
    __syncthreads();
    if (warp < 4) acc_store(acc, D, LDS, wr, wc, lane);
  }
  __syncthreads();
  auto sync = [] { __syncthreads(); };
  const bool bad = diag_tile_t<decltype(sync), true>(
      D, LDS, rg, ld, a.F, a.inv + sl.inv + int64_t(j + 1) * TB * TB, Ls, dis, ys, tid, sync,
      W + int64_t(j + 1) * TB * ld + int64_t(j + 1) * TB, ld, ui, true);
  if (tid == 0 && bad) atomicOr(&a.status[sl.k], 4);
}

// Phase 2 of a factorisation step (256 threads, warp w: rows 16 w .. + 15,
// in two passes of 8).  sC holds C (row tiles i0, and i0 + 1 when arows =
// 2 TB; kColRows x LDS).  L[i, j] solves L[i, j] U_j = C with U_j = L_jj^T
// (the factor of the diagonal tile, loaded into sU), by blocked row solves
// (warp_rows_trsm8_tc); it is stored in the workspace and written back over C
// in sC (in place); then the forward substitution r_i -=
// L[i, j] y_j.  vec holds TB + TB kMaxF doubles (1 / diag(U_j), y_j).  Ends
// with a barrier.
__device__ void step_trsm(const BigArgs &a, const BigSlot &sl, int j, int i0, int arows,
                          double *sC, double *sU, double *vec) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int ld = sl.ld, F = a.F;
  double *W = a.W + sl.base;
  double *rcol = W + int64_t(sl.T) * TB;
  double *dinv = vec, *ysh = vec + TB;
  load_factor_async(sU, W + int64_t(j) * TB * ld + int64_t(j) * TB, ld, tid, kColThreads);
  cp_async_commit();
  {
    const double *yg = rcol + int64_t(j) * TB * ld;
    for (int e = tid; e < TB * kMaxF; e += kColThreads) {
      const int r = e / kMaxF, f = e % kMaxF;
      ysh[e] = f < F ? __ldcg(yg + int64_t(r) * ld + f) : 0.0;
    }
  }
  cp_async_wait<0>();
  __syncthreads();
  if (tid < TB) dinv[tid] = 1.0 / sU[tid * LDS + tid];
  __syncthreads();
  double *C = W + int64_t(i0) * TB * ld + int64_t(j) * TB;
  double *rg = rcol + int64_t(i0) * TB * ld;
  for (int pass = 0; pass < 2; ++pass) {
    const int r0 = 16 * warp + 8 * pass;
    if (r0 >= arows) break;
    warp_rows_trsm8_tc(sC + r0 * LDS, sU, dinv, lane);
    double lo[8], hi[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      lo[q] = sC[(r0 + q) * LDS + lane];
      hi[q] = sC[(r0 + q) * LDS + 32 + lane];
      C[int64_t(r0 + q) * ld + lane] = lo[q];
      C[int64_t(r0 + q) * ld + 32 + lane] = hi[q];
    }
    for (int f = 0; f < F; ++f) {
      const double yl = ysh[lane * kMaxF + f], yh = ysh[(lane + 32) * kMaxF + f];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        double sum = __fma_rn(lo[q], yl, hi[q] * yh);
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        if (lane == 0) rg[int64_t(r0 + q) * ld + f] -= sum;
      }
    }
  }
  __syncthreads();
}

// ---------------------------------------------------------------------------
// Column updates on the int8 tensor cores (precision "mixed")
// ---------------------------------------------------------------------------
//
// Every finished off-diagonal tile L[i, p] is also kept as kOzS int8 digit
// slices of x = L / sigma (sigma >= sqrt(max_r A_rr) bounds every entry of L,
// since the rows of L have norm sqrt(A_rr)): x = sum_s d_s 128^-s, d_1 in
// [-127, 127], d_s in [-64, 64] after.  The update
//   sum_p L[i, p] L[j, p]^T = sigma^2 sum_{a,b} 128^-(a+b) D_a[i] D_b[j]^T
// keeps the slice pairs with a + b <= kOzS + 2 (levels 2..9) and sums each
// level exactly in int32 on the tcgen05 tensor cores (kind::i8); the levels
// are combined in int64 and FP64 at the end.  A digit product is at most
// 2^12 in magnitude, so a dropped term (level >= 10) is below 2^-58 sigma^2:
// the truncation of a K-long sum stays near the FP64 rounding of the same
// sum.  Dropping level 9 as well (2^-51 per term) is not enough: on patches
// with cond(A) ~ 1e13 it multiplies the error of the local values by ~15.
// This is the split-integer emulation of an FP64 product (Ozaki, Ogita, Oishi
// and Rump 2012; Uchino, Ozaki and Imamura 2024 for integer tensor cores).
//
// Slice tile layout (28 KB): [16-byte K chunk (4)][slice (kOzS)][8-row group
// (8)][8 rows x 16 bytes], i.e. the K-major core-matrix layout of the tensor
// core, copied to shared memory with bulk async copies.  Every tile is written
// twice: by itself, and interleaved slice by slice with the other tile of its
// row pair (16 row groups per slice).
constexpr int kOzS = 7;
constexpr int kOzTileBytes = 4 * kOzS * 8 * 128;      // 28672
constexpr int kOzTmemCols = 512;                      // 8 column groups of 64 (levels 2..9)
constexpr int kOzWaitLimit = 1 << 22;                 // bounded mbarrier polls
// Polls of the waits that drain a pipeline after it gave up: they wait for
// copies and tensor-core operations already issued, which complete by
// themselves, so they get a longer limit than the pipeline waits
// (BigArgs::wait_limit) and are never shortened.
constexpr int kOzDrainLimit = 1 << 24;


__device__ __forceinline__ uint32_t saddr(const void *p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint64_t *b, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(saddr(b)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *b, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(saddr(b)),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive_cnt(uint64_t *b, uint32_t cnt) {
  asm volatile("mbarrier.arrive.release.cta.shared::cta.b64 _, [%0], %1;\n" ::"r"(saddr(b)),
               "r"(cnt)
               : "memory");
}
__device__ __forceinline__ bool mbar_try(uint64_t *b, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      "selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(done)
      : "r"(saddr(b)), "r"(parity)
      : "memory");
  return done != 0;
}
// Bounded wait for the phase with the given parity; false on time-out.
__device__ __forceinline__ bool mbar_wait(uint64_t *b, uint32_t parity, int limit = kOzWaitLimit) {
  bool done = false;
  for (int it = 0; it < limit && !done; ++it) done = mbar_try(b, parity);
  return done;
}
// Pipeline wait of the int8 K loop: bounded by `limit` polls, and given up
// at once when the other side of the pipeline has aborted.
__device__ __forceinline__ bool mbar_wait_pipe(uint64_t *b, uint32_t parity, int limit,
                                               volatile int *abort_flag) {
  for (int it = 0; it < limit; ++it) {
    if (mbar_try(b, parity)) return true;
    if (*abort_flag) return false;
  }
  return false;
}
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, uint32_t bytes, uint64_t *b) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
          saddr(dst)),
      "l"(src), "r"(bytes), "r"(saddr(b))
      : "memory");
}
// Shared-memory matrix descriptor, K-major core matrices without swizzle
// (layout type 0, descriptor version 1): lbo = byte step between 16-byte K
// chunks, sbo = byte step between 8-row groups.
__device__ __forceinline__ uint64_t umma_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  return uint64_t((addr >> 4) & 0x3FFF) | (uint64_t((lbo >> 4) & 0x3FFF) << 16) |
         (uint64_t((sbo >> 4) & 0x3FFF) << 32) | (uint64_t(1) << 46);
}
// Instruction descriptor: D s32, A and B signed int8, both K-major, M = 128.
__device__ __forceinline__ uint32_t umma_idesc_i8(int n) {
  return (2u << 4) | (1u << 7) | (1u << 10) | (uint32_t(n >> 3) << 17) | (uint32_t(128 >> 4) << 24);
}
__device__ __forceinline__ void umma_i8(uint32_t dtmem, uint64_t ad, uint64_t bd, uint32_t idesc,
                                        uint32_t accumulate) {
  asm volatile(
      "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n}\n" ::"r"(dtmem),
      "l"(ad), "l"(bd), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void umma_commit(uint64_t *b) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(
                   saddr(b))
               : "memory");
}
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
}

// Slice storage of a slot with T tile rows, in bytes from its sli: first the
// plain tiles of the strictly lower triangle, row by row (operand B: the
// column tile row's slices stacked along N), then the pair tiles, the rows
// 2u and 2u + 1 interleaved per slice (operand A: M = 128), pair u with its
// 2u + 1 columns.
constexpr int kOzPairBytes = 2 * kOzTileBytes;
__host__ __device__ __forceinline__ int64_t oz_tile_off(int i, int p) {
  return (int64_t(i) * (i - 1) / 2 + p) * kOzTileBytes;
}
__host__ __device__ __forceinline__ int64_t oz_pair_off(int T, int u, int p) {
  return int64_t(T) * (T - 1) / 2 * kOzTileBytes + (int64_t(u) * u + p) * kOzPairBytes;
}

// The kOzS balanced base-128 digits of x = v mul / 128 in [-1, 1]: y = x
// 128^kOzS rounded to an integer (in the low bits of a double at 1.5 2^52),
// plus 64 in each of the lower digits, is a row of unsigned 7-bit fields f with
// d = f - 64 and a signed top digit in [-127, 127].  bytes[s] |= the field of
// digit s, shifted; oz_bytes turns four fields into four int8 digits.
__device__ __forceinline__ void oz_fields(double v, double mul, int shift, uint32_t *bytes) {
  constexpr double kOne = 0x1.8p52, kMax = 127.49 * 0x1p42;
  constexpr long long kBias = 64ll * (1 + (1ll << 7) + (1ll << 14) + (1ll << 21) + (1ll << 28) +
                                      (1ll << 35));
  double t = __fma_rn(v, mul * 0x1p42, kOne);
  t = fmin(fmax(t, kOne - kMax), kOne + kMax);
  const long long y = __double_as_longlong(t) - __double_as_longlong(kOne) + kBias;
  const uint32_t lo = uint32_t(y), hi = uint32_t(uint64_t(y) >> 32);
  const uint32_t f[kOzS] = {hi >> 10,          hi >> 3,  __funnelshift_r(lo, hi, 28),
                            lo >> 21,          lo >> 14, lo >> 7,
                            lo};
  bytes[0] |= (f[0] & 0xffu) << shift;
#pragma unroll
  for (int s = 1; s < kOzS; ++s) bytes[s] |= (f[s] & 0x7fu) << shift;
}
// Four 7-bit fields -> four int8 values field - 64.
__device__ __forceinline__ uint32_t oz_bytes(uint32_t f) {
  const uint32_t r = f ^ 0x40404040u;
  return r | ((r & 0x40404040u) << 1);
}
// Stores the 16-byte word of every slice of row r (0..63), K chunk c16 of
// L[i, p] in the plain and the pair tile.
__device__ __forceinline__ void oz_store(const uint4 (&w)[kOzS], int r, int c16, uint8_t *slices,
                                         int T, int i, int p) {
  uint8_t *tile = slices + oz_tile_off(i, p) + c16 * kOzS * 1024 + r * 16;
  uint8_t *pair = slices + oz_pair_off(T, i >> 1, p) + c16 * kOzS * 2048 + (i & 1) * 1024 + r * 16;
#pragma unroll
  for (int sl = 0; sl < kOzS; ++sl) {
    *reinterpret_cast<uint4 *>(tile + sl * 1024) = w[sl];
    *reinterpret_cast<uint4 *>(pair + sl * 2048) = w[sl];
  }
}

// The digits of row r (0..63) and 16-column K chunk c16 of L[i, p], held in
// shared memory at sL (row stride LDS).
__device__ __forceinline__ void slice_row_chunk(const double *sL, int r, int c16, double mul,
                                                uint8_t *slices, int T, int i, int p) {
  uint4 w[kOzS];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    uint32_t b[kOzS] = {};
#pragma unroll
    for (int cc = 0; cc < 4; ++cc)
      oz_fields(sL[r * LDS + 16 * c16 + 4 * q + cc], mul, 8 * cc, b);
#pragma unroll
    for (int sl = 0; sl < kOzS; ++sl) {
      const uint32_t v = sl ? oz_bytes(b[sl]) : b[sl];
      (q == 0 ? w[sl].x : q == 1 ? w[sl].y : q == 2 ? w[sl].z : w[sl].w) = v;
    }
  }
  oz_store(w, r, c16, slices, T, i, p);
}

// The digits of a warp's 8 rows r0.. of L[i, p] from the accumulator layout
// (lane: row r0 + lane / 4, columns 8 nt + 2 t, + 1): a lane's four bytes of
// every K chunk are exchanged among the four lanes of its row, after which
// lane t holds the whole 16-byte word of chunk t.
__device__ __forceinline__ void slice_rows_acc(const double (&c)[8][2], int r0, int lane,
                                               double mul, uint8_t *slices, int T, int i, int p) {
  const int t = lane & 3;
  uint32_t v[4][kOzS];  // [chunk][slice]: columns 2t, 2t + 1, 8 + 2t, 9 + 2t of the chunk
#pragma unroll
  for (int ch = 0; ch < 4; ++ch) {
    uint32_t b[kOzS] = {};
#pragma unroll
    for (int e = 0; e < 4; ++e) oz_fields(c[2 * ch + (e >> 1)][e & 1], mul, 8 * e, b);
#pragma unroll
    for (int sl = 0; sl < kOzS; ++sl) v[ch][sl] = sl ? oz_bytes(b[sl]) : b[sl];
  }
  uint4 w[kOzS];
#pragma unroll
  for (int sl = 0; sl < kOzS; ++sl) {
    // 4 x 4 transpose over the lanes t (bit 1, then bit 0).
    const bool up = t & 2, odd = t & 1;
    const uint32_t s0 = up ? v[0][sl] : v[2][sl], s1 = up ? v[1][sl] : v[3][sl];
    const uint32_t k0 = up ? v[2][sl] : v[0][sl], k1 = up ? v[3][sl] : v[1][sl];
    const uint32_t g0 = __shfl_xor_sync(0xffffffffu, s0, 2), g1 = __shfl_xor_sync(0xffffffffu, s1, 2);
    // Lower lanes now hold chunks 0 and 1 of the lanes t and t + 2, upper
    // lanes chunks 2 and 3 of the lanes t - 2 and t.
    const uint32_t a0 = up ? g0 : k0, a1 = up ? g1 : k1;  // from the lower lane of the two
    const uint32_t b0 = up ? k0 : g0, b1 = up ? k1 : g1;  // from the upper one
    const uint32_t sa = odd ? a0 : a1, sb = odd ? b0 : b1;
    const uint32_t ka = odd ? a1 : a0, kb = odd ? b1 : b0;
    const uint32_t ga = __shfl_xor_sync(0xffffffffu, sa, 1), gb = __shfl_xor_sync(0xffffffffu, sb, 1);
    // o[q]: the bytes of lane q of the row for this lane's chunk.
    const uint32_t o0 = odd ? ga : ka, o1 = odd ? ka : ga;
    const uint32_t o2 = odd ? gb : kb, o3 = odd ? kb : gb;
    w[sl] = make_uint4(__byte_perm(o0, o1, 0x5410), __byte_perm(o2, o3, 0x5410),
                       __byte_perm(o0, o1, 0x7632), __byte_perm(o2, o3, 0x7632));
  }
  oz_store(w, r0 + (lane >> 2), t, slices, T, i, p);
}

// Step j of the factorisation, one launch over all slots with T > j + 1.
// CTA l of a slot owns row tiles i0 = j + 1 + 2l and i0 + 1 of tile column j:
//  1. C = A[i, j] - sum_{p<j} L[i, p] L[j, p]^T: eight warps hold 32 x 32
//     accumulators (starting at -A) for the whole K loop, the L panels stream
//     through a cp.async pipeline;
//  2. L[i, j] U_j = C, the triangular solve against the diagonal tile's
//     factor (made one step earlier), stored; then the forward
//     substitution r_i -= L[i, j] y_j;
//  3. CTA 0 (i0 = j + 1) forms the next diagonal tile
//     D = A[j+1, j+1] - sum_{p<=j} L[j+1, p] L[j+1, p]^T and factors it:
//     X_{j+1} and y_{j+1} = X_{j+1} r_{j+1} for step j + 1.
template <bool SLICE>
__global__ void __launch_bounds__(kColThreads, 2)
    k_col_step(BigArgs a, const BigSlot *__restrict__ slots, const int *__restrict__ pre, int cnt,
               int j) {
  extern __shared__ double sm[];
  // The first cnt CTAs are the slots' CTA 0 (the longest: they also form the
  // next diagonal tile), so they start in the first wave; the other CTAs
  // (l >= 1) follow, addressed through the prefix counts.
  int q, l;
  if (int(blockIdx.x) < cnt) {
    q = blockIdx.x;
    l = 0;
  } else {
    const int b = blockIdx.x - cnt;
    q = find_slot(pre, cnt, b);
    l = 1 + b - pre[q];
  }
  const BigSlot sl = slots[q];
  const int i0 = j + 1 + 2 * l;
  const bool two = i0 + 1 < sl.T;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int wr = (warp >> 1) * 32, wc = (warp & 1) * 32;
  const int ld = sl.ld, F = a.F;
  double *W = a.W + sl.base;
  double *rcol = W + int64_t(sl.T) * TB;
  const double *gA = W + int64_t(i0) * TB * ld;
  const double *gB = W + int64_t(j) * TB * ld;
  const int arows = two ? kColRows : TB;
  const int nch = j * (TB / kKC);
  auto load = [&](int c, int stage) {
    double *sA = sm + stage * kColStage;
    double *sB = sA + kColRows * kKLD;
    const int col = c * kKC;
    for (int idx = tid; idx < (kColRows + TB) * (kKC / 2); idx += kColThreads) {
      const int r = idx / (kKC / 2), c2 = idx % (kKC / 2);
      if (r < kColRows) {
        if (r < arows) cp_async16(sA + r * kKLD + 2 * c2, gA + int64_t(r) * ld + col + 2 * c2);
      } else {
        const int rb = r - kColRows;
        cp_async16(sB + rb * kKLD + 2 * c2, gB + int64_t(rb) * ld + col + 2 * c2);
      }
    }
  };
  const bool active = two || wr < TB;
  double acc[4][4][2];
  gen_tile(a, sl, i0, j, arows, sm, sm + kColRows * LDS, tid, kColThreads, sync_all);  // A[i, j]
  __syncthreads();
  if (active) {
    acc_load(acc, sm, LDS, wr, wc, lane);
    acc_neg(acc);
  }
  __syncthreads();
#pragma unroll
  for (int s = 0; s < kStages - 1; ++s) {
    if (s < nch) load(s, s);
    cp_async_commit();
  }
  for (int c = 0; c < nch; ++c) {
    cp_async_wait<kStages - 2>();
    __syncthreads();
    if (c + kStages - 1 < nch) load(c + kStages - 1, (c + kStages - 1) % kStages);
    cp_async_commit();
    if (active) {
      const double *sA = sm + (c % kStages) * kColStage;
      mma_chunk_nt(sA, sA + kColRows * kKLD, acc, wr, wc, lane);
    }
  }
  cp_async_wait<0>();
  __syncthreads();

  // 2. L[i, j] U_j = C through shared memory, then the forward substitution.
  if (active) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int jj = 0; jj < 4; ++jj)
        *reinterpret_cast<double2 *>(sm + (wr + 8 * i + g) * LDS + wc + 8 * jj + 2 * t) =
            make_double2(-acc[i][jj][0], -acc[i][jj][1]);
  }
  __syncthreads();
  step_trsm(a, sl, j, i0, arows, sm, sm + kColRows * LDS, sm + (kColRows + TB) * LDS);
  if (SLICE) {  // int8 slices of the new L tiles for the int8 steps that follow
    for (int u = tid; u < arows * 4; u += kColThreads) {
      const int h = u >> 8;
      slice_row_chunk(sm + h * TB * LDS, u & 63, (u >> 6) & 3, a.oz_mul, a.slices + sl.sli, sl.T,
                      i0 + h, j);
    }
  }
  if (l != 0) return;

  // 3. The diagonal tile of step j + 1 (this CTA's first row tile).
  __syncthreads();
  constexpr int kDStage = TB * kKLD;
  double *sL = sm + 2 * kDStage;  // L[j+1, j], TB x LDS (rows 0..63 of sC are below it)
  static_assert(2 * kDStage >= TB * LDS, "L[j+1, j] overlaps its copy source");
  for (int e = tid; e < TB * TB; e += kColThreads) sL[(e >> 6) * LDS + (e & 63)] = sm[(e >> 6) * LDS + (e & 63)];
  __syncthreads();
  auto loadd = [&](int c, int stage) {
    double *sD = sm + stage * kDStage;
    const int col = c * kKC;
    for (int idx = tid; idx < TB * (kKC / 2); idx += kColThreads) {
      const int r = idx / (kKC / 2), c2 = idx % (kKC / 2);
      cp_async16(sD + r * kKLD + 2 * c2, gA + int64_t(r) * ld + col + 2 * c2);
    }
  };
  const bool dact = wr < TB;
  double *Dgen = sm + 2 * kDStage + TB * LDS;  // A[j+1, j+1], after sL
  gen_tile(a, sl, j + 1, j + 1, TB, Dgen, sm, tid, kColThreads, sync_all);
  __syncthreads();
  if (dact) {
    acc_load(acc, Dgen, LDS, wr, wc, lane);
    acc_neg(acc);
  }
  __syncthreads();
#pragma unroll
  for (int s = 0; s < kStages - 1; ++s) {
    if (s < nch) loadd(s, s);
    cp_async_commit();
  }
  for (int c = 0; c < nch; ++c) {
    cp_async_wait<kStages - 2>();
    __syncthreads();
    if (c + kStages - 1 < nch) loadd(c + kStages - 1, (c + kStages - 1) % kStages);
    cp_async_commit();
    if (dact) {
      const double *sD = sm + (c % kStages) * kDStage;
      mma_chunk_nt(sD, sD, acc, wr, wc, lane);
    }
  }
  cp_async_wait<0>();
  __syncthreads();
  if (dact) mma64<false, true>(sL, sL, acc, 1.0, wr, wc, lane);
  double *Ds = sm;  // TB x LDS, over the finished stages
  if (dact) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int jj = 0; jj < 4; ++jj)
        *reinterpret_cast<double2 *>(Ds + (wr + 8 * i + g) * LDS + wc + 8 * jj + 2 * t) =
            make_double2(-acc[i][jj][0], -acc[i][jj][1]);
  }
  __syncthreads();
  // Scratch of the factorisation over the consumed L[j+1, j] (sL).
  double *Xs = sm + TB * LDS;
  double(*ysd)[kMaxF] = reinterpret_cast<double(*)[kMaxF]>(Xs + TB * LDS);
  double *dis = Xs + TB * LDS + TB * kMaxF;
  const bool bad = diag_tile(Ds, LDS, rcol + int64_t(j + 1) * TB * ld, ld, F,
                             a.inv + sl.inv + int64_t(j + 1) * TB * TB, Xs, dis, ysd,
                             W + int64_t(j + 1) * TB * ld + int64_t(j + 1) * TB, ld);
  if (tid == 0 && bad) atomicOr(&a.status[sl.k], 4);
}

// ---------------------------------------------------------------------------
// Warp-specialised int8 step (k_col_step_ws)
// ---------------------------------------------------------------------------
//
// Step j of the factorisation with the column update on the int8 tensor
// cores, organised so that the int8 K loop of one item overlaps the FP64
// epilogue of the previous one on the same SM.  An item is the pair of row
// tiles 2u, 2u + 1 of column j, as far as they lie below row j
// (C = A[i, j] - sum_{p<j} L[i, p] L[j, p]^T, then L[i, j] U_j = C solved
// against the diagonal tile's factor, the forward substitution and the int8
// slices of L[i, j]), or the diagonal item of a slot (D' of tile j + 1, left
// in dpart for k_diag_next).  The CTAs take the items round robin; nothing
// waits on another CTA.
//   warp 0 (one thread): bulk copies of the slice half-tiles (K = 32) of the
//     row pair and of the column tile row through a kWsStages ring;
//   warp 1 (one thread): the tcgen05 MMAs into one TMEM accumulator;
//   warps 2..17: per item the Wendland tiles (during the K loop), the TMEM
//     drain (after which the MMA thread starts the next item), the level
//     combination and the FP64 epilogue.
// The MMA operand A is one slice of the pair (rows 0..63 tile 2u, 64..127 tile
// 2u + 1), B the slices of the column tile stacked along N; the accumulator
// of slice pair (a, b) is TMEM column group a + b - 2 (64 columns), so the
// eight groups hold the levels 2..9 of both tiles and eleven MMAs per K = 32
// cover the 34 slice pairs with a + b <= 9, none of them twice.
//
// Why pairs and sixteen epilogue warps: with one row tile per item (two
// slices stacked in M, six MMAs with 38 of the digit products per tile, eight
// epilogue warps) a K = 32 half took 1,170 cycles for 28 KB of copies and 63
// KB of operand reads, and up to step 12 the item's time was its epilogue, whose
// FP64 chains eight warps could not hide.  A pair shares the column's copy and
// operand reads (43 KB and 112 KB for two tiles) and drains two tiles in the
// time of one.  The items go round robin, so that the CTAs at work on a slot
// read the column's slices together from L2 (in contiguous ranges they came
// from DRAM once per item: 5.3 TB/s, 2% L2 hits).  After the solve the rows of
// L stay in registers for the store, the forward substitution and the digits
// (through shared memory these took 23k cycles of an item, now 9k).
// 1M refined points, all steps of one slot group: 68 -> 53 ms; step 18 of a
// quarter of it, under ncu: tensor pipe 60% of active cycles, DRAM 53%.
//
// The FP64 tensor instructions of the solve share the tensor pipe with the
// MMAs (6.5k cycles without, 14k beside them), and the K loop in turn is
// slowed.  While the K loop is shorter than the rest of an item (steps below
// kWsLate) the accumulator goes back after the solve instead of after the
// drain: steps 2..8 take 10-15% less that way, steps from 12 on 5-8% more.
constexpr int kWsStages = 2;
constexpr int kWsChunk = kOzS * 1024;                    // 7168: one 16-byte K chunk, 7 slices
constexpr int kWsHalf = 2 * kWsChunk;                    // 14336: one K = 32 half of a slice tile
constexpr int kWsChunkA = 2 * kWsChunk;                  // the same of a row pair
constexpr int kWsHalfA = 2 * kWsHalf;
constexpr int kWsStage = kWsHalfA + kWsHalf;             // pair half + column half
constexpr int kWsEpi = 512;                              // epilogue threads
constexpr int kWsThreads = kWsEpi + 64;                  // + 2 issue warps
constexpr int kWsRows = 2 * TB;
constexpr int kWsLate = 9;                               // steps that hand the accumulator back late
constexpr int kWsCOff = kWsStages * kWsStage;            // C / L / D' (kWsRows x LDS doubles)
constexpr int kWsXOff = kWsCOff + kWsRows * LDS * 8;     // U_j, the diagonal tile's factor
constexpr int kWsPtsOff = kWsXOff + TB * LDS * 8;        // points of two items
constexpr int kWsPts = kWsRows + TB;
constexpr int kWsRedOff = kWsPtsOff + 2 * kWsPts * 32;   // y_j, r_i
constexpr int kWsUiOff = kWsRedOff + (TB + kWsRows) * kMaxF * 8;  // U_j's diagonal block inverses
constexpr int kWsBarOff = kWsUiOff + 4 * 16 * kUiLd * 8;
constexpr size_t kWsSmem = size_t(kWsBarOff) + 256;
static_assert(kWsSmem <= 232448, "shared memory of k_col_step_ws");
static_assert(kWsStage % 1024 == 0, "stages start on 1 KB boundaries");

struct WsBars {
  uint64_t full[kWsStages], empty[kWsStages], acc_full, acc_empty, done;
  int abort_flag, ep_stop;
  uint32_t tmem;
};
static_assert(sizeof(WsBars) <= 256, "barrier area");

// Row pairs of a slot with T tile rows that reach below row j.
__host__ __device__ __forceinline__ int ws_pairs(int T, int j) {
  return (T - 1) / 2 - (j + 1) / 2 + 1;
}
// The item `it` of step j: slot q (prefix counts ipre over the cnt active
// slots), and r = it - ipre[q]: r == 0 the diagonal item, else pair
// (j + 1) / 2 + r - 1.
struct WsItem {
  int q, r;
};
__device__ __forceinline__ WsItem ws_item(const int *ipre, int cnt, int it) {
  const int q = find_slot(ipre, cnt, it);
  return {q, it - ipre[q]};
}
__device__ __forceinline__ int ws_pair(int j, int r) { return (j + 1) / 2 + (r ? r - 1 : 0); }
// The item by a whole warp, searching on from slot q0 (at or before the
// item's): the lanes look at 32 slots at once, one load's latency where a
// thread stepping from slot to slot pays one for each.
__device__ __forceinline__ WsItem ws_find(const int *__restrict__ ipre, int cnt, int it, int q0,
                                          int lane) {
  for (;; q0 += 32) {
    const int e = q0 + 1 + lane;
    const int end = e <= cnt ? ipre[e] : 0x7fffffff;
    const unsigned int m = __ballot_sync(0xffffffffu, end > it);
    if (m) {
      const int q = q0 + __ffs(m) - 1;
      return {q, it - ipre[q]};
    }
  }
}

// The MMAs of one K = 32 half.  On the first half of an item the first MMA to
// reach a column overwrites it: slice 1 groups 0..3, slice 5 groups 4..7,
// issued first.
__device__ __forceinline__ void ws_mma_half(uint32_t tmem, uint32_t sA, uint32_t sB, bool first) {
  const uint32_t acc = first ? 0u : 1u;
  auto ad = [&](int a) { return umma_desc(sA + (a - 1) * 2048, kWsChunkA, 128); };
  const uint64_t b1 = umma_desc(sB, kWsChunk, 128);             // slices 1..4
  const uint64_t b5 = umma_desc(sB + 4 * 1024, kWsChunk, 128);  // slices 5..7
  umma_i8(tmem, ad(1), b1, umma_idesc_i8(256), acc);         // groups 0..3
  umma_i8(tmem + 256, ad(5), b1, umma_idesc_i8(256), acc);   // groups 4..7
  umma_i8(tmem + 256, ad(1), b5, umma_idesc_i8(192), 1u);    // 1 x 5..7: groups 4..6
  umma_i8(tmem + 64, ad(2), b1, umma_idesc_i8(256), 1u);     // 2 x 1..4: groups 1..4
  umma_i8(tmem + 320, ad(2), b5, umma_idesc_i8(192), 1u);    // 2 x 5..7: groups 5..7
  umma_i8(tmem + 128, ad(3), b1, umma_idesc_i8(256), 1u);    // 3 x 1..4: groups 2..5
  umma_i8(tmem + 384, ad(3), b5, umma_idesc_i8(128), 1u);    // 3 x 5..6: groups 6..7
  umma_i8(tmem + 192, ad(4), b1, umma_idesc_i8(256), 1u);    // 4 x 1..4: groups 3..6
  umma_i8(tmem + 448, ad(4), b5, umma_idesc_i8(64), 1u);     // 4 x 5: group 7
  umma_i8(tmem + 320, ad(6), b1, umma_idesc_i8(192), 1u);    // 6 x 1..3: groups 5..7
  umma_i8(tmem + 384, ad(7), b1, umma_idesc_i8(128), 1u);    // 7 x 1..2: groups 6..7
}

// An epilogue warp reads TMEM lanes 32 qd .. + 31 (rows of the pair) and
// columns 16 h .. + 15 of every column group: the sums of levels 2..9 of its
// rows.  The levels are merged in int64 first: a level's sum is below 2^31
// (kOzMaxT), so the top three shifted
// by 7 bits each stay below 2^53 and convert exactly, and the lower five
// (below 2^60 in units of 128^-9) round to within 2^-57; then two FP64 terms
// (in units of sigma^2), of which sig2 x their sum is subtracted from sC
// (which holds A).
__device__ __forceinline__ void ws_drain(uint32_t tmem, int qd, int h, double *sC, double sig2,
                                         int lane) {
  constexpr int kG = 8;  // column groups, levels 2..9
  const uint32_t base = tmem + (uint32_t(32 * qd) << 16) + uint32_t(16 * h);
  // Four columns per step: the levels are merged into (hi, lo), the loads of
  // step cb + 1 are issued, and the conversions and stores of step cb run
  // while they are in flight.
  uint32_t z[kG][4];
  auto issue = [&](int cb) {
#pragma unroll
    for (int g = 0; g < kG; ++g)
      asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];\n"
                   : "=r"(z[g][0]), "=r"(z[g][1]), "=r"(z[g][2]), "=r"(z[g][3])
                   : "r"(base + uint32_t(64 * g + 4 * cb)));
  };
  double *cr = sC + (32 * qd + lane) * LDS + 16 * h;
  issue(0);
#pragma unroll
  for (int cb = 0; cb < 4; ++cb) {
    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
    long long hi[4], lo[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const long long z0 = int32_t(z[0][c]), z1 = int32_t(z[1][c]), z2 = int32_t(z[2][c]);
      const long long z3 = int32_t(z[3][c]), z4 = int32_t(z[4][c]), z5 = int32_t(z[5][c]);
      const long long z6 = int32_t(z[6][c]), z7 = int32_t(z[7][c]);
      hi[c] = (z0 * 128 + z1) * 128 + z2;
      lo[c] = (((z3 * 128 + z4) * 128 + z5) * 128 + z6) * 128 + z7;
    }
    if (cb < 3) issue(cb + 1);
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const double val = __fma_rn(double(hi[c]), 0x1p-28, double(lo[c]) * 0x1p-63);
      cr[4 * cb + c] = __fma_rn(-sig2, val, cr[4 * cb + c]);
    }
  }
}

__device__ __forceinline__ void ws_sync() { asm volatile("bar.sync 1, 512;\n" ::: "memory"); }
static_assert(kWsEpi == 512, "ws_sync counts the epilogue threads");

// Points of an item, kWsPts of them: the rows 2u TB .. of the pair, then the
// columns of tile tj.  Thread e loads the membership index of its point early
// (ws_point_index) and copies the point into pts[e] later (ws_point_copy,
// cp.async; zeros past n), so that the next item's points arrive while the
// current item's epilogue runs.
__device__ __forceinline__ int ws_point_index(const BigArgs &a, const BigSlot &sl, int u, int tj,
                                              int e) {
  const int gi = e < kWsRows ? 2 * u * TB + e : tj * TB + (e - kWsRows);
  return gi < sl.n ? a.sidx[a.soff[sl.k] + gi] : -1;
}
__device__ __forceinline__ void ws_point_copy(const BigArgs &a, double4 *pts, int e, int idx) {
  if (idx >= 0) {
    const double *g = reinterpret_cast<const double *>(a.src + idx);
    double *d = reinterpret_cast<double *>(pts + e);
    cp_async16(d, g);
    cp_async16(d + 2, g + 2);
  } else {
    pts[e] = make_double4(0.0, 0.0, 0.0, 0.0);
  }
}

// Rows [64 h0, 64 h1) of A[2u.., tj] into sT (row stride LDS) by the epilogue
// threads from the item's points.  Thread t takes column t % 64 of every
// eighth row; the evaluations are free of branches, so that their FP64 chains
// overlap.
__device__ __forceinline__ void ws_gen_rows(const BigArgs &a, const BigSlot &sl, int u, int tj,
                                            int h0, int h1, double *sT, const double4 *pts,
                                            int t) {
  const int c = t & 63, gj = tj * TB + c;
  const double4 pc = pts[kWsRows + c];
  with_basis(a.basis, [&](auto B) {
#pragma unroll 4
    for (int m = 8 * h0; m < 8 * h1; ++m) {
      const int r = (t >> 6) + 8 * m;
      const int gi = 2 * u * TB + r;
      const double4 pr = pts[r];
      const double w = phi_at<B>(sqdist3(pr.x, pr.y, pr.z, pc.x, pc.y, pc.z), a.rinv);
      const double pad = (gi == gj) ? 1.0 : 0.0;
      sT[r * LDS + c] = (gi < sl.n && gj < sl.n) ? w : pad;
    }
  });
}

__global__ void __launch_bounds__(kWsThreads, 1)
    k_col_step_ws(BigArgs a, const BigSlot *__restrict__ slots, const int *__restrict__ ipre,
                  int cnt, int j) {
  extern __shared__ __align__(1024) uint8_t smb[];
  WsBars *bar = reinterpret_cast<WsBars *>(smb + kWsBarOff);
  volatile int *abort_flag = &bar->abort_flag;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nitems = ipre[cnt];
  const int it0 = blockIdx.x, it1 = nitems, step = gridDim.x;
  const int nh = 2 * j;  // K = 32 halves per item
  if (tid == 0) {
    for (int i = 0; i < kWsStages; ++i) {
      mbar_init(&bar->full[i], 1);
      mbar_init(&bar->empty[i], 1);
    }
    mbar_init(&bar->acc_full, 1);
    mbar_init(&bar->acc_empty, kWsEpi / 32);
    mbar_init(&bar->done, 1);
    bar->abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(
                     saddr(&bar->tmem)),
                 "r"(kOzTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = bar->tmem;

  if (warp == 0) {
    // Producer: the warp finds the items, lane 0 issues the copies.
    int hc = 0;
    bool ok = true;
    WsItem w{0, 0};
    for (int it = it0; it < it1 && ok; it += step) {
      w = ws_find(ipre, cnt, it, w.q, lane);
      if (lane == 0) {
        const int T = slots[w.q].T;
        const uint8_t *sl0 = a.slices + slots[w.q].sli;
        const uint8_t *ra = sl0 + oz_pair_off(T, ws_pair(j, w.r), 0);
        const uint8_t *rb = sl0 + oz_tile_off(w.r == 0 ? j + 1 : j, 0);
        for (int hh = 0; hh < nh; ++hh, ++hc) {
          const int st = hc % kWsStages, u = hc / kWsStages;
          if (hc >= kWsStages &&
              !mbar_wait_pipe(&bar->empty[st], uint32_t((u - 1) & 1), a.wait_limit, abort_flag)) {
            *abort_flag = 1;
            break;
          }
          uint8_t *sA = smb + st * kWsStage;
          mbar_expect_tx(&bar->full[st], uint32_t(kWsHalfA + kWsHalf));
          bulk_g2s(sA, ra + int64_t(hh) * kWsHalfA, kWsHalfA, &bar->full[st]);
          bulk_g2s(sA + kWsHalfA, rb + int64_t(hh) * kWsHalf, kWsHalf, &bar->full[st]);
        }
        ok = !*abort_flag;
      }
      ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
    }
    // Drain: only the latest use of each stage can still be in flight.
    if (lane == 0)
      for (int st = 0; st < kWsStages && st < hc; ++st) {
        const int last = st + kWsStages * ((hc - 1 - st) / kWsStages);
        if (!mbar_wait(&bar->full[st], uint32_t((last / kWsStages) & 1), kOzDrainLimit))
          *abort_flag = 1;
      }
  } else if (warp == 1) {
    if (lane == 0) {
      // MMA issue.
      int hc = 0, k = 0;
      bool ok = true;
      for (int it = it0; it < it1 && ok; it += step, ++k) {
        // The accumulator is free once the epilogue drained the previous item.
        if (k > 0 && !mbar_wait_pipe(&bar->acc_empty, uint32_t((k - 1) & 1), a.wait_limit,
                                     abort_flag)) {
          ok = false;
          break;
        }
        tc_fence_after();
        for (int hh = 0; hh < nh; ++hh, ++hc) {
          const int st = hc % kWsStages, u = hc / kWsStages;
          if (!mbar_wait_pipe(&bar->full[st], uint32_t(u & 1), a.wait_limit, abort_flag)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t sA = saddr(smb + st * kWsStage);
          ws_mma_half(tmem, sA, sA + kWsHalfA, hh == 0);
          umma_commit(&bar->empty[st]);
        }
        if (!ok) break;
        umma_commit(&bar->acc_full);
      }
      if (!ok) *abort_flag = 1;
      umma_commit(&bar->done);  // arrives once every MMA issued above has completed
    }
  } else {
    // Epilogue: 16 warps, etid 0..511.
    const int etid = tid - 64, ew = warp - 2;
    const int qd = warp & 3, h4 = ew >> 2;
    double *sC = reinterpret_cast<double *>(smb + kWsCOff);
    double *sX = reinterpret_cast<double *>(smb + kWsXOff);
    double4 *pts = reinterpret_cast<double4 *>(smb + kWsPtsOff);  // 2 x kWsPts
    double *ysh = reinterpret_cast<double *>(smb + kWsRedOff);    // TB x kMaxF
    double *rsh = ysh + TB * kMaxF;                               // r_i, kWsRows x kMaxF
    double *sUi = reinterpret_cast<double *>(smb + kWsUiOff);     // [b][k][c] = U_bb^-1[k][c]
                                                                  // (row stride kUiLd)
    volatile int *ep_stop = &bar->ep_stop;  // written by epilogue threads only
    if (etid == 0) *ep_stop = 0;
    // The step may be launched while the previous launch (k_diag_next of
    // step j - 1, which writes U_j, X_j and y_j and reads dpart) still runs:
    // the copy and MMA warps need only the slices of earlier steps, which
    // the launch before that wrote, but the epilogue waits for it here.
    asm volatile("griddepcontrol.wait;\n" ::: "memory");
    int xq = -1;  // slot whose U_j (factor of the diagonal tile, transposed) is in sX
    int k = 0;
    WsItem nw{0, 0};  // the next item, whose points are prefetched
    int nidx = -1;    // membership index of this thread's point of it
    auto next_index = [&](int it) {
      nw = ws_find(ipre, cnt, it, nw.q, lane);
      if (etid < kWsPts)
        nidx = ws_point_index(a, slots[nw.q], ws_pair(j, nw.r), nw.r ? j : j + 1, etid);
    };
    if (it0 < it1) {
      next_index(it0);
      if (etid < kWsPts) ws_point_copy(a, pts, etid, nidx);
    }
    cp_async_commit();
    for (int it = it0; it < it1; it += step, ++k) {
      const WsItem w = nw;
      const BigSlot &sl = slots[w.q];
      const int ld = sl.ld, F = a.F;
      double *W = a.W + sl.base;
      double *rcol = W + int64_t(sl.T) * TB;
      const bool diag = w.r == 0;
      const int u = ws_pair(j, w.r);
      // The halves of the pair that the item needs: [h0, h1).
      const int h0 = diag ? (j + 1) & 1 : (2 * u > j ? 0 : 1);
      const int h1 = diag ? h0 + 1 : (2 * u + 1 < sl.T ? 2 : 1);
      const int rows0 = TB * h0, rows1 = TB * h1;
      // The item's points have landed, and every warp is done with the
      // previous item's C, factor and residual rows.
      cp_async_wait<0>();
      ws_sync();
      if (!diag) {
        // U_j (and its block inverses) and y_j once per slot, the
        // residual rows r_i of every item: copied while the tiles are made.
        if (xq != w.q) {
          load_factor_async(sX, W + int64_t(j) * TB * ld + int64_t(j) * TB, ld, etid, kWsEpi);
          // U_bb^-1 = (X_j's diagonal block b)^T, X_j = L_jj^-1 row-major.
          const double *xg = a.inv + sl.inv + int64_t(j) * TB * TB;
          for (int e = etid; e < 4 * 256; e += kWsEpi) {
            const int b = e >> 8, kk = (e >> 4) & 15, c = e & 15;
            cp_async8(sUi + (16 * b + kk) * kUiLd + c, xg + (16 * b + c) * TB + 16 * b + kk);
          }
          const double *yg = rcol + int64_t(j) * TB * ld;
          for (int e = etid; e < TB * F; e += kWsEpi)
            cp_async8(ysh + (e / F) * kMaxF + e % F, yg + int64_t(e / F) * ld + e % F);
          xq = w.q;
        }
        const double *rg = rcol + int64_t(2 * u) * TB * ld;
        for (int e = rows0 * F + etid; e < rows1 * F; e += kWsEpi)
          cp_async8(rsh + (e / F) * kMaxF + e % F, rg + int64_t(e / F) * ld + e % F);
      }
      cp_async_commit();
      // The next item's membership index, loaded while this one runs.
      if (it + step < it1) next_index(it + step);
      // A[i, j] (or A[j+1, j+1]) while the MMAs of this item run.
      ws_gen_rows(a, sl, u, diag ? j + 1 : j, h0, h1, sC, pts + (k & 1) * kWsPts, etid);
      // Drain the accumulator, then hand it back to the MMA thread.
      // Every epilogue thread waits; the decision to stop is made uniform
      // through ep_stop (the global abort flag may change at any time).
      if (!mbar_wait_pipe(&bar->acc_full, uint32_t(k & 1), a.wait_limit, abort_flag)) *ep_stop = 1;
      ws_sync();
      if (*ep_stop) {
        *abort_flag = 1;
        break;
      }
      tc_fence_after();
      // C = A - sigma^2 (level sums).  At j = 0 there are no products (no
      // MMAs were issued) and C = A.
      if (j > 0 && (qd >> 1) >= h0 && (qd >> 1) < h1) ws_drain(tmem, qd, h4, sC, a.oz_sig2, lane);
      tc_fence_before();
      __syncwarp();
      auto release = [&] {
        if (lane == 0) mbar_arrive_cnt(&bar->acc_empty, 1);
      };
      cp_async_wait<0>();  // the factor and the residual rows
      ws_sync();
      if (it + step < it1 && etid < kWsPts)
        ws_point_copy(a, pts + ((k + 1) & 1) * kWsPts, etid, nidx);
      cp_async_commit();
      const int r0 = 8 * ew;
      const bool mine = !diag && r0 >= rows0 && r0 < rows1;
      const bool late = mine && j < kWsLate;
      if (!late) release();
      if (diag) {
        // D' to dpart, where the next launch (k_diag_next) factors D.
        double *dst = a.dpart + int64_t(sl.q) * TB * TB;
        for (int e = etid; e < TB * TB; e += kWsEpi)
          dst[e] = sC[(rows0 + (e >> 6)) * LDS + (e & 63)];
        continue;
      }
      // Warp ew's rows 8 ew .. + 7: L[i, j] U_j = C by blocked row solves, then
      // from the registers the store, the forward substitution and the int8
      // slices.
      if (!mine) continue;
      double c[8][2];
      warp_rows_solve8<false>(sC + r0 * LDS, sX, sUi, lane, c);
      if (late) release();
      const int row = r0 + (lane >> 2), t2 = 2 * (lane & 3);
      double *Lg = W + (int64_t(2 * u) * TB + row) * ld + int64_t(j) * TB + t2;
#pragma unroll
      for (int nt = 0; nt < 8; ++nt)
        *reinterpret_cast<double2 *>(Lg + 8 * nt) = make_double2(c[nt][0], c[nt][1]);
      double *rg = rcol + (int64_t(2 * u) * TB + row) * ld;
      for (int f = 0; f < F; ++f) {
        double sum = 0.0;
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) {
          sum = __fma_rn(c[nt][0], ysh[(8 * nt + t2) * kMaxF + f], sum);
          sum = __fma_rn(c[nt][1], ysh[(8 * nt + t2 + 1) * kMaxF + f], sum);
        }
        sum += __shfl_xor_sync(0xffffffffu, sum, 1);
        sum += __shfl_xor_sync(0xffffffffu, sum, 2);
        if (t2 == 0) rg[f] = rsh[row * kMaxF + f] - sum;
      }
      slice_rows_acc(c, r0 & 63, lane, a.oz_mul, a.slices + sl.sli, sl.T, 2 * u + (r0 >> 6), j);
    }
    cp_async_wait<0>();
  }
  __syncthreads();
  if (!mbar_wait(&bar->done, 0u, kOzDrainLimit)) *abort_flag = 1;
  tc_fence_after();
  __syncthreads();
  // After a time-out, the patches of every item of this CTA's range are
  // marked for the FP64 LU.
  if (*abort_flag)
    for (int it = it0 + tid * step; it < it1; it += kWsThreads * step)
      atomicOr(&a.status[slots[ws_item(ipre, cnt, it).q].k], 8);
  tc_fence_before();
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem),
                 "r"(kOzTmemCols)
                 : "memory");
}

// Backward sweep L^T z = y of one slot (CTA per slot), tile row by tile row
// from the last: z_s = X_s^T (y_s - sum_{t>s} L[t, s]^T z_t), with the tile
// inverses X_s of the factorisation.  The sweep is a chain of T dependent
// levels, so the time of a large slot is set by how fast its tiles reach the
// SM: warp 8 streams them with 16-byte cp.async (one 512-byte row per
// instruction, completion counted on an mbarrier), in sweep order and
// independent of z, through a ring of kBkStages 32 KB stages (the tiles
// L[t, s], t > s, then X_s), up to kBkStages tiles ahead of the arithmetic.
// (Bulk copies of the 512-byte rows were slower: the per-request cost of the
// bulk-copy engine capped one SM near 20 GB/s.)  Warps 0..7 take the L tiles of a
// level in turn (lane: two columns r of the tile, all rows c), then meet to
// finish z_s.  z goes to zc (per slot) and, in the forward, to alpha_c per
// (patch, source).  Every wait is bounded; a time-out marks the patch
// (status 8), the CTA keeps its barrier sequence, stops issuing copies and
// waits for the copies it issued before it returns.
//
// A slot of many tile rows is swept by a thread-block cluster of C CTAs (C = 1:
// one CTA).  Level l solves block l of the sweep; rank r of the cluster holds
// the solved blocks p = r (mod C): in every level it multiplies its own tiles
// by its own blocks and sends the 64 x F partial sums to the level's solver,
// rank l mod C, through distributed shared memory (an mbarrier there counts
// the senders' warps).  The solver adds them in rank order and finishes the
// block, which only it needs again.  A rank's partial of level l + C contains
// a block solved after level l was consumed, so one receive buffer per rank
// suffices.
constexpr int kBkTile = TB * TB * 8;  // bytes of one stage
// Ring depth: 3 stages for one or two fields, two CTAs per SM (the many short
// slots are latency-bound, and a second CTA hides it); 5 stages, one CTA per
// SM, for more fields (registers).
constexpr int bk_stages(int F) { return F <= 2 ? 3 : 5; }

// Cluster size for the slots with at least kBkLong tile rows, whose sweep one
// SM's copy rate would draw out (15-30 GB/s: 5.8 ms for the slot group with T =
// 78); its ring has four stages for eight fields (the receive buffer's room).
// The line: a cluster's level costs about 4 us whatever its few tiles, so short
// slots are faster one to an SM.  A kept-factor call at 400k refined points
// takes 5.9, 5.0, 4.7, 5.1, 5.6, 5.5 ms with the line at 12, 24, 32, 40, 56 and
// without clusters; the two sweep launches of a slot group at 1M 2.1 instead of
// 4.5-5.8 ms.
constexpr int kBkCluster = 8;
constexpr int kBkLong = 32;
constexpr int bk_cluster_stages(int F) { return F <= 2 ? 3 : 4; }

size_t chol_back_smem(int F, int S = 0, int C = 1) {
  // stages, part, accs, receive buffer, full/empty barriers, the receive
  // barrier, abort flag and issue counter
  if (S == 0) S = bk_stages(F);
  return size_t(S) * kBkTile + size_t(8 * TB * F + TB * F + (C > 1 ? C * TB * F : 0)) * 8 +
         2 * S * 8 + 8 + 16;
}
// The deep ring of the one-field backward sweep (one CTA per SM, twice the
// tiles in flight): a slot's sweep streams its T (T - 1) / 2 tiles through
// one SM, so the largest slots' sweeps are set by the bytes one SM keeps in
// flight (PACMAN_B200_BACK_STAGES = 6 selects it).
constexpr int kBkDeep = 6;


// Bounded wait for a phase that gives up early once the CTA has aborted.
__device__ __forceinline__ bool mbar_wait_abort(uint64_t *b, uint32_t parity,
                                                volatile int *abort_flag) {
  return mbar_wait_pipe(b, parity, kOzWaitLimit, abort_flag);
}

// One 64 x 64 FP64 tile (rows ld doubles apart) into a pipeline stage by the
// 32 lanes of a warp, 16-byte cp.async each (row r: the lane's 16 bytes, so
// every instruction moves one 512-byte row); the stage's full barrier
// (initialised to 32 arrivals) counts this lane once its copies have landed.
__device__ __forceinline__ void warp_tile_g2s(double *dst, const double *src, int64_t ld,
                                              int lane, uint64_t *full) {
#pragma unroll 8
  for (int r = 0; r < TB; ++r) cp_async16(dst + r * TB + 2 * lane, src + r * ld + 2 * lane);
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];\n" ::"r"(saddr(full))
               : "memory");
}

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;\n" ::
                   : "memory");
}
// The address of this CTA's shared variable p in CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t cluster_addr(const void *p, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(r) : "r"(saddr(p)), "r"(rank));
  return r;
}
__device__ __forceinline__ void cluster_store(uint32_t addr, double v) {
  asm volatile("st.shared::cluster.f64 [%0], %1;\n" ::"r"(addr), "d"(v) : "memory");
}
__device__ __forceinline__ void cluster_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];\n" ::"r"(bar)
               : "memory");
}
// Bounded wait for the partial sums of all ranks.
__device__ __forceinline__ bool cluster_wait(uint64_t *b, uint32_t parity,
                                             volatile int *abort_flag) {
  for (int it = 0; it < kOzWaitLimit; ++it) {
    uint32_t done;
    asm volatile(
        "{\n.reg .pred p;\nmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(saddr(b)), "r"(parity)
        : "memory");
    if (done) return true;
    if (*abort_flag) return false;
  }
  return false;
}

// Bounded wait until item x is issued, then for its data.
template <int kBkStages>
__device__ __forceinline__ bool bk_wait_item(volatile int *issued, volatile int *abort_flag,
                                             uint64_t *full, int x) {
  bool ok = false;
  for (int it = 0; it < kOzWaitLimit && !ok; ++it) {
    ok = *issued > x;
    if (*abort_flag) return false;
  }
  return ok && mbar_wait_abort(&full[x % kBkStages], uint32_t((x / kBkStages) & 1), abort_flag);
}

template <int KF, int kBkStages, int C = 1>  // fields in registers (F <= KF), ring depth, cluster
__global__ void __launch_bounds__(288, kBkStages == 3 ? 2 : 1)
    k_chol_back(BigArgs a, const BigSlot *__restrict__ slots) {
  extern __shared__ __align__(128) uint8_t smem[];
  const BigSlot sl = slots[blockIdx.x / C];
  const int rank = C > 1 ? int(cluster_rank()) : 0;
  const int F = a.F, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double *stage0 = reinterpret_cast<double *>(smem);
  double *part = reinterpret_cast<double *>(smem + size_t(kBkStages) * kBkTile);  // [8][TB][F]
  double *accs = part + 8 * TB * F;                                                // [TB][F]
  double *recv = accs + TB * F;                                                    // [C][TB][F]
  uint64_t *full = reinterpret_cast<uint64_t *>(recv + (C > 1 ? C * TB * F : 0));
  uint64_t *empty = full + kBkStages;
  uint64_t *got = empty + kBkStages;
  volatile int *abort_flag = reinterpret_cast<volatile int *>(got + 1);
  // Items the producer has issued.  A consumer waits on the full barrier of
  // item x only once x is issued: x - kBkStages, the previous item of that
  // stage, has then landed and been released, so the barrier is in the
  // phase of x and the parity wait cannot match an older phase.
  volatile int *issued = abort_flag + 1;
  const int ld = sl.ld, T = sl.T;
  const double *W = a.W + sl.base;
  const double *rcol = W + int64_t(T) * TB;
  const double *X0 = a.inv + sl.inv;
  double *zc = a.zc + sl.zoff;
  if (tid == 0) {
    for (int i = 0; i < kBkStages; ++i) {
      mbar_init(&full[i], 32);  // one arrival per producer lane
      mbar_init(&empty[i], 8);
    }
    mbar_init(got, 8 * C);
    *abort_flag = 0;
    *issued = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  __syncthreads();
  if (C > 1) cluster_sync_all();  // every rank's barriers are ready
  if (warp == 8) {
    // Producer: item g of the stream goes to stage g % kBkStages.
    int g = 0;
    bool ok = true;
    for (int l = 0; l < T && ok; ++l) {
      const int s = T - 1 - l, nq = l > rank ? (l - 1 - rank) / C + 1 : 0;
      for (int q = 0; q < nq + (l % C == rank ? 1 : 0) && ok; ++q, ++g) {  // q == nq: X_s
        const int st = g % kBkStages, u = g / kBkStages;
        if (g >= kBkStages) {
          if (lane == 0) ok = mbar_wait_abort(&empty[st], uint32_t((u - 1) & 1), abort_flag);
          ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
          if (!ok) break;
        }
        double *dst = reinterpret_cast<double *>(smem + size_t(st) * kBkTile);
        const int t = T - 1 - (rank + C * q);
        if (q < nq)
          warp_tile_g2s(dst, W + int64_t(t) * TB * ld + int64_t(s) * TB, ld, lane, &full[st]);
        else
          warp_tile_g2s(dst, X0 + int64_t(s) * TB * TB, TB, lane, &full[st]);
        __syncwarp();
        if (lane == 0) {
          __threadfence_block();
          *issued = g + 1;
        }
      }
    }
    if (!ok && lane == 0) {
      *abort_flag = 1;
      atomicOr(&a.status[sl.k], 8);
    }
    // Wait (bounded) for every issued copy: the latest item of each stage.
    if (lane == 0)
      for (int st = 0; st < kBkStages && st < g; ++st) {
        const int last = st + kBkStages * ((g - 1 - st) / kBkStages);
        mbar_wait(&full[st], uint32_t((last / kBkStages) & 1));
      }
    asm volatile("cp.async.wait_all;\n" ::: "memory");
  } else {
    int g = 0;
    const int rr = tid & 63, quarter = tid >> 6;
    for (int l = 0; l < T; ++l) {
      const int s = T - 1 - l;
      const int nt = l > rank ? (l - 1 - rank) / C + 1 : 0;  // this rank's tiles of the level
      // Block t of the rank's q-th tile.
      auto block_of = [&](int q) { return T - 1 - (rank + C * q); };
      double acc0[KF], acc1[KF];
#pragma unroll
      for (int f = 0; f < KF; ++f) acc0[f] = acc1[f] = 0.0;
      // z_t of the warp's next tile, one coalesced load per lane and field
      // (rows lane and lane + 32), issued before the wait for the tile; the
      // rows c are then broadcast from the lanes by shuffles.
      double zn0[KF], zn1[KF];
      if (warp < nt) {
        const double *zt = zc + int64_t(block_of(warp)) * TB * F;
#pragma unroll
        for (int f = 0; f < KF; ++f) {
          zn0[f] = f < F ? zt[lane * F + f] : 0.0;
          zn1[f] = f < F ? zt[(lane + 32) * F + f] : 0.0;
        }
      }
      for (int k = warp; k < nt; k += 8) {
        const int gi = g + k, st = gi % kBkStages;
        double z0[KF], z1[KF];
#pragma unroll
        for (int f = 0; f < KF; ++f) {
          z0[f] = zn0[f];
          z1[f] = zn1[f];
        }
        if (k + 8 < nt) {
          const double *zt = zc + int64_t(block_of(k + 8)) * TB * F;
#pragma unroll
          for (int f = 0; f < KF; ++f)
            if (f < F) {
              zn0[f] = zt[lane * F + f];
              zn1[f] = zt[(lane + 32) * F + f];
            }
        }
        bool ok = !*abort_flag;
        if (ok) ok = bk_wait_item<kBkStages>(issued, abort_flag, full, gi);
        if (!ok) {
          *abort_flag = 1;
          continue;
        }
        const double *tile = stage0 + size_t(st) * TB * TB;
#pragma unroll 8
        for (int c = 0; c < TB; ++c) {
          const double l0 = tile[c * TB + lane], l1 = tile[c * TB + lane + 32];
#pragma unroll
          for (int f = 0; f < KF; ++f)
            if (f < F) {
              const double z = __shfl_sync(0xffffffffu, c < 32 ? z0[f] : z1[f], c & 31);
              acc0[f] = __fma_rn(l0, z, acc0[f]);
              acc1[f] = __fma_rn(l1, z, acc1[f]);
            }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive_cnt(&empty[st], 8);
      }
      g += nt;
#pragma unroll
      for (int f = 0; f < KF; ++f)
        if (f < F) {
          part[(warp * TB + lane) * F + f] = acc0[f];
          part[(warp * TB + lane + 32) * F + f] = acc1[f];
        }
      asm volatile("bar.sync 1, 256;\n" ::: "memory");
      for (int e = tid; e < TB * F; e += 256) {
        const int r = e / F, f = e % F;
        double sum = 0.0;
#pragma unroll
        for (int w = 0; w < 8; ++w) sum += part[(w * TB + r) * F + f];
        if (C == 1) accs[r * F + f] = rcol[int64_t(s * TB + r) * ld + f] - sum;
        else cluster_store(cluster_addr(recv + rank * TB * F + e, l % C), sum);
      }
      if (C > 1) {
        __syncwarp();
        if (lane == 0) cluster_arrive(cluster_addr(got, l % C));
        if (l % C != rank) {
          // part is written again in the next level.
          asm volatile("bar.sync 1, 256;\n" ::: "memory");
          continue;
        }
        if (!cluster_wait(got, uint32_t((l / C) & 1), abort_flag)) *abort_flag = 1;
        for (int e = tid; e < TB * F; e += 256) {
          const int r = e / F, f = e % F;
          double sum = 0.0;
#pragma unroll
          for (int c = 0; c < C; ++c) sum += recv[c * TB * F + e];
          accs[e] = rcol[int64_t(s * TB + r) * ld + f] - sum;
        }
      }
      // X_s: every consumer warp reads it, each releases one of 8 arrivals.
      const int st = g % kBkStages;
      bool okx = !*abort_flag;
      if (okx) okx = bk_wait_item<kBkStages>(issued, abort_flag, full, g);
      if (!okx) *abort_flag = 1;
      asm volatile("bar.sync 1, 256;\n" ::: "memory");
      // z_s[rr][f] = sum_{c >= rr} X_s[c][rr] acc_s[c][f]; quarters of c, then summed.
      const double *xs = stage0 + size_t(st) * TB * TB;
      double zp[KF];
#pragma unroll
      for (int f = 0; f < KF; ++f) zp[f] = 0.0;
      if (okx) {
#pragma unroll 4
        for (int c = quarter; c < TB; c += 4) {
          if (c < rr) continue;
          const double x = xs[c * TB + rr];
#pragma unroll
          for (int f = 0; f < KF; ++f)
            if (f < F) zp[f] = __fma_rn(x, accs[c * F + f], zp[f]);
        }
      }
      __syncwarp();
      if (lane == 0 && okx) mbar_arrive_cnt(&empty[st], 1);
      g += 1;
#pragma unroll
      for (int f = 0; f < KF; ++f)
        if (f < F) part[(quarter * TB + rr) * F + f] = zp[f];
      asm volatile("bar.sync 1, 256;\n" ::: "memory");
      for (int e = tid; e < TB * F; e += 256) {
        const int r = e / F, f = e % F;
        const double z = part[(0 * TB + r) * F + f] + part[(1 * TB + r) * F + f] +
                         part[(2 * TB + r) * F + f] + part[(3 * TB + r) * F + f];
        const int j = s * TB + r;
        zc[int64_t(j) * F + f] = z;
        if (a.alpha_c != nullptr && j < sl.n) a.alpha_c[(a.soff[sl.k] + j) * F + f] = z;
      }
      asm volatile("bar.sync 1, 256;\n" ::: "memory");
    }
    if (tid == 0 && *abort_flag) atomicOr(&a.status[sl.k], 8);
  }
  __syncthreads();
  if (C > 1) cluster_sync_all();  // no rank leaves while others write to it
}

// Forward sweep L y = r of one slot from kept factors (CTA per slot), for
// an execute that reuses the factorisation: y_s = X_s (r_s - sum_{t<s}
// L[s, t] y_t), tile row by tile row from the first, with the tile inverses
// X_s of the factorisation.  r is the residual column (first F columns of
// column tile T) and is overwritten with y, as the factorising steps leave
// it.  Warp 8 streams the tiles L[s, t], t < s, then X_s, through the same
// cp.async ring as k_chol_back; every consumer warp reads
// every tile: warp w owns rows 8w .. 8w + 7 and its lanes the columns c and
// c + 32, so the partial sums stay in registers until the level ends.
template <int KF, int kBkStages, int C = 1>  // fields in registers (F <= KF), ring depth, cluster
__global__ void __launch_bounds__(288, kBkStages == 3 ? 2 : 1)
    k_chol_fwd(BigArgs a, const BigSlot *__restrict__ slots) {
  extern __shared__ __align__(128) uint8_t smem[];
  const BigSlot sl = slots[blockIdx.x / C];
  const int rank = C > 1 ? int(cluster_rank()) : 0;
  const int F = a.F, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double *stage0 = reinterpret_cast<double *>(smem);
  double *accs = reinterpret_cast<double *>(smem + size_t(kBkStages) * kBkTile);  // [TB][F]
  double *recv = accs + TB * F;                                                    // [C][TB][F]
  uint64_t *full = reinterpret_cast<uint64_t *>(recv + (C > 1 ? C * TB * F : 0));
  uint64_t *empty = full + kBkStages;
  uint64_t *got = empty + kBkStages;
  volatile int *abort_flag = reinterpret_cast<volatile int *>(got + 1);
  volatile int *issued = abort_flag + 1;  // as in k_chol_back
  const int ld = sl.ld, T = sl.T;
  const double *W = a.W + sl.base;
  double *rcol = a.W + sl.base + int64_t(T) * TB;
  const double *X0 = a.inv + sl.inv;
  if (tid == 0) {
    for (int i = 0; i < kBkStages; ++i) {
      mbar_init(&full[i], 32);  // one arrival per producer lane
      mbar_init(&empty[i], 8);
    }
    mbar_init(got, 8 * C);
    *abort_flag = 0;
    *issued = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  __syncthreads();
  if (C > 1) cluster_sync_all();  // every rank's barriers are ready
  if (warp == 8) {
    int g = 0;
    bool ok = true;
    for (int s = 0; s < T && ok; ++s) {
      const int nq = s > rank ? (s - 1 - rank) / C + 1 : 0;
      for (int q = 0; q < nq + (s % C == rank ? 1 : 0) && ok; ++q, ++g) {  // q == nq: X_s
        const int t = rank + C * q;
        const int st = g % kBkStages, u = g / kBkStages;
        if (g >= kBkStages) {
          if (lane == 0) ok = mbar_wait_abort(&empty[st], uint32_t((u - 1) & 1), abort_flag);
          ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
          if (!ok) break;
        }
        double *dst = reinterpret_cast<double *>(smem + size_t(st) * kBkTile);
        if (q < nq)
          warp_tile_g2s(dst, W + int64_t(s) * TB * ld + int64_t(t) * TB, ld, lane, &full[st]);
        else
          warp_tile_g2s(dst, X0 + int64_t(s) * TB * TB, TB, lane, &full[st]);
        __syncwarp();
        if (lane == 0) {
          __threadfence_block();
          *issued = g + 1;
        }
      }
    }
    if (!ok && lane == 0) {
      *abort_flag = 1;
      atomicOr(&a.status[sl.k], 8);
    }
    if (lane == 0)
      for (int st = 0; st < kBkStages && st < g; ++st) {
        const int last = st + kBkStages * ((g - 1 - st) / kBkStages);
        mbar_wait(&full[st], uint32_t((last / kBkStages) & 1));
      }
    asm volatile("cp.async.wait_all;\n" ::: "memory");
  } else {
    int g = 0;
    const int r0 = 8 * warp;
    for (int s = 0; s < T; ++s) {
      double part[8][KF];
#pragma unroll
      for (int r = 0; r < 8; ++r)
#pragma unroll
        for (int f = 0; f < KF; ++f) part[r][f] = 0.0;
      // y_t of the lane's columns, loaded one tile ahead of its use.
      double yn0[KF], yn1[KF];
#pragma unroll
      for (int f = 0; f < KF; ++f) {
        const double *y0 = rcol + int64_t(rank) * TB * ld;
        yn0[f] = (rank < s && f < F) ? y0[int64_t(lane) * ld + f] : 0.0;
        yn1[f] = (rank < s && f < F) ? y0[int64_t(lane + 32) * ld + f] : 0.0;
      }
      for (int t = rank; t < s; t += C, ++g) {
        double y0[KF], y1[KF];
#pragma unroll
        for (int f = 0; f < KF; ++f) {
          y0[f] = yn0[f];
          y1[f] = yn1[f];
        }
        if (t + C < s) {
          const double *yt = rcol + int64_t(t + C) * TB * ld;
#pragma unroll
          for (int f = 0; f < KF; ++f)
            if (f < F) {
              yn0[f] = yt[int64_t(lane) * ld + f];
              yn1[f] = yt[int64_t(lane + 32) * ld + f];
            }
        }
        bool ok = !*abort_flag;
        if (ok) ok = bk_wait_item<kBkStages>(issued, abort_flag, full, g);
        if (!ok) {
          *abort_flag = 1;
          continue;
        }
        const double *tile = stage0 + size_t(g % kBkStages) * TB * TB;
#pragma unroll
        for (int r = 0; r < 8; ++r) {
          const double l0 = tile[(r0 + r) * TB + lane], l1 = tile[(r0 + r) * TB + lane + 32];
#pragma unroll
          for (int f = 0; f < KF; ++f)
            if (f < F) part[r][f] = __fma_rn(l1, y1[f], __fma_rn(l0, y0[f], part[r][f]));
        }
        __syncwarp();
        if (lane == 0) mbar_arrive_cnt(&empty[g % kBkStages], 1);
      }
      // acc_s = r_s - sum over the level, rows of this warp.
#pragma unroll
      for (int r = 0; r < 8; ++r)
#pragma unroll
        for (int f = 0; f < KF; ++f)
          if (f < F) {
            double v = part[r][f];
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (lane != 0) continue;
            if (C == 1) accs[(r0 + r) * F + f] = rcol[int64_t(s * TB + r0 + r) * ld + f] - v;
            else cluster_store(cluster_addr(recv + rank * TB * F + (r0 + r) * F + f, s % C), v);
          }
      if (C > 1) {
        if (lane == 0) cluster_arrive(cluster_addr(got, s % C));
        if (s % C != rank) continue;
        if (!cluster_wait(got, uint32_t((s / C) & 1), abort_flag)) *abort_flag = 1;
        for (int e = lane; e < 8 * F; e += 32) {  // the warp's rows
          const int r = r0 + e / F, f = e % F;
          double sum = 0.0;
#pragma unroll
          for (int c = 0; c < C; ++c) sum += recv[c * TB * F + r * F + f];
          accs[r * F + f] = rcol[int64_t(s * TB + r) * ld + f] - sum;
        }
      }
      bool okx = !*abort_flag;
      if (okx) okx = bk_wait_item<kBkStages>(issued, abort_flag, full, g);
      if (!okx) *abort_flag = 1;
      asm volatile("bar.sync 1, 256;\n" ::: "memory");
      // y_s[rr] = sum_{c <= rr} X_s[rr][c] acc_s[c], rows rr of this warp.
      if (okx) {
        const double *xs = stage0 + size_t(g % kBkStages) * TB * TB;
#pragma unroll
        for (int r = 0; r < 8; ++r) {
          const int rr = r0 + r;
          const double x0 = lane <= rr ? xs[rr * TB + lane] : 0.0;
          const double x1 = lane + 32 <= rr ? xs[rr * TB + lane + 32] : 0.0;
#pragma unroll
          for (int f = 0; f < KF; ++f)
            if (f < F) {
              double v = __fma_rn(x1, accs[(lane + 32) * F + f], x0 * accs[lane * F + f]);
              for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
              if (lane == 0) rcol[int64_t(s * TB + rr) * ld + f] = v;
            }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive_cnt(&empty[g % kBkStages], 1);
      }
      g += 1;
      asm volatile("bar.sync 1, 256;\n" ::: "memory");
    }
    if (tid == 0 && *abort_flag) atomicOr(&a.status[sl.k], 8);
  }
  __syncthreads();
  if (C > 1) cluster_sync_all();  // no rank leaves while others write to it
}

size_t chol_fwd_smem(int F, int S = 0, int C = 1) {
  // as chol_back_smem without part
  if (S == 0) S = bk_stages(F);
  return size_t(S) * kBkTile + size_t(TB * F + (C > 1 ? C * TB * F : 0)) * 8 + 2 * S * 8 + 8 + 16;
}

// local = E alpha + V beta for the targets of one slot, 32 at a time: a target
// per lane, the sources (and their coefficients) staged in shared memory and
// split between the block's four warps, whose sums are added in warp order.
// Bound by the FP64 pipe (about 26 operations per pair and one per field).
// Shell 1M, 8 fields: 1.05 ms per slot group, 1M refined points, 1 field: 0.28
// ms; a warp per target with lanes over the sources gathered every source
// again for every target and took 5 shuffle steps per field: 7.8 and 2.2 ms.
constexpr int kEvThreads = 128;
constexpr int kEvChunk = 128;  // sources staged at a time
template <int KF>
__global__ void __launch_bounds__(kEvThreads)
    k_chol_eval(BigArgs a, const BigSlot *__restrict__ slots) {
  constexpr int REC = (3 + KF + 1) / 2 * 2;  // x, y, z, alpha_f: 16-byte records
  __shared__ __align__(16) double rec[kEvChunk * REC];
  __shared__ double red[4][KF][32];
  const BigSlot &sl = slots[blockIdx.x];
  const int F = a.F, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int n = sl.n, m = sl.m;
  const int64_t s0 = a.soff[sl.k], t0 = a.toff[sl.k];
  const double *beta = a.beta + sl.q * 4 * kMaxF;
  const int *act = a.act + sl.q * 3;
  int bad = 0;
  for (int i0 = 32 * blockIdx.y; i0 < m; i0 += 32 * gridDim.y) {
    const int i = i0 + lane;
    const double4 y = a.tgt[a.tidx[t0 + (i < m ? i : i0)]];
    double acc[KF], odd[KF];
#pragma unroll
    for (int f = 0; f < KF; ++f) acc[f] = odd[f] = 0.0;
    for (int j0 = 0; j0 < n; j0 += kEvChunk) {
      const int cnt = min(kEvChunk, n - j0);
      __syncthreads();
      if (threadIdx.x < cnt) {
        const int64_t e = s0 + j0 + threadIdx.x;
        const double4 x = a.src[a.sidx[e]];
        double *r = rec + threadIdx.x * REC;
        r[0] = x.x;
        r[1] = x.y;
        r[2] = x.z;
#pragma unroll
        for (int f = 0; f < KF; ++f) r[3 + f] = f < F ? a.alpha_c[e * F + f] : 0.0;
      }
      __syncthreads();
      with_basis(a.basis, [&](auto B) {
        auto at = [&](int jj, double *sum) {
          double r[REC];
#pragma unroll
          for (int v = 0; v < REC; v += 2)
            *reinterpret_cast<double2 *>(r + v) =
                *reinterpret_cast<const double2 *>(rec + jj * REC + v);
          const double ph = phi_at<B>(sqdist3(y.x, y.y, y.z, r[0], r[1], r[2]), a.rinv);
#pragma unroll
          for (int f = 0; f < KF; ++f) sum[f] = __fma_rn(ph, r[3 + f], sum[f]);
        };
        int jj = warp;
        for (; jj + 4 < cnt; jj += 8) {
          at(jj, acc);
          at(jj + 4, odd);
        }
        if (jj < cnt) at(jj, acc);
      });
    }
#pragma unroll
    for (int f = 0; f < KF; ++f) red[warp][f][lane] = acc[f] + odd[f];
    __syncthreads();
    // Warp w finishes the fields w, w + 4.
    if (i < m)
      for (int f = warp; f < F; f += 4) {
        const double sum = ((red[0][f][lane] + red[1][f][lane]) + red[2][f][lane]) + red[3][f][lane];
        const double yc[3] = {y.x, y.y, y.z};
        double v = beta[4 * f];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          const int ax = act[d];
          if (ax >= 0)
            v = __fma_rn(ax == 0 ? yc[0] : (ax == 1 ? yc[1] : yc[2]), beta[4 * f + 1 + d], v);
        }
        const double out = sum + v;
        if (!isfinite(out)) bad = 1;
        a.local[(t0 + i) * F + f] = out;
      }
  }
  if (bad) atomicOr(&a.status[sl.k], 2);
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------

CholPlan chol_prefix(const std::vector<BigSlot> &slots) {
  // Step j serves the slots with T > j + 1 (a prefix: slots are sorted by
  // decreasing T), ceil((T - j - 1) / 2) CTAs each: CTA 0 of every slot first,
  // then the prefix counts of the others.
  CholPlan cp;
  const int ns = int(slots.size());
  const int steps = ns ? std::max(0, slots.front().T - 1) : 0;
  cp.ns = ns;
  cp.cnt.resize(steps);
  cp.off.resize(steps + 1);
  for (int j = 0; j < steps; ++j) {
    int c = 0;
    while (c < ns && slots[c].T > j + 1) ++c;
    cp.cnt[j] = c;
    cp.off[j] = int(cp.pre.size());
    int64_t acc = 0;
    cp.pre.push_back(0);
    for (int q = 0; q < c; ++q) {
      acc += (slots[q].T - j) / 2 - 1;  // CTAs l >= 1
      cp.pre.push_back(int(acc));
    }
    if (acc > 0x7fffffffll) throw Error{PACMAN_B200_ERR_LIMIT, "too many tiles in one launch"};
  }
  cp.off[steps] = int(cp.pre.size());
  // Items of the warp-specialised int8 step: per slot its diagonal item, then
  // the pairs of row tiles that reach below row j.
  cp.ioff.resize(steps);
  for (int j = 0; j < steps; ++j) {
    const int c = cp.cnt[j];
    cp.ioff[j] = int(cp.pre.size());
    int64_t acc = 0;
    cp.pre.push_back(0);
    for (int q = 0; q < c; ++q) {
      acc += 1 + ws_pairs(slots[q].T, j);
      cp.pre.push_back(int(acc));
    }
    if (acc > 0x7fffffffll) throw Error{PACMAN_B200_ERR_LIMIT, "too many tiles in one launch"};
  }
  return cp;
}

static void set_attributes() {
  PB_CUDA(cudaFuncSetAttribute(k_col_step<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               int(kColSmem)));
  PB_CUDA(cudaFuncSetAttribute(k_col_step<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               int(kColSmem)));
  PB_CUDA(cudaFuncSetAttribute(k_col_step_ws, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               int(kWsSmem)));
  PB_CUDA(cudaFuncSetAttribute(k_diag_chol, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               int(kDiagSmem)));
  PB_CUDA(cudaFuncSetAttribute(k_diag_next, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               int(kDiagNextSmem)));
  {
#define PB_SWEEP_ATTR(K, F)                                                                   \
  PB_CUDA(cudaFuncSetAttribute(K<F, bk_stages(F)>, cudaFuncAttributeMaxDynamicSharedMemorySize, \
                               int(std::max(chol_back_smem(F), chol_fwd_smem(F)))));         \
  PB_CUDA(cudaFuncSetAttribute(K<F, bk_cluster_stages(F), kBkCluster>,                          \
                               cudaFuncAttributeMaxDynamicSharedMemorySize,                   \
                               int(chol_back_smem(F, bk_cluster_stages(F), kBkCluster))))
    PB_SWEEP_ATTR(k_chol_back, 1);
    PB_CUDA(cudaFuncSetAttribute(k_chol_back<1, kBkDeep>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 int(chol_back_smem(1, kBkDeep))));
    PB_SWEEP_ATTR(k_chol_back, 2);
    PB_SWEEP_ATTR(k_chol_back, 4);
    PB_SWEEP_ATTR(k_chol_back, kMaxF);
    PB_SWEEP_ATTR(k_chol_fwd, 1);
    PB_SWEEP_ATTR(k_chol_fwd, 2);
    PB_SWEEP_ATTR(k_chol_fwd, 4);
    PB_SWEEP_ATTR(k_chol_fwd, kMaxF);
#undef PB_SWEEP_ATTR
  }
}

void chol_set_smem_attributes() {
  static OncePerDevice once;
  once(set_attributes);
}

void chol_launch_steps(const BigArgs &a, const BigSlot *ds, const std::vector<BigSlot> &hs,
                       const CholPlan &cp, const int *dpre, cudaStream_t st, SolveReport &rep,
                       cudaEvent_t tail_event) {
  if (cp.ns == 0) return;
  k_diag_chol<<<cp.ns, 256, kDiagSmem, st>>>(a, ds, 0);
  note_launch();
  const int steps = int(cp.cnt.size());
  const Tuning &tu = tuning_for_current_device();
  const int sms = tu.sms;
  // First step on the int8 tensor cores: tuned, PACMAN_B200_INT8_FROM overrides.
  const int oz_from = std::max(0, tuned_int("PACMAN_B200_INT8_FROM", tu.int8_from));
  bool tail = tail_event == nullptr;
  for (int j = 0; j < steps; ++j) {
    const int c = cp.cnt[j];
    const int n = c + cp.pre[cp.off[j] + c];
    if (!tail && n < 2 * sms) {  // from here on the steps leave SMs idle
      PB_CUDA(cudaEventRecord(tail_event, st));
      tail = true;
    }
    SolveReport::TimedLaunch tl{};
    if (rep.time_kernels) {
      PB_CUDA(cudaEventCreate(&tl.e0));
      PB_CUDA(cudaEventCreate(&tl.e1));
      PB_CUDA(cudaEventRecord(tl.e0, st));
    }
    // With int8 slices: the FP64 kernel (two CTAs per SM) for the short K
    // loops of the first steps, writing the slices; the int8 kernel after.
    const bool i8 = a.slices != nullptr && j >= oz_from;
    if (a.slices == nullptr)
      k_col_step<false><<<n, kColThreads, kColSmem, st>>>(a, ds, dpre + cp.off[j], c, j);
    else if (!i8)
      k_col_step<true><<<n, kColThreads, kColSmem, st>>>(a, ds, dpre + cp.off[j], c, j);
    else {
      const int items = cp.pre[cp.ioff[j] + c];
      // Programmatic dependent launch: the step's copies and MMAs overlap
      // the tail of the previous k_diag_next (see griddepcontrol.wait in the
      // kernel); not behind an FP64 step, whose slices the copies read, and
      // not with kernel timing, where events separate the launches.
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(std::min(items, sms));
      cfg.blockDim = dim3(kWsThreads);
      cfg.dynamicSmemBytes = kWsSmem;
      cfg.stream = st;
      cudaLaunchAttribute attr[1];
      attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
      attr[0].val.programmaticStreamSerializationAllowed = rep.time_kernels || j == oz_from ? 0 : 1;
      cfg.attrs = attr;
      cfg.numAttrs = 1;
      PB_CUDA(cudaLaunchKernelEx(&cfg, k_col_step_ws, a, ds, static_cast<const int *>(dpre + cp.ioff[j]), c, j));
      note_launch();
      k_diag_next<<<c, 256, kDiagNextSmem, st>>>(a, ds, j);
    }
    note_launch();
    if (rep.time_kernels) {
      PB_CUDA(cudaEventRecord(tl.e1, st));
      // Tile products: (T - j - 1) row tiles x (j + 1) (update + solve), and
      // j + 1 for the next diagonal tile.
      tl.kind = i8 ? 1 : 0;
      for (int q = 0; q < c; ++q) {
        tl.flops += 2.0 * TB * TB * TB * double(hs[q].T - j) * double(j + 1);
        if (i8) tl.mma_products += double(hs[q].T - j) * double(j);
      }
      rep.timed.push_back(tl);
    }
  }
  if (!tail) PB_CUDA(cudaEventRecord(tail_event, st));
}

void finish_kernel_timing(SolveReport &rep, cudaEvent_t ref) {
  if (rep.timed.empty()) return;
  // Intervals [start, end) in ms after ref, per kind and for both kinds; the
  // span is the length of their union (launches of different slot groups
  // overlap in time on their own streams).
  std::vector<std::pair<double, double>> iv[3];
  for (const auto &t : rep.timed) {
    float a0 = 0.f, a1 = 0.f;
    PB_CUDA(cudaEventElapsedTime(&a0, ref, t.e0));
    PB_CUDA(cudaEventElapsedTime(&a1, ref, t.e1));
    iv[t.kind].push_back({a0, a1});
    iv[2].push_back({a0, a1});
    rep.flops_kind[t.kind] += t.flops;
    rep.mma_products_i8 += t.mma_products;
    rep.launches_kind[t.kind] += 1;
    rep.update_flops += t.flops;
    rep.update_launches += 1;
    cudaEventDestroy(t.e0);
    cudaEventDestroy(t.e1);
  }
  rep.timed.clear();
  double span[3] = {0.0, 0.0, 0.0};
  for (int k = 0; k < 3; ++k) {
    std::sort(iv[k].begin(), iv[k].end());
    double cs = 0.0, ce = -1.0;
    bool open = false;
    for (const auto &x : iv[k]) {
      if (!open || x.first > ce) {
        if (open) span[k] += ce - cs;
        cs = x.first;
        ce = x.second;
        open = true;
      } else if (x.second > ce) {
        ce = x.second;
      }
    }
    if (open) span[k] += ce - cs;
  }
  rep.ms_kind[0] += span[0];
  rep.ms_kind[1] += span[1];
  rep.ms_update += span[2];
}

int chol_long_slots(const std::vector<BigSlot> &hs) {
  int c = 0;
  while (c < int(hs.size()) && hs[c].T >= kBkLong) ++c;
  return c;
}

namespace {

// One sweep over ns slots, by clusters or by single CTAs.
template <typename Single, typename Long>
void launch_sweep(const BigArgs &a, const BigSlot *ds, int ns, bool clusters, size_t smem,
                  size_t smem_cluster, Single single, Long cluster, cudaStream_t st) {
  if (clusters) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ns * kBkCluster);
    cfg.blockDim = dim3(288);
    cfg.dynamicSmemBytes = smem_cluster;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = kBkCluster;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    PB_CUDA(cudaLaunchKernelEx(&cfg, cluster, a, ds));
  } else {
    single<<<ns, 288, smem, st>>>(a, ds);
  }
  note_launch();
}

}  // namespace

void chol_launch_finish(const BigArgs &a, const BigSlot *ds, int ns, bool clusters, bool adjoint,
                        cudaStream_t st) {
  auto go = [&](auto F, auto single, int S) {
    constexpr int kF = decltype(F)::value, kS = bk_cluster_stages(kF);
    launch_sweep(a, ds, ns, clusters, chol_back_smem(a.F, S), chol_back_smem(a.F, kS, kBkCluster),
                 single, k_chol_back<kF, kS, kBkCluster>, st);
  };
  const bool deep = tuned_int("PACMAN_B200_BACK_STAGES", tuning_for_current_device().back_stages) ==
                    kBkDeep;
  using std::integral_constant;
  if (a.F == 1 && deep) go(integral_constant<int, 1>{}, k_chol_back<1, kBkDeep>, kBkDeep);
  else if (a.F == 1) go(integral_constant<int, 1>{}, k_chol_back<1, bk_stages(1)>, bk_stages(1));
  else if (a.F <= 2) go(integral_constant<int, 2>{}, k_chol_back<2, bk_stages(2)>, bk_stages(2));
  else if (a.F <= 4) go(integral_constant<int, 4>{}, k_chol_back<4, bk_stages(4)>, bk_stages(4));
  else go(integral_constant<int, kMaxF>{}, k_chol_back<kMaxF, bk_stages(kMaxF)>, bk_stages(kMaxF));
  if (!adjoint) {
    // Up to eight blocks share a slot's targets.
    const dim3 grid(ns, 8);
    if (a.F == 1) k_chol_eval<1><<<grid, kEvThreads, 0, st>>>(a, ds);
    else if (a.F <= 4) k_chol_eval<4><<<grid, kEvThreads, 0, st>>>(a, ds);
    else k_chol_eval<kMaxF><<<grid, kEvThreads, 0, st>>>(a, ds);
    note_launch();
  }
}

void chol_launch_forward(const BigArgs &a, const BigSlot *ds, int ns, bool clusters,
                         cudaStream_t st) {
  auto go = [&](auto F) {
    constexpr int kF = decltype(F)::value, kS = bk_cluster_stages(kF);
    launch_sweep(a, ds, ns, clusters, chol_fwd_smem(a.F, bk_stages(kF)),
                 chol_fwd_smem(a.F, kS, kBkCluster), k_chol_fwd<kF, bk_stages(kF)>,
                 k_chol_fwd<kF, kS, kBkCluster>, st);
  };
  using std::integral_constant;
  if (a.F == 1) go(integral_constant<int, 1>{});
  else if (a.F <= 2) go(integral_constant<int, 2>{});
  else if (a.F <= 4) go(integral_constant<int, 4>{});
  else go(integral_constant<int, kMaxF>{});
}

size_t oz_slot_bytes(int T) { return size_t(oz_pair_off(T, (T + 1) / 2, 0)); }

}  // namespace pacman_b200
