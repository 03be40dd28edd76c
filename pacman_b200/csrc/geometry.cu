// Geometry phase of the B200 RBF-PUM transfer: patch radius, centre cover,
// per-patch membership lists and the partition-of-unity gather.
//
// Replaces the ArborX BVH queries of the reference (src/rbf_pum/callbacks.hpp,
// clustering/clusters_radius.hpp, clustering/clustering.hpp, solver/solver.hpp
// :45-66 and :137-168) by uniform-grid searches over coalesced double4 points.
// Every predicate uses the exact arithmetic of common.cuh, so the radius, the
// centres and the sorted membership lists equal the CPU restatement's bit for
// bit.
#include <cub/cub.cuh>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstddef>
#include <cstring>

#include "plan.hpp"

namespace pacman_b200 {
namespace {

constexpr int kThreads = 256;

inline int grid_for(int64_t n, int per_block = kThreads, int cap = 148 * 16) {
  int64_t b = (n + per_block - 1) / per_block;
  if (b < 1) b = 1;
  if (b > cap) b = cap;
  return int(b);
}

// ---------------------------------------------------------------------------
// Packing and bounding box
// ---------------------------------------------------------------------------

// Device scratch of one geometry build, zeroed by one memset: the bounding
// box, the radius search's state and the counters of the kernels whose last
// block finishes the job (every block adds itself to a ticket after its own
// results are visible; the one that takes the last ticket goes on).
constexpr int kMaxSamples = 7;     // 2 dim + 1
constexpr int kNearBlocks = 148 * 4;
constexpr int kKnnCap = 2048;      // keys gathered for the exact selection

struct GeoScratch {
  // Order-preserving images (dbl_to_ordered) of the box, lower bounds
  // complemented so that zero is neutral for both halves.
  unsigned long long box[6];
  double samples[kMaxSamples][3];
  double proj[kMaxSamples][3];
  unsigned long long prefix[kMaxSamples];
  long long krem[kMaxSamples];
  double kth[kMaxSamples];
  double lo[3], hi[3];
  double radius;
  int nsamples;
  int overflow;                    // more than kKnnCap keys shared a 16-bit prefix
  unsigned int ticket[16];
  unsigned int ncand[kMaxSamples];
  unsigned int hist[8][kMaxSamples][256];
  // Written before they are read: not part of the memset.
  unsigned long long near_bits[kMaxSamples][kNearBlocks];
  unsigned int near_id[kMaxSamples][kNearBlocks];
  unsigned long long cand[kMaxSamples][kKnnCap];
};
constexpr size_t kGeoZero = offsetof(GeoScratch, near_bits);
// What the host reads back after the radius search.
constexpr size_t kGeoReport = offsetof(GeoScratch, ticket);

// True in every thread of the block that finishes last.
__device__ __forceinline__ bool last_block(unsigned int *ticket) {
  __shared__ bool last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(ticket, 1u) == gridDim.x * gridDim.y - 1u;
  __syncthreads();
  if (last) __threadfence();
  return last;
}

// Row-major [n x dim] doubles -> zero-padded double4 for the sources
// (blockIdx.y = 0, with their exact bounding box in sc->box) and the targets.
__global__ void k_pack(const double *__restrict__ src, int64_t n, double4 *src4,
                       const double *__restrict__ tgt, int64_t m, double4 *tgt4, int dim,
                       GeoScratch *sc) {
  const bool is_src = blockIdx.y == 0;
  const double *in = is_src ? src : tgt;
  double4 *out = is_src ? src4 : tgt4;
  const int64_t count = is_src ? n : m;
  unsigned long long mn[3] = {0ull, 0ull, 0ull}, mx[3] = {0ull, 0ull, 0ull};
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < count;
       i += (int64_t)gridDim.x * blockDim.x) {
    double c[3] = {0.0, 0.0, 0.0};
    for (int d = 0; d < dim; ++d) c[d] = in[i * dim + d];
    out[i] = make_double4(c[0], c[1], c[2], 0.0);
    if (is_src) {
      for (int d = 0; d < 3; ++d) {
        const unsigned long long o = dbl_to_ordered(c[d]);
        mn[d] = ~o > mn[d] ? ~o : mn[d];
        mx[d] = o > mx[d] ? o : mx[d];
      }
    }
  }
  if (!is_src) return;
  for (int d = 0; d < 3; ++d) {
    for (int s = 16; s > 0; s >>= 1) {
      const unsigned long long a = __shfl_xor_sync(0xffffffffu, mn[d], s);
      const unsigned long long b = __shfl_xor_sync(0xffffffffu, mx[d], s);
      mn[d] = a > mn[d] ? a : mn[d];
      mx[d] = b > mx[d] ? b : mx[d];
    }
  }
  // One atomic per block and bound: with one per warp the six addresses were
  // the kernel's time (1M points: 84 us).
  __shared__ unsigned long long red[6][kThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0)
    for (int d = 0; d < 3; ++d) {
      red[d][warp] = mn[d];
      red[3 + d][warp] = mx[d];
    }
  __syncthreads();
  if (threadIdx.x < 6) {
    unsigned long long v = 0ull;
    for (int w = 0; w < kThreads / 32; ++w) v = red[threadIdx.x][w] > v ? red[threadIdx.x][w] : v;
    atomicMax(&sc->box[threadIdx.x], v);
  }
}

// ---------------------------------------------------------------------------
// FindRadius (src/rbf_pum/clustering/clusters_radius.hpp:22-125)
// ---------------------------------------------------------------------------
//
// Every kernel reads the sources once for all 2 dim + 1 samples, and its last
// block does the short serial step that the next one needs.

// Box and sample points (:60-97).
__device__ void radius_samples(const GeoScratch *sc, int dim, double lo[3], double hi[3],
                               double (*samples)[3]) {
  double center[3] = {0.0, 0.0, 0.0};
  for (int d = 0; d < 3; ++d) {
    lo[d] = d < dim ? ordered_to_dbl(~sc->box[d]) : 0.0;
    hi[d] = d < dim ? ordered_to_dbl(sc->box[3 + d]) : 0.0;
  }
  for (int d = 0; d < dim; ++d) center[d] = __ddiv_rn(__dadd_rn(lo[d], hi[d]), 2.0);
  for (int s = 0; s < kMaxSamples; ++s)
    for (int d = 0; d < 3; ++d) samples[s][d] = center[d];
  for (int a = 0; a < dim; ++a) {
    const double len = fabs(__dsub_rn(hi[a], lo[a]));
    double s_a = __dsub_rn(center[a], __dmul_rn(len, 0.25));
    samples[a + 1][a] = s_a;
    s_a = __dadd_rn(s_a, __dmul_rn(len, 0.5));
    samples[dim + a + 1][a] = s_a;
  }
}

// Nearest source of each sample (lowest id on ties): the lexicographic minimum
// of (squared distance, id), per block and then over the blocks.  The bit
// pattern of a squared distance is monotone for values >= 0.
__global__ void k_nearest(const double4 *__restrict__ pts, int64_t n, int dim, long long k,
                          GeoScratch *sc) {
  __shared__ double smp[kMaxSamples][3];
  __shared__ unsigned long long rb[kMaxSamples][kThreads / 32];
  __shared__ unsigned int ri[kMaxSamples][kThreads / 32];
  const int ns = 2 * dim + 1;
  if (threadIdx.x == 0) {
    // Every block works on its own copy; the first one reports it.
    double lo[3], hi[3];
    radius_samples(sc, dim, lo, hi, smp);
    if (blockIdx.x == 0) {
      for (int d = 0; d < 3; ++d) {
        sc->lo[d] = lo[d];
        sc->hi[d] = hi[d];
      }
      for (int s = 0; s < kMaxSamples; ++s)
        for (int d = 0; d < 3; ++d) sc->samples[s][d] = smp[s][d];
      sc->nsamples = ns;
    }
  }
  __syncthreads();
  unsigned long long bits[kMaxSamples];
  unsigned int id[kMaxSamples];
#pragma unroll
  for (int s = 0; s < kMaxSamples; ++s) {
    bits[s] = ~0ull;
    id[s] = 0xffffffffu;
  }
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const double4 p = pts[i];
#pragma unroll
    for (int s = 0; s < kMaxSamples; ++s) {
      if (s >= ns) break;
      const unsigned long long b = (unsigned long long)__double_as_longlong(
          sqdist3(smp[s][0], smp[s][1], smp[s][2], p.x, p.y, p.z));
      if (b < bits[s]) {  // ids ascend within a thread
        bits[s] = b;
        id[s] = (unsigned int)i;
      }
    }
  }
  auto better = [](unsigned long long b, unsigned int i, unsigned long long c, unsigned int j) {
    return b < c || (b == c && i < j);
  };
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  auto reduce = [&](int s) {
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long b = __shfl_xor_sync(0xffffffffu, bits[s], o);
      const unsigned int j = __shfl_xor_sync(0xffffffffu, id[s], o);
      if (better(b, j, bits[s], id[s])) {
        bits[s] = b;
        id[s] = j;
      }
    }
    if (lane == 0) {
      rb[s][warp] = bits[s];
      ri[s][warp] = id[s];
    }
  };
#pragma unroll
  for (int s = 0; s < kMaxSamples; ++s)
    if (s < ns) reduce(s);
  __syncthreads();
  if (threadIdx.x < ns) {
    const int s = threadIdx.x;
    unsigned long long b = ~0ull;
    unsigned int j = 0xffffffffu;
    for (int w = 0; w < kThreads / 32; ++w)
      if (better(rb[s][w], ri[s][w], b, j)) {
        b = rb[s][w];
        j = ri[s][w];
      }
    sc->near_bits[s][blockIdx.x] = b;
    sc->near_id[s][blockIdx.x] = j;
  }
  if (!last_block(&sc->ticket[0])) return;
  // The last block: warp s reduces sample s over the blocks.
  if (warp < ns) {
    const int s = warp;
    unsigned long long b = ~0ull;
    unsigned int j = 0xffffffffu;
    for (unsigned int u = lane; u < gridDim.x; u += 32) {
      const unsigned long long c = __ldcg(&sc->near_bits[s][u]);
      const unsigned int q = __ldcg(&sc->near_id[s][u]);
      if (better(c, q, b, j)) {
        b = c;
        j = q;
      }
    }
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long c = __shfl_xor_sync(0xffffffffu, b, o);
      const unsigned int q = __shfl_xor_sync(0xffffffffu, j, o);
      if (better(c, q, b, j)) {
        b = c;
        j = q;
      }
    }
    if (lane == 0) {
      // Without a comparable distance (NaN coordinates) the first source.
      const double4 p = pts[j == 0xffffffffu ? 0u : j];
      sc->proj[s][0] = p.x;
      sc->proj[s][1] = p.y;
      sc->proj[s][2] = p.z;
      sc->krem[s] = k;
    }
  }
}

// The k-th smallest squared distance (raw bits) from projected sample s to the
// sources.  One 8-bit radix-select pass: histogram of the digit among the
// keys that share the prefix found so far, then (last block) the digit that
// holds the k-th key.
__global__ void k_knn_hist(const double4 *__restrict__ pts, int64_t n, int dim, int pass,
                           GeoScratch *sc) {
  __shared__ unsigned int h[kMaxSamples][256];
  __shared__ double smp[kMaxSamples][3];
  __shared__ unsigned long long pre[kMaxSamples];
  const int ns = 2 * dim + 1;
  for (int i = threadIdx.x; i < ns * 256; i += blockDim.x) (&h[0][0])[i] = 0u;
  if (threadIdx.x < ns) {
    for (int d = 0; d < 3; ++d) smp[threadIdx.x][d] = sc->proj[threadIdx.x][d];
    pre[threadIdx.x] = sc->prefix[threadIdx.x];
  }
  __syncthreads();
  const int shift = 56 - 8 * pass;
  const unsigned long long hmask = pass == 0 ? 0ull : (~0ull << (64 - 8 * pass));
  for (int64_t i0 = blockIdx.x * (int64_t)blockDim.x; i0 < n;
       i0 += (int64_t)gridDim.x * blockDim.x) {  // block-uniform: whole warps vote below
    const int64_t i = i0 + threadIdx.x;
    const double4 p = pts[i < n ? i : n - 1];
#pragma unroll
    for (int s = 0; s < kMaxSamples; ++s) {
      if (s >= ns) break;
      const unsigned long long key = (unsigned long long)__double_as_longlong(
          sqdist3(smp[s][0], smp[s][1], smp[s][2], p.x, p.y, p.z));
      const bool in = i < n && (key & hmask) == pre[s];
      const unsigned int dig = (unsigned int)(key >> shift) & 0xffu;
      // Nearly all keys of a warp share the leading digit: one add for them.
      const unsigned int m = __ballot_sync(0xffffffffu, in);
      if (in) {
        const unsigned int same = __match_any_sync(m, dig);
        if ((threadIdx.x & 31) == __ffs(same) - 1) atomicAdd(&h[s][dig], __popc(same));
      }
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < ns * 256; i += blockDim.x) {
    const unsigned int v = (&h[0][0])[i];
    if (v) atomicAdd(&sc->hist[pass][0][0] + i, v);
  }
  if (!last_block(&sc->ticket[1 + pass])) return;
  const int lane = threadIdx.x & 31, s = threadIdx.x >> 5;
  if (s >= ns) return;
  // Lane l sums bins 8 l .. 8 l + 7; the lane whose range crosses k finds the
  // digit (the last bin if the counts never reach k).
  unsigned int c[8];
  long long mine = 0;
  for (int q = 0; q < 8; ++q) {
    c[q] = __ldcg(&sc->hist[pass][s][8 * lane + q]);
    mine += c[q];
  }
  long long incl = mine;
  for (int o = 1; o < 32; o <<= 1) {
    const long long v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  const long long k = sc->krem[s];
  const unsigned int reach = __ballot_sync(0xffffffffu, incl >= k);
  const int owner = reach ? __ffs(reach) - 1 : 31;
  __syncwarp();
  if (lane == owner) {
    long long cum = incl - mine;
    int d = 0;
    while (d < 7 && cum + (long long)c[d] < k) cum += c[d++];
    sc->krem[s] = k - cum;
    sc->prefix[s] |= ((unsigned long long)(8 * lane + d)) << shift;
    if (pass == 7) sc->kth[s] = __longlong_as_double((long long)(sc->prefix[s]));
  }
}

// Kokkos::sort of the per-sample maxima and the median pick
// (clusters_radius.hpp:121-124).
__device__ void radius_median(GeoScratch *sc, int dim) {
  double v[kMaxSamples];
  const int ns = 2 * dim + 1;
  for (int s = 0; s < ns; ++s) v[s] = *(volatile double *)&sc->kth[s];
  for (int i = 1; i < ns; ++i) {
    const double x = v[i];
    int j = i - 1;
    while (j >= 0 && v[j] > x) {
      v[j + 1] = v[j];
      --j;
    }
    v[j + 1] = x;
  }
  sc->radius = __dsqrt_rn(v[dim]);
}

__global__ void k_radius_final(GeoScratch *sc, int dim) {
  if (threadIdx.x == 0) radius_median(sc, dim);
}

// After two passes few keys share the 16-bit prefix (a sixteenth of an octave
// of squared distance): they are gathered, and the last block selects among
// them by rank.  More than kKnnCap of them (many equal distances) set
// `overflow`, and the host runs the remaining passes instead.
__global__ void k_knn_gather(const double4 *__restrict__ pts, int64_t n, int dim,
                             GeoScratch *sc) {
  __shared__ double smp[kMaxSamples][3];
  __shared__ unsigned long long pre[kMaxSamples];
  const int ns = 2 * dim + 1;
  if (threadIdx.x < ns) {
    for (int d = 0; d < 3; ++d) smp[threadIdx.x][d] = sc->proj[threadIdx.x][d];
    pre[threadIdx.x] = sc->prefix[threadIdx.x];
  }
  __syncthreads();
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const double4 p = pts[i];
#pragma unroll
    for (int s = 0; s < kMaxSamples; ++s) {
      if (s >= ns) break;
      const unsigned long long key = (unsigned long long)__double_as_longlong(
          sqdist3(smp[s][0], smp[s][1], smp[s][2], p.x, p.y, p.z));
      if ((key & (~0ull << 48)) == pre[s]) {
        const unsigned int at = atomicAdd(&sc->ncand[s], 1u);
        if (at < kKnnCap) sc->cand[s][at] = key;
      }
    }
  }
  if (!last_block(&sc->ticket[9])) return;
  __shared__ unsigned long long keys[kKnnCap];
  __shared__ int over;
  if (threadIdx.x == 0) over = 0;
  __syncthreads();
  for (int s = 0; s < ns; ++s) {
    const unsigned int cnt = __ldcg(&sc->ncand[s]);
    if (cnt > kKnnCap || cnt == 0u) {  // block-uniform
      if (threadIdx.x == 0) over = 1;
      break;
    }
    for (unsigned int i = threadIdx.x; i < cnt; i += blockDim.x) keys[i] = __ldcg(&sc->cand[s][i]);
    __syncthreads();
    const long long k = sc->krem[s];
    for (unsigned int i = threadIdx.x; i < cnt; i += blockDim.x) {
      const unsigned long long v = keys[i];
      long long less = 0, eq = 0;
      for (unsigned int j = 0; j < cnt; ++j) {
        less += keys[j] < v;
        eq += keys[j] == v;
      }
      if (less < k && k <= less + eq)  // equal keys write the same value
        *(volatile double *)&sc->kth[s] = __longlong_as_double((long long)v);
    }
    __syncthreads();
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    sc->overflow = over;
    if (!over) radius_median(sc, dim);
  }
}

// ---------------------------------------------------------------------------
// Uniform grids
// ---------------------------------------------------------------------------

struct GridSpec {
  double lo[3];
  double hi[3];  // inclusive upper bound of the grid domain
  double inv_h;
  int nc[3];
  int ncells;
  int clamp;     // points outside the domain go to the nearest cell
};

GridSpec make_grid_spec(int dim, const double *bb_lo, const double *bb_hi, double radius,
                        int64_t npts) {
  GridSpec g{};
  const int64_t cap = std::max<int64_t>(std::min<int64_t>(npts * 2, int64_t(1) << 28), 1 << 12);
  double h = radius * (1.0 + 0x1p-20);
  for (int it = 0; it < 200; ++it) {
    int64_t tot = 1;
    bool ok = true;
    for (int d = 0; d < 3; ++d) {
      if (d >= dim) {
        g.nc[d] = 1;
        continue;
      }
      const double ext = (bb_hi[d] - bb_lo[d]) + 2.0 * h;
      const double c = std::floor(ext / h) + 1.0;
      if (!(c < 1.0e9)) {
        ok = false;
        break;
      }
      g.nc[d] = int(c);
      tot *= g.nc[d];
      if (tot > cap) {
        ok = false;
        break;
      }
    }
    if (ok) {
      g.ncells = int(tot);
      break;
    }
    h *= 1.25;
  }
  if (g.ncells == 0) throw Error{PACMAN_B200_ERR_LIMIT, "could not size the search grid"};
  for (int d = 0; d < 3; ++d) {
    g.lo[d] = d < dim ? bb_lo[d] - h : 0.0;
    g.hi[d] = d < dim ? bb_hi[d] + h : 0.0;
  }
  g.inv_h = 1.0 / h;
  return g;
}

// Cell of a point; outside the grid's domain the cell after the last one.
__device__ __forceinline__ int cell_of(const GridSpec &g, const double4 &p) {
  const double c[3] = {p.x, p.y, p.z};
  for (int d = 0; d < 3; ++d)
    if (!g.clamp && !(c[d] >= g.lo[d] && c[d] <= g.hi[d])) return g.ncells;
  const int a = cell_coord(c[0], g.lo[0], g.inv_h, g.nc[0]);
  const int b = cell_coord(c[1], g.lo[1], g.inv_h, g.nc[1]);
  const int e = cell_coord(c[2], g.lo[2], g.inv_h, g.nc[2]);
  return (a * g.nc[1] + b) * g.nc[2] + e;
}

// Counting sort of up to two point sets by grid cell (set 1's cells follow set
// 0's): the count of each cell and every point's rank in its cell, an
// exclusive scan over the cells, then the points moved to their places.  The
// order inside a cell is that of the atomics, which no consumer depends on.
// Against a radix sort of (cell, id) pairs: 5 launches for both sets instead of
// about 9 for each.
__global__ void k_cell_count(const double4 *__restrict__ p0, int64_t n0, GridSpec g0,
                             const double4 *__restrict__ p1, int64_t n1, GridSpec g1,
                             unsigned *__restrict__ count, int *__restrict__ rank) {
  const int lane = threadIdx.x & 31;
  for (int64_t b = blockIdx.x * (int64_t)blockDim.x; b < n0 + n1;
       b += (int64_t)gridDim.x * blockDim.x) {  // block-uniform: whole warps vote below
    const int64_t i = b + threadIdx.x;
    const bool live = i < n0 + n1, first = i < n0;
    int c = -1;
    bool out = false;
    if (live) {
      c = first ? cell_of(g0, p0[i]) : cell_of(g1, p1[i - n0]);
      out = !first && c == g1.ncells;  // targets outside: one add per warp
      if (!first) c += g0.ncells + 1;
    }
    const unsigned int m = __ballot_sync(0xffffffffu, out);
    int r = 0;
    if (m) {
      const int leader = __ffs(m) - 1;
      if (lane == leader) r = int(atomicAdd(&count[c], unsigned(__popc(m))));
      r = __shfl_sync(0xffffffffu, r, leader) + __popc(m & ((1u << lane) - 1u));
    }
    if (live) rank[i] = out ? r : int(atomicAdd(&count[c], 1u));
  }
}

// The sorted copy of a point carries its id in w (an integer below 2^31,
// exact).
__global__ void k_cell_place(const double4 *__restrict__ p0, int64_t n0, GridSpec g0,
                             const double4 *__restrict__ p1, int64_t n1, GridSpec g1,
                             const unsigned *__restrict__ start, const int *__restrict__ rank,
                             double4 *__restrict__ sorted) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n0 + n1;
       i += (int64_t)gridDim.x * blockDim.x) {
    const bool first = i < n0;
    double4 p = first ? p0[i] : p1[i - n0];
    const int c = first ? cell_of(g0, p) : g0.ncells + 1 + cell_of(g1, p);
    p.w = double(first ? i : i - n0);
    sorted[start[c] + unsigned(rank[i])] = p;
  }
}

__global__ void k_ids(const double4 *__restrict__ pts, int64_t n, int *__restrict__ out) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    out[i] = int(pts[i].w);
}

GridView view_of(const GridSpec &g, const unsigned *start) {
  GridView v{};
  for (int d = 0; d < 3; ++d) {
    v.lo[d] = g.lo[d];
    v.nc[d] = g.nc[d];
  }
  v.inv_h = g.inv_h;
  v.ncells = g.ncells;
  v.start = reinterpret_cast<const int *>(start);
  return v;
}

// Bump allocation inside one device block.
struct Slab {
  char *cur = nullptr;
  size_t used = 0;
  template <typename T> T *take(size_t count) {
    T *r = reinterpret_cast<T *>(cur ? cur + used : nullptr);
    used += (sizeof(T) * count + 255) & ~size_t(255);
    return r;
  }
};

// Sorts set 0 (and set 1) into the cells of g0 (and g1), each followed by its
// points outside the domain: set 1 starts at sorted[n0].  Each set has less than
// 2^31 points; positions in both together are unsigned.  With a null slab the
// call only counts the memory it needs.
void sort_into_cells(Slab &slab, const double4 *p0, int64_t n0, const GridSpec &g0,
                     const double4 *p1, int64_t n1, const GridSpec &g1, GridView &v0, GridView &v1,
                     const double4 *&sorted, cudaStream_t st) {
  const size_t cells = size_t(g0.ncells) + 1 + size_t(n1 > 0 ? g1.ncells + 1 : 0);
  const size_t npts = size_t(std::max<int64_t>(n0 + n1, 1));
  if (cells + 1 > 0x7fffffffull)
    throw Error{PACMAN_B200_ERR_LIMIT, "more than 2^31 - 1 cells in one search grid"};
  unsigned *count = slab.take<unsigned>(cells + 1);
  unsigned *start = slab.take<unsigned>(cells + 1);
  int *rank = slab.take<int>(npts);
  double4 *out = slab.take<double4>(npts);
  size_t tb = 0;
  PB_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, tb, count, start, int(cells + 1), st));
  void *tmp = slab.take<char>(tb);
  if (!slab.cur) return;
  PB_CUDA(cudaMemsetAsync(count, 0, sizeof(unsigned) * (cells + 1), st));
  k_cell_count<<<grid_for(n0 + n1), kThreads, 0, st>>>(p0, n0, g0, p1, n1, g1, count, rank);
  PB_CUDA(cub::DeviceScan::ExclusiveSum(tmp, tb, count, start, int(cells + 1), st));
  k_cell_place<<<grid_for(n0 + n1), kThreads, 0, st>>>(p0, n0, g0, p1, n1, g1, start, rank, out);
  note_launch(2);
  PB_CUDA(cudaGetLastError());
  v0 = view_of(g0, start);
  v1 = view_of(g1, start + g0.ncells + 1);
  if (n1 == 0) v1.start = nullptr;
  sorted = out;
}

// The grid of centres (few points): radix sort of (cell, id), ids ascending in
// a cell.
__global__ void k_cell_keys(const double4 *__restrict__ pts, int64_t n, GridSpec g, int *keys,
                            int *ids) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    keys[i] = cell_of(g, pts[i]);
    ids[i] = int(i);
  }
}

// start[c] = first sorted position whose key >= c, for c in [0, ncells], and
// the points in that order.
__global__ void k_cell_start(const int *skeys, const int *items, const double4 *__restrict__ pts,
                             int64_t n, int ncells, int *start, double4 *sorted) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i <= n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int prev = (i == 0) ? -1 : skeys[i - 1];
    const int cur = (i == n) ? ncells + 1 : skeys[i];
    for (int c = prev + 1; c <= cur && c <= ncells; ++c) start[c] = int(i);
    if (i < n) {
      double4 p = pts[items[i]];
      p.w = double(items[i]);
      sorted[i] = p;
    }
  }
}

void build_grid(DevGrid &out, const double4 *pts, int64_t n, int dim, const double *bb_lo,
                const double *bb_hi, double radius, cudaStream_t st) {
  const GridSpec g = make_grid_spec(dim, bb_lo, bb_hi, radius, n);
  const int64_t nn = std::max<int64_t>(n, 1);
  out.sorted.alloc(sizeof(double4) * nn, st);
  out.start.alloc(sizeof(int) * (size_t(g.ncells) + 2), st);
  if (n > 0) {
    int end_bit = 1;
    while ((int64_t(1) << end_bit) <= g.ncells) ++end_bit;
    DevMem mem;
    Slab slab;
    int *keys = nullptr, *ids = nullptr, *skeys = nullptr, *items = nullptr;
    void *tmp = nullptr;
    size_t tb = 0;
    for (int pass = 0; pass < 2; ++pass) {
      if (pass) {
        mem.alloc(slab.used, st);
        slab = Slab{mem.as<char>(), 0};
      }
      keys = slab.take<int>(nn);
      ids = slab.take<int>(nn);
      skeys = slab.take<int>(nn);
      items = slab.take<int>(nn);
      if (!pass)
        PB_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, tb, keys, skeys, ids, items, int(n), 0,
                                                end_bit, st));
      tmp = slab.take<char>(tb);
    }
    k_cell_keys<<<grid_for(n), kThreads, 0, st>>>(pts, n, g, keys, ids);
    PB_CUDA(cub::DeviceRadixSort::SortPairs(tmp, tb, keys, skeys, ids, items, int(n), 0, end_bit,
                                            st));
    k_cell_start<<<grid_for(n + 1), kThreads, 0, st>>>(skeys, items, pts, n, g.ncells,
                                                       out.start.as<int>(),
                                                       out.sorted.as<double4>());
    note_launch(2);
  } else {
    PB_CUDA(cudaMemsetAsync(out.start.p, 0, sizeof(int) * (size_t(g.ncells) + 1), st));
  }
  PB_CUDA(cudaGetLastError());
  out.view = view_of(g, out.start.as<unsigned>());
  out.view.sorted = out.sorted.as<double4>();
}

// ---------------------------------------------------------------------------
// Centre cover (src/rbf_pum/clustering/clustering.hpp:127-271)
// ---------------------------------------------------------------------------

struct CandSpec {
  int dim;
  int shape[3];
  double dist[3];
  double lo[3];
  double r2;
  long long nb;
};

enum : unsigned char { kDead = 0, kAlive0 = 1, kSurvive = 2, kPending = 3 };

// Calls fn(point, in range) for the cell-sorted points in the 3^3 cells around
// q, 32 per call of the whole warp, until fn returns false (warp-uniform).
template <typename Fn>
__device__ __forceinline__ void warp_neighbors(const GridView &g, const double4 *__restrict__ pts,
                                               double qx, double qy, double qz, int lane,
                                               Fn &&fn) {
  const int cx = cell_coord(qx, g.lo[0], g.inv_h, g.nc[0]);
  const int cy = cell_coord(qy, g.lo[1], g.inv_h, g.nc[1]);
  const int cz = cell_coord(qz, g.lo[2], g.inv_h, g.nc[2]);
  const int x0 = max(cx - 1, 0), x1 = min(cx + 1, g.nc[0] - 1);
  const int y0 = max(cy - 1, 0), y1 = min(cy + 1, g.nc[1] - 1);
  const int z0 = max(cz - 1, 0), z1 = min(cz + 1, g.nc[2] - 1);
  const int ny = y1 - y0 + 1, runs = (x1 - x0 + 1) * ny;
  // Lane r < runs (at most 9) holds the r-th run of cells [s, e).
  unsigned rs = 0, re = 0;
  if (lane < runs) {
    const int base = ((x0 + lane / ny) * g.nc[1] + y0 + lane % ny) * g.nc[2];
    rs = unsigned(g.start[base + z0]);
    re = unsigned(g.start[base + z1 + 1]);
  }
  for (int r = 0; r < runs; ++r) {
    const unsigned s = __shfl_sync(0xffffffffu, rs, r), e = __shfl_sync(0xffffffffu, re, r);
    for (unsigned u = lane; u - lane < e - s; u += 32) {
      const bool ok = u < e - s;
      if (!fn(pts[ok ? s + u : s], ok)) return;
    }
  }
}

// Whether some point of the grid lies within squared distance r2 of q.
__device__ __forceinline__ bool warp_any_within(const GridView &g, const double4 *pts, double qx,
                                                double qy, double qz, double r2, int lane) {
  bool found = false;
  warp_neighbors(g, pts, qx, qy, qz, lane, [&](const double4 &p, bool ok) {
    found = __any_sync(0xffffffffu, ok && sqdist3(qx, qy, qz, p.x, p.y, p.z) <= r2);
    return !found;
  });
  return found;
}

// Steps 5-8: candidate coordinates (row-major storage, last axis fastest),
// source and target emptiness tags (nearest within r, i.e. squared distance
// <= r*r), snap to the nearest source (lowest id on ties).
// One warp per candidate centre (dense blobs put thousands of sources in a
// candidate's 3^3 cells, too many for one thread): the lanes split the
// neighbourhood, the nearest source is the lexicographic minimum of (squared
// distance, index) over the warp, so the result does not depend on the split.
__global__ void k_candidates(CandSpec cs, GridView sg, GridView tg,
                             const double4 *__restrict__ ssorted,
                             const double4 *__restrict__ src, int has_targets, double4 *cpos,
                             unsigned char *state) {
  const int lane = threadIdx.x & 31;
  const long long nw = (long long)gridDim.x * (blockDim.x >> 5);
  for (long long s = blockIdx.x * (long long)(blockDim.x >> 5) + (threadIdx.x >> 5); s < cs.nb;
       s += nw) {
    long long t = s;
    int coords[3] = {0, 0, 0};
    for (int a = cs.dim - 1; a >= 0; --a) {
      coords[a] = int(t % cs.shape[a]);
      t /= cs.shape[a];
    }
    double q[3] = {0.0, 0.0, 0.0};
    for (int a = 0; a < cs.dim; ++a) q[a] = __fma_rn(cs.dist[a], double(coords[a]), cs.lo[a]);
    double best = INFINITY;
    int bi = 0x7fffffff;
    warp_neighbors(sg, ssorted, q[0], q[1], q[2], lane, [&](const double4 &p, bool ok) {
      const double d2 = sqdist3(q[0], q[1], q[2], p.x, p.y, p.z);
      const int i = int(p.w);
      if (ok && (d2 < best || (d2 == best && i < bi))) {
        best = d2;
        bi = i;
      }
      return true;
    });
    for (int o = 16; o > 0; o >>= 1) {
      const double ob = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ob < best || (ob == best && oi < bi)) {
        best = ob;
        bi = oi;
      }
    }
    bool alive = (bi != 0x7fffffff) && (best <= cs.r2);
    if (alive && has_targets)
      alive = warp_any_within(tg, ssorted, q[0], q[1], q[2], cs.r2, lane);
    if (lane == 0) {
      state[s] = alive ? kAlive0 : kDead;
      cpos[s] = alive ? src[bi] : make_double4(q[0], q[1], q[2], 0.0);
    }
  }
}

// Step 9 (order-dependent pruning, clustering.hpp:228-254), parallel form.
// Centre i dies if a later neighbour j > i (in the 26-offset table) is alive
// before the loop and closer than the threshold, or if an earlier neighbour
// j < i that survived its own turn is that close.  The first case is decided
// here; the second is recorded as a bit mask and resolved by k_prune_resolve.
struct PruneOffsets {
  int n;
  long long off[26];
};

// What the host reads back after the cover, and the count of pending centres.
struct CoverReport {
  int K, status, pending;
};

__global__ void k_prune_mark(long long nb, PruneOffsets po, double thr,
                             const double4 *__restrict__ cpos,
                             const unsigned char *__restrict__ state0, unsigned char *state1,
                             unsigned int *mask, int *pending, CoverReport *rep) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nb;
       i += (long long)gridDim.x * blockDim.x) {
    unsigned int m = 0u;
    unsigned char st = kDead;
    if (state0[i] == kAlive0) {
      const double4 c = cpos[i];
      bool fwd = false;
      for (int o = 0; o < po.n; ++o) {
        const long long j = i + po.off[o];
        if (j < 0 || j >= nb || state0[j] != kAlive0) continue;
        const double4 q = cpos[j];
        if (sqdist3(c.x, c.y, c.z, q.x, q.y, q.z) < thr) {
          if (j > i) fwd = true;
          else m |= 1u << o;
        }
      }
      st = fwd ? kDead : (m ? kPending : kSurvive);
    }
    state1[i] = st;
    if (st == kPending) {
      mask[i] = m;
      pending[atomicAdd(&rep->pending, 1)] = int(i);
    }
  }
}

// Resolves the pending centres in ascending-id order semantics: a pending
// centre dies iff one of its masked earlier neighbours survived.  Each sweep
// over the pending list settles at least its smallest id, so as many sweeps as
// it has entries suffice.
__global__ void k_prune_resolve(PruneOffsets po, const unsigned int *__restrict__ mask,
                                const int *__restrict__ pending, unsigned char *state1_,
                                CoverReport *rep) {
  volatile unsigned char *state1 = state1_;
  const int np = rep->pending;
  for (int sweep = 0; sweep <= np; ++sweep) {
    int open = 0;
    for (int u = threadIdx.x; u < np; u += blockDim.x) {
      const long long i = pending[u];
      if (state1[i] != kPending) continue;
      const unsigned int m = mask[i];
      bool any_alive = false, undecided = false;
      for (int o = 0; o < po.n; ++o) {
        if (!(m & (1u << o))) continue;
        const unsigned char sj = state1[i + po.off[o]];
        if (sj == kSurvive) any_alive = true;
        else if (sj == kPending) undecided = true;
      }
      if (any_alive) state1[i] = kDead;
      else if (!undecided) state1[i] = kSurvive;
      else open = 1;
    }
    if (!__syncthreads_or(open)) return;
  }
  if (threadIdx.x == 0) rep->status = 1;
}

// Step 10: re-tag surviving centres without a target within r, a warp each.
__global__ void k_retag(long long nb, const double4 *__restrict__ cpos,
                        const unsigned char *__restrict__ state1, GridView tg,
                        const double4 *__restrict__ sorted, int has_targets, double r2,
                        unsigned char *flags) {
  const int lane = threadIdx.x & 31;
  const long long nw = (long long)gridDim.x * (blockDim.x >> 5);
  for (long long s = blockIdx.x * (long long)(blockDim.x >> 5) + (threadIdx.x >> 5); s < nb;
       s += nw) {
    bool keep = state1[s] == kSurvive;
    if (keep && has_targets) {
      const double4 c = cpos[s];
      keep = warp_any_within(tg, sorted, c.x, c.y, c.z, r2, lane);
    }
    if (lane == 0) flags[s] = keep ? 1 : 0;
  }
}

// ---------------------------------------------------------------------------
// Patch membership lists (solver.hpp:45-66): sqrt(d2) <= radius (ArborX
// sphere-point intersection), warp per patch; lists 0..K-1 the sources, lists
// K..2K-1 the targets, counted, scanned and filled together.
// ---------------------------------------------------------------------------

constexpr int kWarpSort = 256;    // lists up to here are sorted by the warp that fills them
constexpr int kBlockSort = 32768; // and up to here by a block

__global__ void k_member_count(int K, const double4 *__restrict__ centers, GridView sg,
                               GridView tg, const double4 *__restrict__ sorted, double rs,
                               double rt, int has_targets, int *cnt, int *long_list,
                               int *long_count) {
  const int lane = threadIdx.x & 31;
  const int warps = (blockDim.x >> 5) * gridDim.x;
  for (int k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; k < 2 * K; k += warps) {
    const bool is_src = k < K;
    const double4 c = centers[is_src ? k : k - K];
    const double radius = is_src ? rs : rt;
    int total = 0;
    if (is_src || has_targets)
      warp_neighbors(is_src ? sg : tg, sorted, c.x, c.y, c.z, lane,
                     [&](const double4 &p, bool ok) {
                       const bool in =
                           ok && __dsqrt_rn(sqdist3(c.x, c.y, c.z, p.x, p.y, p.z)) <= radius;
                       total += __popc(__ballot_sync(0xffffffffu, in));
                       return true;
                     });
    if (lane == 0) {
      cnt[k] = total;
      if (total > kWarpSort) long_list[atomicAdd(long_count, 1)] = k;
    }
  }
}

// Ascending bitonic sort of n2 (a power of two) integers in shared memory by
// nt threads; sync() is their barrier.
template <class Sync>
__device__ __forceinline__ void bitonic_sort(int *v, int n2, int t, int nt, Sync sync) {
  for (int k = 2; k <= n2; k <<= 1)
    for (int j = k >> 1; j > 0; j >>= 1) {
      for (int u = t; u < n2 / 2; u += nt) {
        const int i = 2 * u - (u & (j - 1));  // bit j clear
        const int a = v[i], b = v[i + j];
        if ((a > b) == ((i & k) == 0)) {
          v[i] = b;
          v[i + j] = a;
        }
      }
      sync();
    }
}

__global__ void __launch_bounds__(kThreads)
    k_member_fill(int K, const double4 *__restrict__ centers, GridView sg, GridView tg,
                  const double4 *__restrict__ sorted, double rs, double rt, int has_targets,
                  const int64_t *__restrict__ scan, int64_t *soff, int64_t *toff, int *sidx,
                  int *tidx) {
  __shared__ int buf[kThreads / 32][kWarpSort];
  const int lane = threadIdx.x & 31;
  int *v = buf[threadIdx.x >> 5];
  const int warps = (blockDim.x >> 5) * gridDim.x;
  const int64_t nsrc = scan[K];
  for (int k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; k < 2 * K; k += warps) {
    const bool is_src = k < K;
    const int64_t o = scan[k] - (is_src ? 0 : nsrc);
    const int n = int(scan[k + 1] - scan[k]);
    if (lane == 0) {
      (is_src ? soff : toff)[is_src ? k : k - K] = o;
      if (k == K - 1) soff[K] = nsrc;
      if (k == 2 * K - 1) toff[K] = o + n;
    }
    int *idx = (is_src ? sidx : tidx) + o;
    const double4 c = centers[is_src ? k : k - K];
    const double radius = is_src ? rs : rt;
    const bool here = n <= kWarpSort;
    int pos = 0;
    if (is_src || has_targets)
      warp_neighbors(is_src ? sg : tg, sorted, c.x, c.y, c.z, lane,
                     [&](const double4 &p, bool ok) {
                       const bool in =
                           ok && __dsqrt_rn(sqdist3(c.x, c.y, c.z, p.x, p.y, p.z)) <= radius;
                       const unsigned int bal = __ballot_sync(0xffffffffu, in);
                       if (in) (here ? v : idx)[pos + __popc(bal & ((1u << lane) - 1u))] = int(p.w);
                       pos += __popc(bal);
                       return true;
                     });
    if (!here) continue;  // k_member_sort
    int n2 = 2;
    while (n2 < n) n2 <<= 1;
    for (int u = n + lane; u < n2; u += 32) v[u] = 0x7fffffff;
    __syncwarp();
    bitonic_sort(v, n2, lane, 32, [] { __syncwarp(); });
    for (int u = lane; u < n; u += 32) idx[u] = v[u];
    __syncwarp();
  }
}

// Lists longer than kWarpSort, a block each, in shared memory.
__global__ void __launch_bounds__(512)
    k_member_sort(int K, const int64_t *__restrict__ scan, const int *__restrict__ long_list,
                  int *sidx, int *tidx) {
  extern __shared__ int vs[];
  const int k = long_list[blockIdx.x];
  const int n = int(scan[k + 1] - scan[k]);
  int *idx = k < K ? sidx + scan[k] : tidx + (scan[k] - scan[K]);
  int n2 = 2;
  while (n2 < n) n2 <<= 1;
  for (int u = threadIdx.x; u < n2; u += blockDim.x) vs[u] = u < n ? idx[u] : 0x7fffffff;
  __syncthreads();
  bitonic_sort(vs, n2, threadIdx.x, blockDim.x, [] { __syncthreads(); });
  for (int u = threadIdx.x; u < n; u += blockDim.x) idx[u] = vs[u];
}

// Lists beyond a block's shared memory (one set): CUB's segmented sort.
void sort_lists(DevMem &idx, int64_t nnz, int K, const int64_t *off, cudaStream_t st) {
  if (nnz == 0) return;
  DevMem out, tmp;
  out.alloc(sizeof(int) * nnz, st);
  size_t tb = 0;
  PB_CUDA(cub::DeviceSegmentedSort::SortKeys(nullptr, tb, idx.as<int>(), out.as<int>(), nnz, K,
                                             off, off + 1, st));
  tmp.alloc(tb, st);
  PB_CUDA(cub::DeviceSegmentedSort::SortKeys(tmp.p, tb, idx.as<int>(), out.as<int>(), nnz, K, off,
                                             off + 1, st));
  idx = std::move(out);
}

void build_lists(Plan &p, const GridView &sg, const GridView &tg, const double4 *sorted,
                 double r) {
  cudaStream_t st = p.stream;
  const int K = p.K;
  const int has_targets = p.m > 0 ? 1 : 0;
  p.soff.alloc(sizeof(int64_t) * (K + 1), st);
  p.toff.alloc(sizeof(int64_t) * (K + 1), st);
  p.n_host.resize(K);
  p.m_host.resize(K);
  p.snnz = p.tnnz = 0;
  if (K == 0) {
    p.sidx.alloc(sizeof(int), st);
    p.tidx.alloc(sizeof(int), st);
    PB_CUDA(cudaMemsetAsync(p.soff.p, 0, sizeof(int64_t), st));
    PB_CUDA(cudaMemsetAsync(p.toff.p, 0, sizeof(int64_t), st));
    return;
  }
  if (K > 0x3ffffffe) throw Error{PACMAN_B200_ERR_LIMIT, "too many patches"};
  DevMem mem;
  Slab slab;
  int *cnt = nullptr, *long_list = nullptr, *long_count = nullptr;
  int64_t *scan = nullptr;
  void *tmp = nullptr;
  size_t tb = 0;
  for (int pass = 0; pass < 2; ++pass) {
    if (pass) {
      mem.alloc(slab.used, st);
      slab = Slab{mem.as<char>(), 0};
    }
    cnt = slab.take<int>(2 * size_t(K) + 1);
    long_count = cnt + 2 * size_t(K);  // scanned as the closing entry, never added
    scan = slab.take<int64_t>(2 * size_t(K) + 1);
    long_list = slab.take<int>(2 * size_t(K));
    if (!pass)
      PB_CUDA(cub::DeviceScan::ExclusiveScan(nullptr, tb, cnt, scan, cub::Sum(), int64_t(0),
                                             2 * K + 1, st));
    tmp = slab.take<char>(tb);
  }
  PB_CUDA(cudaMemsetAsync(long_count, 0, sizeof(int), st));
  const int blocks = std::max(1, std::min((2 * K + 7) / 8, 148 * 32));
  // Sources within r, targets within r - 1e-14 (solver.hpp:264-270).
  k_member_count<<<blocks, kThreads, 0, st>>>(K, p.centers.as<double4>(), sg, tg, sorted, r,
                                              r - kEps, has_targets, cnt, long_list, long_count);
  PB_CUDA(cub::DeviceScan::ExclusiveScan(tmp, tb, cnt, scan, cub::Sum(), int64_t(0), 2 * K + 1,
                                         st));
  note_launch();
  int *h = static_cast<int *>(HostArena::get().alloc(sizeof(int) * (2 * size_t(K) + 1)));
  PB_CUDA(cudaMemcpyAsync(h, cnt, sizeof(int) * (2 * size_t(K) + 1), cudaMemcpyDeviceToHost, st));
  PB_CUDA(host_sync(st));
  int longest[2] = {0, 0};
  for (int k = 0; k < K; ++k) {
    p.n_host[k] = h[k];
    p.m_host[k] = h[K + k];
    p.snnz += h[k];
    p.tnnz += h[K + k];
    longest[0] = std::max(longest[0], h[k]);
    longest[1] = std::max(longest[1], h[K + k]);
  }
  const int nlong = h[2 * size_t(K)];
  if (p.snnz > (int64_t(1) << 31) - 1 || p.tnnz > (int64_t(1) << 31) - 1)
    throw Error{PACMAN_B200_ERR_LIMIT, "more than 2^31 patch memberships"};
  p.sidx.alloc(sizeof(int) * std::max<int64_t>(p.snnz, 1), st);
  p.tidx.alloc(sizeof(int) * std::max<int64_t>(p.tnnz, 1), st);
  k_member_fill<<<blocks, kThreads, 0, st>>>(K, p.centers.as<double4>(), sg, tg, sorted, r,
                                             r - kEps, has_targets, scan, p.soff.as<int64_t>(),
                                             p.toff.as<int64_t>(), p.sidx.as<int>(),
                                             p.tidx.as<int>());
  note_launch();
  const int most = std::max(longest[0], longest[1]);
  if (most > kBlockSort) {
    sort_lists(p.sidx, p.snnz, K, p.soff.as<int64_t>(), st);
    sort_lists(p.tidx, p.tnnz, K, p.toff.as<int64_t>(), st);
  } else if (nlong > 0) {
    int n2 = 2;
    while (n2 < most) n2 <<= 1;
    const size_t smem = sizeof(int) * size_t(n2);
    PB_CUDA(cudaFuncSetAttribute(k_member_sort, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 int(sizeof(int) * kBlockSort)));
    k_member_sort<<<nlong, 512, smem, st>>>(K, scan, long_list, p.sidx.as<int>(),
                                            p.tidx.as<int>());
    note_launch();
  }
  PB_CUDA(cudaGetLastError());
}

// ---------------------------------------------------------------------------
// Partition-of-unity gather (solver.hpp:137-168 and :275-285): for each
// target, the centres within r in ascending order, Shepard-normalised
// Wendland C2 weights, and the weighted sum of the local values of the
// patches whose target list holds it (binary search in that sorted list).
// Deterministic and equal to the reference's serial patch-order accumulation.
// ---------------------------------------------------------------------------

constexpr int kMaxPatchesPerTarget = 64;

__device__ __forceinline__ int64_t find_sorted(const int *a, int64_t n, int v) {
  int64_t lo = 0, hi = n;
  while (lo < hi) {
    const int64_t mid = (lo + hi) >> 1;
    if (a[mid] < v) lo = mid + 1;
    else hi = mid;
  }
  return (lo < n && a[lo] == v) ? lo : -1;
}

// Targets in the order of the search grid's cells, so that a warp's targets
// share their centres, patches and lists.  1M targets: 0.24 ms (20,000: 0.030
// ms), against 0.55 ms (0.049) in the caller's order with centres gathered by
// id.
__global__ void k_pu_gather(int64_t M, const int *__restrict__ torder,
                            const double4 *__restrict__ tgt, GridView cg, double r, double rinv,
                            const int64_t *__restrict__ toff, const int *__restrict__ tidx,
                            const double *__restrict__ local, int F, double *out) {
  // The M targets of torder: all, or those of a shard's list.
  for (int64_t it = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; it < M;
       it += (int64_t)gridDim.x * blockDim.x) {
    const int64_t t = torder[it];
    const double4 y = tgt[t];
    int ids[kMaxPatchesPerTarget];
    double ws[kMaxPatchesPerTarget];
    int cnt = 0;
    bool overflow = false;
    for_neighbors(cg, y.x, y.y, y.z, [&](const double4 &c) {
      const double d = __dsqrt_rn(sqdist3(y.x, y.y, y.z, c.x, c.y, c.z));
      if (d <= r) {
        const int k = int(c.w);
        if (cnt < kMaxPatchesPerTarget) {
          int j = cnt - 1;
          const double w = wendland<double>(kWendlandC2, d, rinv);
          while (j >= 0 && ids[j] > k) {
            ids[j + 1] = ids[j];
            ws[j + 1] = ws[j];
            --j;
          }
          ids[j + 1] = k;
          ws[j + 1] = w;
          ++cnt;
        } else {
          overflow = true;
        }
      }
    });
    double acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    if (!overflow) {
      double sum = 0.0;
      for (int i = 0; i < cnt; ++i) sum = __dadd_rn(sum, ws[i]);
      for (int i = 0; i < cnt; ++i) {
        const int k = ids[i];
        const int64_t b = toff[k];
        const int64_t pos = find_sorted(tidx + b, toff[k + 1] - b, int(t));
        if (pos < 0) continue;
        const double wn = __ddiv_rn(ws[i], sum);
        for (int f = 0; f < F; ++f)
          acc[f] = __dadd_rn(acc[f], __dmul_rn(wn, local[(b + pos) * F + f]));
      }
    } else {
      // More than kMaxPatchesPerTarget centres: walk them in ascending order
      // by repeated selection (same arithmetic, fewer registers).
      double sum = 0.0;
      int last = -1;
      for (;;) {
        int nk = 0x7fffffff;
        double nd = 0.0;
        for_neighbors(cg, y.x, y.y, y.z, [&](const double4 &c) {
          const int k = int(c.w);
          if (k > last && k < nk) {
            const double d = __dsqrt_rn(sqdist3(y.x, y.y, y.z, c.x, c.y, c.z));
            if (d <= r) {
              nk = k;
              nd = d;
            }
          }
        });
        if (nk == 0x7fffffff) break;
        sum = __dadd_rn(sum, wendland<double>(kWendlandC2, nd, rinv));
        last = nk;
      }
      last = -1;
      for (;;) {
        int nk = 0x7fffffff;
        double nd = 0.0;
        for_neighbors(cg, y.x, y.y, y.z, [&](const double4 &c) {
          const int k = int(c.w);
          if (k > last && k < nk) {
            const double d = __dsqrt_rn(sqdist3(y.x, y.y, y.z, c.x, c.y, c.z));
            if (d <= r) {
              nk = k;
              nd = d;
            }
          }
        });
        if (nk == 0x7fffffff) break;
        last = nk;
        const int64_t b = toff[nk];
        const int64_t pos = find_sorted(tidx + b, toff[nk + 1] - b, int(t));
        if (pos < 0) continue;
        const double wn = __ddiv_rn(wendland<double>(kWendlandC2, nd, rinv), sum);
        for (int f = 0; f < F; ++f)
          acc[f] = __dadd_rn(acc[f], __dmul_rn(wn, local[(b + pos) * F + f]));
      }
    }
    for (int f = 0; f < F; ++f) out[t * F + f] = acc[f];
  }
}

int neighbor_offsets(int dim, const int *shape, long long *off) {
  // ZCurveNeighborOffsets, clustering.hpp:34-116 (3D table :96-102).
  if (dim == 1) {
    off[0] = -1;
    off[1] = 1;
    return 2;
  }
  if (dim == 2) {
    static const int o2[8][2] = {{-1, -1}, {-1, 0}, {-1, 1}, {0, -1},
                                 {0, 1},   {1, -1}, {1, 0},  {1, 1}};
    for (int i = 0; i < 8; ++i) off[i] = o2[i][1] + (long long)o2[i][0] * shape[1];
    return 8;
  }
  static const int o3[26][3] = {{-1, -1, -1}, {-1, -1, 0}, {-1, -1, 1}, {-1, 0, 0},  {-1, 0, 1},
                                {-1, 0, -1},  {-1, 1, 0},  {-1, 1, 1},  {-1, 1, -1}, {0, -1, -1},
                                {0, -1, 0},   {0, -1, 1},  {0, 0, 1},   {0, 0, -1},  {0, 1, 0},
                                {0, 1, 1},    {0, 1, -1},  {1, -1, -1}, {1, -1, 0},  {1, -1, 1},
                                {1, 0, 0},    {1, 0, 1},   {1, 0, -1},  {1, 1, 0},   {1, 1, 1},
                                {1, 1, -1}};
  for (int i = 0; i < 26; ++i)
    off[i] = o3[i][2] + (long long)o3[i][1] * shape[2] + (long long)o3[i][0] * shape[2] * shape[1];
  return 26;
}

}  // namespace

// Full geometry phase on p.stream.  src_dev / tgt_dev are row-major device
// arrays of the caller's points.  About 27 launches and three waits (radius,
// number of centres, list sizes); 20,000 -> 20,000 uniform points: 0.33 ms of
// device time, against 62 launches and 0.88 ms with a kernel per radix digit,
// radix-sorted grids, a thread per re-tagged centre and segmented sorts.
void build_geometry(Plan &p, const double *src_dev, const double *tgt_dev) {
  cudaStream_t st = p.stream;
  const int dim = p.dim;
  const int64_t n = p.n, m = p.m;
  cudaEvent_t e0, e1;
  PB_CUDA(cudaEventCreate(&e0));
  PB_CUDA(cudaEventCreate(&e1));
  PB_CUDA(cudaEventRecord(e0, st));

  p.src4.alloc(sizeof(double4) * std::max<int64_t>(n, 1), st);
  p.tgt4.alloc(sizeof(double4) * std::max<int64_t>(m, 1), st);
  const double4 *src4 = p.src4.as<double4>(), *tgt4 = p.tgt4.as<double4>();
  DevMem scm;
  scm.alloc(sizeof(GeoScratch), st);
  GeoScratch *sc = scm.as<GeoScratch>();
  PB_CUDA(cudaMemsetAsync(sc, 0, kGeoZero, st));
  k_pack<<<dim3(grid_for(std::max(n, m), kThreads, 148 * 8), m > 0 ? 2 : 1), kThreads, 0, st>>>(
      src_dev, n, p.src4.as<double4>(), tgt_dev, m, p.tgt4.as<double4>(), dim, sc);

  // Patch radius.
  const long long kk = std::min<long long>(p.opts.nodes_per_cluster, n);
  const int nb_near = grid_for(n, kThreads, kNearBlocks);
  k_nearest<<<nb_near, kThreads, 0, st>>>(src4, n, dim, kk, sc);
  for (int pass = 0; pass < 2; ++pass)
    k_knn_hist<<<nb_near, kThreads, 0, st>>>(src4, n, dim, pass, sc);
  k_knn_gather<<<nb_near, kThreads, 0, st>>>(src4, n, dim, sc);
  note_launch(5);
  PB_CUDA(cudaGetLastError());
  GeoScratch *rs = static_cast<GeoScratch *>(HostArena::get().alloc(kGeoReport));
  PB_CUDA(cudaMemcpyAsync(rs, sc, kGeoReport, cudaMemcpyDeviceToHost, st));
  PB_CUDA(host_sync(st));
  if (rs->overflow) {  // many equal distances: the remaining digits one by one
    for (int pass = 2; pass < 8; ++pass)
      k_knn_hist<<<nb_near, kThreads, 0, st>>>(src4, n, dim, pass, sc);
    k_radius_final<<<1, 32, 0, st>>>(sc, dim);
    note_launch(7);
    PB_CUDA(cudaGetLastError());
    PB_CUDA(cudaMemcpyAsync(rs, sc, kGeoReport, cudaMemcpyDeviceToHost, st));
    PB_CUDA(host_sync(st));
  }
  for (int d = 0; d < 3; ++d) {
    p.lo[d] = rs->lo[d];
    p.hi[d] = rs->hi[d];
  }
  p.radius = rs->radius;
  if (std::getenv("PACMAN_B200_DEBUG")) {
    std::fprintf(stderr, "[pacman_b200] bbox lo %.17g %.17g %.17g hi %.17g %.17g %.17g\n",
                 rs->lo[0], rs->lo[1], rs->lo[2], rs->hi[0], rs->hi[1], rs->hi[2]);
    for (int s = 0; s < rs->nsamples; ++s)
      std::fprintf(stderr, "[pacman_b200] sample %d (%.17g %.17g %.17g) proj (%.17g %.17g %.17g) kth %.17g\n",
                   s, rs->samples[s][0], rs->samples[s][1], rs->samples[s][2], rs->proj[s][0],
                   rs->proj[s][1], rs->proj[s][2], rs->kth[s]);
    std::fprintf(stderr, "[pacman_b200] radius %.17g\n", rs->radius);
  }
  if (!(p.radius > 0.0) || !std::isfinite(p.radius))
    throw Error{PACMAN_B200_ERR_DEGENERATE, "degenerate patch radius (zero or non-finite)"};
  const double r = p.radius;
  const double r2 = r * r;

  // Candidate grid (clustering.hpp:142-203), host arithmetic as the reference.
  CandSpec cs{};
  cs.dim = dim;
  const double spacing = std::sqrt(4.0 / dim) * r * (1.0 - p.opts.relative_overlap);
  double min_d = 1.7976931348623157e308;
  long long nb = 1;
  for (int a = 0; a < 3; ++a) {
    cs.shape[a] = 1;
    cs.dist[a] = 0.0;
    cs.lo[a] = 0.0;
  }
  for (int a = 0; a < dim; ++a) {
    double edge = p.hi[a] - p.lo[a];
    edge = (edge < 0) ? -edge : edge;
    const double q = std::max(1.0, edge / spacing);
    if (!(q < 2.0e9)) throw Error{PACMAN_B200_ERR_LIMIT, "candidate centre grid too large"};
    cs.shape[a] = int(std::ceil(q));
    cs.dist[a] = edge / double(cs.shape[a]);
    if (cs.dist[a] < min_d) min_d = cs.dist[a];
    cs.shape[a] += 1;
    nb *= cs.shape[a];
    if (nb > 0x7fffffffll) throw Error{PACMAN_B200_ERR_LIMIT, "candidate centre grid exceeds int32"};
    cs.lo[a] = p.lo[a];
  }
  cs.r2 = r2;
  cs.nb = nb;
  p.ncand = nb;
  double thr = 0.4 * min_d;
  thr *= thr;

  // Both point sets sorted into cells, and the buffers of the cover.
  const GridSpec gs = make_grid_spec(dim, p.lo, p.hi, r, n);
  const GridSpec gt = make_grid_spec(dim, p.lo, p.hi, r, m);
  p.centers.alloc(sizeof(double4) * nb, st);
  DevMem mem;
  Slab slab;
  GridView sg{}, tg{};
  const double4 *sorted = nullptr;
  CoverReport *rep = nullptr;
  double4 *cpos = nullptr;
  unsigned char *s0 = nullptr, *s1 = nullptr, *flags = nullptr;
  unsigned int *mask = nullptr;
  int *pending = nullptr;
  void *tmp = nullptr;
  size_t tb = 0;
  for (int pass = 0; pass < 2; ++pass) {
    if (pass) {
      mem.alloc(slab.used, st);
      slab = Slab{mem.as<char>(), 0};
    }
    sort_into_cells(slab, src4, n, gs, tgt4, m, gt, sg, tg, sorted, st);
    rep = slab.take<CoverReport>(1);
    cpos = slab.take<double4>(nb);
    s0 = slab.take<unsigned char>(nb);
    s1 = slab.take<unsigned char>(nb);
    flags = slab.take<unsigned char>(nb);
    mask = slab.take<unsigned int>(nb);
    pending = slab.take<int>(nb);
    if (!pass)
      PB_CUDA(cub::DeviceSelect::Flagged(nullptr, tb, cpos, flags, p.centers.as<double4>(),
                                         &rep->K, int(nb), st));
    tmp = slab.take<char>(tb);
  }
  const int has_targets = m > 0 ? 1 : 0;
  p.torder.alloc(sizeof(int) * std::max<int64_t>(m, 1), st);
  if (m > 0) {
    k_ids<<<grid_for(m), kThreads, 0, st>>>(sorted + n, m, p.torder.as<int>());
    note_launch();
  }
  PruneOffsets po{};
  po.n = neighbor_offsets(dim, cs.shape, po.off);
  PB_CUDA(cudaMemsetAsync(rep, 0, sizeof(CoverReport), st));
  k_candidates<<<grid_for(nb * 32), kThreads, 0, st>>>(cs, sg, tg, sorted, src4, has_targets, cpos,
                                                       s0);
  k_prune_mark<<<grid_for(nb), kThreads, 0, st>>>(nb, po, thr, cpos, s0, s1, mask, pending, rep);
  k_prune_resolve<<<1, 1024, 0, st>>>(po, mask, pending, s1, rep);
  k_retag<<<grid_for(nb * 32), kThreads, 0, st>>>(nb, cpos, s1, tg, sorted, has_targets, r2,
                                                  flags);
  note_launch(4);
  // Step 11: stable compaction.
  PB_CUDA(cub::DeviceSelect::Flagged(tmp, tb, cpos, flags, p.centers.as<double4>(), &rep->K,
                                     int(nb), st));
  CoverReport *hr = static_cast<CoverReport *>(HostArena::get().alloc(sizeof(CoverReport)));
  PB_CUDA(cudaMemcpyAsync(hr, rep, sizeof(CoverReport), cudaMemcpyDeviceToHost, st));
  PB_CUDA(host_sync(st));
  if (hr->status) throw Error{PACMAN_B200_ERR_LIMIT, "centre pruning did not settle"};
  p.K = hr->K;

  build_lists(p, sg, tg, sorted, r);

  // Grid of centres for the partition-of-unity weights.
  build_grid(p.cgrid, p.centers.as<double4>(), p.K, dim, p.lo, p.hi, r, st);
  PB_CUDA(cudaEventRecord(e1, st));
  // No wait here: the time is read after the execute's own final wait.
  p.geom_ev[0] = e0;
  p.geom_ev[1] = e1;
}

double geometry_ms(Plan &p) {
  if (p.geom_ev[0] && p.geom_ev[1] && cudaEventQuery(p.geom_ev[1]) == cudaSuccess) {
    float ms = 0.f;
    if (cudaEventElapsedTime(&ms, p.geom_ev[0], p.geom_ev[1]) == cudaSuccess) p.ms_geometry = ms;
    cudaEventDestroy(p.geom_ev[0]);
    cudaEventDestroy(p.geom_ev[1]);
    p.geom_ev[0] = p.geom_ev[1] = nullptr;
  }
  cudaGetLastError();
  return p.ms_geometry < 0.0 ? 0.0 : p.ms_geometry;
}

// Both point sets packed and sorted into the cells of the sources' grid, for
// the nearest-neighbour searches of nearest.cu and mls.cu.  `scale` is the
// cell's edge relative to one source per cell of a uniform cloud.
void build_point_search(PointSearch &ps, int dim, const double *src_dev, int64_t n,
                        const double *tgt_dev, int64_t m, double scale, cudaStream_t st) {
  DevMem scm;
  scm.alloc(sizeof(GeoScratch), st);
  GeoScratch *sc = scm.as<GeoScratch>();
  ps.src4.alloc(sizeof(double4) * std::max<int64_t>(n, 1), st);
  ps.tgt4.alloc(sizeof(double4) * std::max<int64_t>(m, 1), st);
  PB_CUDA(cudaMemsetAsync(sc->box, 0, sizeof(sc->box), st));
  k_pack<<<dim3(grid_for(std::max(n, m), kThreads, 148 * 8), m > 0 ? 2 : 1), kThreads, 0, st>>>(
      src_dev, n, ps.src4.as<double4>(), tgt_dev, m, ps.tgt4.as<double4>(), dim, sc);
  note_launch();
  auto *h = static_cast<unsigned long long *>(HostArena::get().alloc(sizeof(sc->box)));
  PB_CUDA(cudaMemcpyAsync(h, sc->box, sizeof(sc->box), cudaMemcpyDeviceToHost, st));
  PB_CUDA(host_sync(st));
  auto to_dbl = [](unsigned long long b) {
    b = (b & 0x8000000000000000ull) ? (b & 0x7fffffffffffffffull) : ~b;
    double d;
    std::memcpy(&d, &b, sizeof(d));
    return d;
  };
  double lo[3] = {0, 0, 0}, hi[3] = {0, 0, 0}, ext = 0.0;
  for (int d = 0; d < dim; ++d) {
    lo[d] = to_dbl(~h[d]);
    hi[d] = to_dbl(h[3 + d]);
    ext = std::max(ext, hi[d] - lo[d]);
  }
  const double per_axis = std::ceil(std::pow(double(n), 1.0 / dim));
  const double cell = ext > 0.0 ? scale * (ext / per_axis) : 1.0;
  const GridSpec g = make_grid_spec(dim, lo, hi, cell, n);
  GridSpec gt = g;
  gt.clamp = 1;
  Slab slab;
  GridView tv{};
  for (int pass = 0; pass < 2; ++pass) {
    if (pass) {
      ps.mem.alloc(slab.used, st);
      slab = Slab{ps.mem.as<char>(), 0};
    }
    sort_into_cells(slab, ps.src4.as<double4>(), n, g, ps.tgt4.as<double4>(), m, gt, ps.grid, tv,
                    ps.sorted, st);
  }
}

void pu_gather(Plan &p, const double *local, int F, double *out_dev) {
  if (p.m == 0) return;
  const bool sharded = p.m_owned >= 0;
  if (p.K == 0 || sharded)  // a shard writes its own targets only: zeros elsewhere
    PB_CUDA(cudaMemsetAsync(out_dev, 0, sizeof(double) * p.m * F, p.stream));
  if (p.K == 0) return;
  const int64_t M = sharded ? p.m_owned : p.m;
  if (M == 0) return;
  const double r = p.radius;
  k_pu_gather<<<grid_for(M, 128, 148 * 64), 128, 0, p.stream>>>(
      M, sharded ? p.tlist.as<int>() : p.torder.as<int>(), p.tgt4.as<double4>(), p.cgrid.view, r,
      1.0 / r, p.toff.as<int64_t>(), p.tidx.as<int>(), local, F, out_dev);
  note_launch();
  PB_CUDA(cudaGetLastError());
}

}  // namespace pacman_b200
