// Minimum-image pair statistics of a batch of configurations: the pair
// distance histogram and the nearest-neighbour distances that the ground-state
// driver writes as g2 and Hp tables.
//
// Reference: src/xla_cco/analysis/pairs.py:41-128 (nearest_neighbor_distances,
// pair_distance_histogram) with the distance rule of _block_distances
// (:173-188): ds = s_j - s_i, ds -= round(ds), the 3^d image shifts of ds
// mapped through the basis, the smallest |r|^2, then sqrt; a particle's own
// zero shift is excluded. Binning follows np.histogram (_bin_counts,
// :191-199): bins are [e_k, e_k+1), the last one closed.
//
// Two shortcuts give the same bits as the rule above:
//  * On a diagonal basis the zero shift of ds in [-1/2, 1/2] is the smallest
//    image: |ds| <= |ds + s| for s = +-1 holds component by component, and
//    rounded products, squares and sums are monotone. One image instead of
//    3^d; a sheared basis keeps the 3^d shifts.
//  * sqrt is correctly rounded and monotone, so r >= e is r2 >= t(e) with
//    t(e) the smallest double whose square root is at least e. The edges
//    become thresholds on r2 (found on the host), and the kernels take no square
//    root per pair. The bin is a guess from an FP32 square root, walked to the
//    exact place (uniform edges, kept in shared memory), or a binary search.
//
// Layout: a CTA of 128 threads takes a range of the upper-triangle pairs of
// 128-particle tiles of one configuration, the column tile staged in shared
// memory, a row per thread. The histogram keeps the CTA's bins in shared memory
// (32-bit, at most one count per pair of its range) and adds them into the
// 64-bit result once, so the counts are exact and independent of the launch
// order. On 256 configurations of d=2 N=1000 (200 bins) histogram and nearest
// neighbours went from 1423 and 1712 us to 235 and 254 us; bound: instruction
// issue (FP64: 6 operations per axis and pair). The column loops are not unrolled
// over 27 images: four times over, nearest neighbours of 8 sheared configurations of
// d=3 N=900 take 584 us instead of 505 (9 images: 164 unrolled, 208 not). Screening
// pairs by FP32 distances of fixed-point differences first ran 272 and 242 us
// (conversions) and was not kept.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <vector>

#include "cco.h"
#include "cco_host.cuh"

namespace cco {
namespace {

constexpr int kPairTile = 128;        // rows per CTA = columns per staged tile
constexpr int kSmemBins = 8192;       // bins kept in shared memory (32 KB)
constexpr int kSmemEdges = 1024;      // thresholds kept in shared memory (8 KB)
constexpr int kMaxUnits = 1 << 17;    // tile pairs of a CTA: 32-bit bins cannot overflow
constexpr int kPairCtas = 148 * 16;   // CTAs to aim for

// The smallest double t >= 0 with sqrt(t) >= e (e >= 0), or > e with `past`: a few
// steps over neighbouring doubles (consecutive bit patterns) from e^2.
__host__ __device__ inline double r2_threshold(double e, bool past) {
  union {
    double x;
    unsigned long long u;
  } t, below;
  t.x = e * e;
  while (!(past ? sqrt(t.x) > e : sqrt(t.x) >= e) && t.x < INFINITY) ++t.u;
  for (; t.u > 0; --t.u) {
    below.u = t.u - 1;
    if (!(past ? sqrt(below.x) > e : sqrt(below.x) >= e)) break;
  }
  return t.x;
}

struct PairGeom {
  double B[9];   // basis rows (lattice vectors), row-major d x d
  int n, n_bins;
  float e0, inv_w;   // uniform edges: first edge, 1 / width (inv_w = 0: not uniform)
};

template <int D>
__device__ __forceinline__ double min_image_r2(const double* si, const double* sj,
                                               const PairGeom& g, bool self) {
  double ds[D];
#pragma unroll
  for (int c = 0; c < D; ++c) {
    const double t = __dadd_rn(sj[c], -si[c]);
    ds[c] = __dadd_rn(t, -rint(t));
  }
  double best = INFINITY;
  constexpr int kShifts = D == 1 ? 3 : (D == 2 ? 9 : 27);
#pragma unroll
  for (int q = 0; q < kShifts; ++q) {
    int rem = q;
    double x[D];
    bool zero = true;
#pragma unroll
    for (int c = 0; c < D; ++c) {
      const int sh = rem % 3 - 1;
      rem /= 3;
      zero &= sh == 0;
      x[c] = __dadd_rn(ds[c], (double)sh);
    }
    if (self && zero) continue;
    double r2 = 0.0;
#pragma unroll
    for (int a = 0; a < D; ++a) {
      double v = 0.0;
#pragma unroll
      for (int c = 0; c < D; ++c) v = __dadd_rn(v, __dmul_rn(x[c], g.B[c * D + a]));
      r2 = __dadd_rn(r2, __dmul_rn(v, v));
    }
    best = fmin(best, r2);
  }
  return best;
}

// r2 of the zero shift on a diagonal basis. SMALL: |t| < 2^51, where the nearest
// integer is two additions instead of a quarter-rate rounding instruction.
template <int D, bool SMALL = false>
__device__ __forceinline__ double diag_r2(const double* si, const double* sj, const double* Bd) {
  double r2 = 0.0;
#pragma unroll
  for (int c = 0; c < D; ++c) {
    const double t = __dadd_rn(sj[c], -si[c]);
    const double k = SMALL ? __dadd_rn(__dadd_rn(t, 0x1.8p52), -0x1.8p52) : rint(t);
    const double v = __dmul_rn(__dadd_rn(t, -k), Bd[c]);
    r2 = __dadd_rn(r2, __dmul_rn(v, v));
  }
  return r2;
}

// np.histogram bin of a pair with t[0] <= r2 < t[n_bins] (t[k]: the threshold
// of edge k; t[n_bins]: of the first r past the last edge, which belongs to the
// last bin): the largest k with t[k] <= r2.
__device__ __forceinline__ int bin_of(double r2, const double* t, const PairGeom& g) {
  if (g.inv_w > 0.f) {
    const float f = (float)r2;
    int k = (int)((f * rsqrtf(f) - g.e0) * g.inv_w);   // a zero r2 gives NaN, bin 0
    k = min(max(k, 0), g.n_bins - 1);
    while (t[k] > r2) --k;
    while (k + 1 < g.n_bins && t[k + 1] <= r2) ++k;
    return k;
  }
  int lo = 0, hi = g.n_bins;   // invariant: t[lo] <= r2 < t[hi]
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (t[mid] <= r2) lo = mid;
    else hi = mid;
  }
  return lo;
}

// Edges to thresholds in place. From kSmemEdges bins on, where the kernels read them
// from global memory, on the device: 8192 took the host 100 to 160 us.
__global__ void k_thresholds(double* t, int n) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < n) t[k] = r2_threshold(t[k], k == n - 1);
}

// Unit u of the upper triangle of tiles x tiles, row by row: (ti, tj >= ti).
__device__ __forceinline__ void pair_unit(long long u, int tiles, int& ti, int& tj) {
  ti = 0;
  while (u >= tiles - ti) u -= tiles - ti++;
  tj = ti + (int)u;
}

template <int D, bool DIAG>
__global__ void __launch_bounds__(kPairTile) k_pair_hist(const double* __restrict__ s, PairGeom g,
                                                         const double* __restrict__ thresholds,
                                                         unsigned long long* counts, int tiles) {
  extern __shared__ double sm[];   // thresholds (if they fit), then the bins
  __shared__ double col[kPairTile * D];
  // In-range pairs of a warp queue up and are binned 32 at a time: with a tenth
  // of the pairs in range nearly every step of a warp has one, and binning it at
  // once would cost every step the whole path (408 against 235 us).
  __shared__ double queues[kPairTile / 32][64];
  const bool local = g.n_bins <= kSmemBins, tl = g.n_bins < kSmemEdges;
  const double* t = tl ? sm : thresholds;
  unsigned int* bins = reinterpret_cast<unsigned int*>(sm + (tl ? g.n_bins + 1 : 0));
  if (tl)
    for (int b = threadIdx.x; b <= g.n_bins; b += blockDim.x) sm[b] = thresholds[b];
  if (local)
    for (int b = threadIdx.x; b < g.n_bins; b += blockDim.x) bins[b] = 0u;
  const double t_lo = thresholds[0], t_hi = thresholds[g.n_bins];
  double Bd[D];
#pragma unroll
  for (int c = 0; c < D; ++c) Bd[c] = g.B[c * D + c];
  const double* sc = s + (size_t)blockIdx.y * g.n * D;
  const long long units = (long long)tiles * (tiles + 1) / 2;
  const long long u0 = units * blockIdx.x / gridDim.x, u1 = units * (blockIdx.x + 1) / gridDim.x;
  double* queue = queues[threadIdx.x >> 5];
  const int wl = threadIdx.x & 31;
  const unsigned below = (1u << wl) - 1u;
  int have = 0;
  auto count = [&](double r2) {
    const int b = bin_of(r2, t, g);
    if (local) atomicAdd(bins + b, 1u);
    else atomicAdd(counts + b, 1ull);
  };
  int ti, tj;
  pair_unit(u0, tiles, ti, tj);
  for (long long u = u0; u < u1; ++u) {
    const int j0 = tj * kPairTile, nj = min(kPairTile, g.n - j0);
    __syncthreads();
    for (int q = threadIdx.x; q < nj * D; q += blockDim.x) col[q] = sc[(size_t)j0 * D + q];
    __syncthreads();
    const int i = ti * kPairTile + threadIdx.x;
    double si[D];
#pragma unroll
    for (int c = 0; c < D; ++c) si[c] = i < g.n ? sc[(size_t)i * D + c] : 0.0;
    // the row's first column: past the diagonal, past the end for a dead row
    const int first = i >= g.n ? nj : tj == ti ? (int)threadIdx.x + 1 : 0;
#pragma unroll (DIAG || D < 3 ? 4 : 1)
    for (int jj = 0; jj < nj; ++jj) {
      const double r2 = DIAG ? diag_r2<D>(si, col + jj * D, Bd)
                             : min_image_r2<D>(si, col + jj * D, g, false);
      const bool in = jj >= first && r2 >= t_lo && r2 < t_hi;   // false for NaN
      const unsigned m = __ballot_sync(0xffffffffu, in);
      if (in) queue[have + __popc(m & below)] = r2;
      have += __popc(m);
      if (have >= 32) {
        __syncwarp();
        count(queue[wl]);
        have -= 32;
        const double rest = queue[32 + wl];
        __syncwarp();
        if (wl < have) queue[wl] = rest;
      }
    }
    if (++tj == tiles) tj = ++ti;
  }
  __syncwarp();
  if (wl < have) count(queue[wl]);
  if (!local) return;
  __syncthreads();
  for (int b = threadIdx.x; b < g.n_bins; b += blockDim.x)
    if (bins[b]) atomicAdd(counts + b, (unsigned long long)bins[b]);
}

template <int D, bool DIAG>
__global__ void __launch_bounds__(kPairTile) k_nearest(const double* __restrict__ s, PairGeom g,
                                                       double* __restrict__ out) {
  __shared__ double col[kPairTile * D];
  const double* sc = s + (size_t)blockIdx.y * g.n * D;
  const int i = blockIdx.x * kPairTile + threadIdx.x;
  double si[D], Bd[D];
#pragma unroll
  for (int c = 0; c < D; ++c) {
    si[c] = i < g.n ? sc[(size_t)i * D + c] : 0.0;
    Bd[c] = g.B[c * D + c];
  }
  // a particle's own nearest image, then every other particle
  double best = min_image_r2<D>(si, si, g, true);
  for (int j0 = 0; j0 < g.n; j0 += kPairTile) {
    const int nj = min(kPairTile, g.n - j0);
    __syncthreads();
    for (int u = threadIdx.x; u < nj * D; u += blockDim.x) col[u] = sc[(size_t)j0 * D + u];
    __syncthreads();
    const int self = i - j0;
#pragma unroll (DIAG || D < 3 ? 4 : 1)
    for (int jj = 0; jj < nj; ++jj) {
      const double r2 = DIAG ? diag_r2<D>(si, col + jj * D, Bd)
                             : min_image_r2<D>(si, col + jj * D, g, false);
      if (jj != self) best = fmin(best, r2);
    }
  }
  if (i < g.n) out[(size_t)blockIdx.y * g.n + i] = sqrt(best);
}

// ------------------------------------------------------------ cell grids
// Diagonal bases, configurations that fit shared memory: every CTA sorts its
// configuration into a grid of cells and a row looks only at the cells a
// partner within range (or nearer than what it has) can be in. A pair that is
// skipped lies more than K cells apart on some axis; with |s| <= 2^16 its
// distance as computed exceeds K / G L by no less than kCellMargin, so the
// counts and the smallest distances stay those of all pairs. A configuration
// with larger or non-finite coordinates, or most of its particles in a few
// cells, takes one cell, all pairs.
// 256 configurations of d=2 N=1000, range 0.2 L, 200 bins: histogram 235 -> 85 us
// (a ninth of the pairs; 200 us while every tested pair took FP64 and the queue,
// 133 with the FP32 screen before the queue; 93 / 82 us with 256 / 1024 threads,
// cells of a half / a third / a quarter of the range 103 / 93 / 92), nearest
// neighbours 254 -> 37 us, about half of it the sort. Instruction issue bounds
// both. The all-pairs kernels below stay for sheared bases, ranges that reach
// most of the box, fewer than 64 particles and configurations past shared memory.
constexpr int kCellThreads = 512;
constexpr double kCellReach = 65536.0;     // largest |s| of a cell grid
constexpr double kCellMargin = 1e-7;       // relative: |s| rounding 2^-37, G <= 2048
constexpr double kCellLeast = 1e-7;        // shortest FP32 distance / longest axis
constexpr int kMaxCells = 8192, kMaxAxisCells = 2048;
constexpr size_t kCellSmem = 200 * 1024;
// cells per histogram range, at least: in 1-D a row's cells are one span, so that
// finer ones cost nothing (one configuration of N=6000, range 0.4 L: 12 / 24 / 48
// cells 263 / 147 / 96 us; 256 of N=1000, 0.2 L: 140 / 136 / 109)
constexpr double kHistReach = 3.0, kHistReach1 = 48.0;
constexpr double kHistFill = 4.0, kNearFill = 2.0;   // particles per cell, at least / about
// Stencil / box. In 1-D the range's pairs then cost what all pairs do (four
// configurations of N=9000, range 0.4 L: all pairs 537 us, cells 1150).
constexpr double kHistMost = 1.0, kHistMost1 = 0.6, kNearMost = 0.5;
constexpr int kHistCells1 = 512;       // 1-D cells, at most
constexpr int kCellMin = 64, kCellCtas = 148 * 3, kCellSplit = 96;
constexpr int kCellCrowd = 64;

struct CellGrid {
  int G[3], K[3], cells;   // cells per axis, stencil reach, all cells
  float lim;               // histogram: FP32 r2 no pair in range exceeds
  float least;             // FP32 r2 below which a pair counts as that far apart: of the
                           // box's own size, so that every allowance scales with it
  float eps;               // and bins around an edge that FP32 cannot tell (0: queue every pair)
  float part;              // stencil / box
};

template <int D>
__device__ __forceinline__ int cell_of(const double* s, const int* G, int* c) {
  int id = 0;
#pragma unroll
  for (int a = 0; a < D; ++a) {
    const double u = s[a] - floor(s[a]);
    c[a] = min(max((int)(u * G[a]), 0), G[a] - 1);
    id = id * G[a] + c[a];
  }
  return id;
}

// Sorts the configuration by cell: positions to ps, rows to idx (optional),
// end[c] = one past the last particle of cell c. The order inside a cell is any,
// so CTAs that share a configuration split it at cells (cell_range). A
// configuration outside the reach, or with a crowded cell, keeps its order in
// one cell (G = 1, K = 0). Returns the grid in use. All threads of the CTA.
template <int D>
__device__ CellGrid cell_sort(const double* __restrict__ s, int n, CellGrid g, double* ps, int* end,
                              int* idx) {
  __shared__ int wsum[kCellThreads / 32];
  const int tid = threadIdx.x;
  int cc[3];
  auto load = [&](int j, double* x) {
    bool in = true;
#pragma unroll
    for (int a = 0; a < D; ++a) {
      x[a] = s[(size_t)j * D + a];
      in = in && fabs(x[a]) <= kCellReach;
    }
    return in ? cell_of<D>(x, g.G, cc) : -1;
  };
  for (int c = tid; c < g.cells; c += kCellThreads) end[c] = 0;
  __syncthreads();
  int bad = 0;
  const int crowd = kCellCrowd + 4 * n / g.cells;
  for (int j = tid; j < n; j += kCellThreads) {
    double x[D];
    const int c = load(j, x);
    bad |= c < 0;
    if (c >= 0) bad |= atomicAdd(end + c, 1) >= crowd;
  }
  if (__syncthreads_or(bad)) {
    for (int q = tid; q < n * D; q += kCellThreads) ps[q] = s[q];
    if (idx)
      for (int j = tid; j < n; j += kCellThreads) idx[j] = j;
    if (tid == 0) end[0] = n;
    __syncthreads();
    for (int a = 0; a < 3; ++a) {
      g.G[a] = 1;
      g.K[a] = 0;
    }
    g.cells = 1;
    return g;
  }
  // exclusive prefix sums: a run of cells per thread
  const int per = (g.cells + kCellThreads - 1) / kCellThreads;
  const int c0 = min(tid * per, g.cells), c1 = min(c0 + per, g.cells);
  int sum = 0;
  for (int c = c0; c < c1; ++c) sum += end[c];
  int incl = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, o);
    if ((tid & 31) >= o) incl += v;
  }
  if ((tid & 31) == 31) wsum[tid >> 5] = incl;
  __syncthreads();
  int at = incl - sum;
  for (int w = 0; w < tid >> 5; ++w) at += wsum[w];
  for (int c = c0; c < c1; ++c) {
    const int v = end[c];
    end[c] = at;
    at += v;
  }
  __syncthreads();
  for (int j = tid; j < n; j += kCellThreads) {
    double x[D];
    const int to = atomicAdd(end + load(j, x), 1);   // leaves end[c] at the cell's end
#pragma unroll
    for (int a = 0; a < D; ++a) ps[to * D + a] = x[a];
    if (idx) idx[to] = j;
  }
  __syncthreads();
  return g;
}

// The particles of this CTA (of gridDim.x): an even split, moved back to the
// start of a cell.
__device__ __forceinline__ int cell_range(const CellGrid& g, const int* end, int n, int part) {
  const int p = (int)((long long)n * part / gridDim.x);
  if (g.cells == 1 || p == 0 || p == n) return p;
  int lo = 0, hi = g.cells - 1;   // the first cell that ends past p
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (end[mid] > p) hi = mid;
    else lo = mid + 1;
  }
  return lo > 0 ? end[lo - 1] : 0;
}

// Particles of columns [c - lo, c + hi] (wrapped) of the cell row `row`:
// [a, a + n1) and [b, b + n2).
struct CellSpan {
  int a, n1, b, n2;
};
__device__ __forceinline__ CellSpan cell_span(const int* end, int row, int G, int c, int lo, int hi) {
  const int base = row * G;
  auto begin = [&](int k) { return base + k > 0 ? end[base + k - 1] : 0; };
  CellSpan r;
  const int f = c - lo, l = c + hi;
  r.a = begin(max(f, 0));
  r.n1 = end[base + min(l, G - 1)] - r.a;
  r.b = 0;
  r.n2 = 0;
  if (f < 0) {
    r.b = begin(f + G);
    r.n2 = end[base + G - 1] - r.b;
  } else if (l >= G) {
    r.b = begin(0);
    r.n2 = end[base + l - G] - r.b;
  }
  return r;
}

__device__ __forceinline__ int wrap(int x, int G) { return x < 0 ? x + G : x >= G ? x - G : x; }

// The histogram over half the stencil: the rest of the row's own cell, the
// cells after it, the cell rows after its own. Lanes are neighbours in the sorted
// order, so their partners are mostly the same. A pair is screened by the FP32
// distance of wrapped coordinates (the image is known from the cells; lim
// allows for their rounding, 1e-6 L). On even edges one that lies more than eps
// bins from every edge is counted at once; the others that pass queue up per
// warp, 32 at a time are measured in FP64 and binned.
template <int D, bool SLICED>
__global__ void __launch_bounds__(kCellThreads)
    k_pair_hist_cells(const double* __restrict__ s, PairGeom g, CellGrid grid,
                      const double* __restrict__ thresholds, unsigned long long* counts) {
  // positions, thresholds (if they fit), FP32 wrapped positions, cell ends, bins
  extern __shared__ double sm[];
  __shared__ unsigned int queues[kCellThreads / 32][64];
  const bool local = g.n_bins <= kSmemBins, tl = g.n_bins < kSmemEdges;
  double* ps = sm;
  double* ts = ps + (size_t)g.n * D;
  const double* t = tl ? ts : thresholds;
  float* pf = reinterpret_cast<float*>(ts + (tl ? g.n_bins + 1 : 0));
  int* end = reinterpret_cast<int*>(pf + (size_t)(g.n + 1) / 2 * 2 * D);
  unsigned int* bins = reinterpret_cast<unsigned int*>(end + grid.cells);
  if (tl)
    for (int b = threadIdx.x; b <= g.n_bins; b += kCellThreads) ts[b] = thresholds[b];
  if (local)
    for (int b = threadIdx.x; b < g.n_bins; b += kCellThreads) bins[b] = 0u;
  const CellGrid cg = cell_sort<D>(s + (size_t)blockIdx.y * g.n * D, g.n, grid, ps, end, nullptr);
  const double t_lo = t[0], t_hi = t[g.n_bins];
  double Bd[D];
  float L[D];
#pragma unroll
  for (int c = 0; c < D; ++c) {
    Bd[c] = g.B[c * D + c];
    L[c] = (float)fabs(Bd[c]);
  }
  const float lim = cg.cells > 1 ? cg.lim : INFINITY;   // one cell: every pair is measured
  for (int q = threadIdx.x; q < g.n * D; q += kCellThreads)
    pf[q] = cg.cells > 1 ? (float)((ps[q] - floor(ps[q])) * fabs(g.B[(q % D) * (D + 1)])) : 0.f;
  __syncthreads();
  // the bin less 1/2 is r inv_w + shift; within `half` of its nearest integer the bin is sure
  const bool direct = cg.cells > 1 && cg.eps > 0.f;
  const float shift = -g.e0 * g.inv_w - 0.5f, half = 0.5f - cg.eps;
  unsigned int* queue = queues[threadIdx.x >> 5];
  const int wl = threadIdx.x & 31;
  const unsigned below = (1u << wl) - 1u;
  int have = 0;
  auto count = [&](unsigned int ij) {
    const double *si = ps + (ij >> 16) * D, *sj = ps + (ij & 0xffffu) * D;
    const double r2 = cg.cells > 1 ? diag_r2<D, true>(si, sj, Bd) : diag_r2<D>(si, sj, Bd);
    if (!(r2 >= t_lo && r2 < t_hi)) return;   // out of range or NaN
    const int b = bin_of(r2, t, g);
    if (local) atomicAdd(bins + b, 1u);
    else atomicAdd(counts + b, 1ull);
  };
  const int rows = D == 1 ? 1 : D == 2 ? cg.K[0] + 1 : cg.K[1] + 1 + cg.K[0] * (2 * cg.K[1] + 1);
  const int ib = cell_range(cg, end, g.n, blockIdx.x), i1 = cell_range(cg, end, g.n, blockIdx.x + 1);
  // the CTA's particles, a warp each 32. SLICED (a CTA has few of them): several warps
  // share 32 particles and take a slice of every span each
  const int groups = SLICED ? (i1 - ib + 31) >> 5 : 0;
  const int slices = SLICED ? max(1, kCellThreads / 32 / max(groups, 1)) : 1;
  for (int u = threadIdx.x & ~31;; u += kCellThreads) {   // the warp's first thread
    int i0 = ib + u, sl = 0;
    if (SLICED) {
      if (u >= 32 * groups * slices) break;
      sl = u / max(32 * groups, 1);
      i0 -= 32 * groups * sl;
    } else if (i0 >= i1) {
      break;
    }
    const int i = i0 + wl;
    const bool live = i < i1;
    double si[D];
#pragma unroll
    for (int c = 0; c < D; ++c) si[c] = ps[(live ? i : 0) * D + c];
    int cc[3] = {0, 0, 0};
    if (cg.cells > 1) cell_of<D>(si, cg.G, cc);
    for (int q = 0; q < rows; ++q) {
      float x[D];   // this row's image of the particle
#pragma unroll
      for (int c = 0; c < D; ++c) x[c] = pf[(live ? i : 0) * D + c];
      int row = 0;
      if (D == 2) {
        row = wrap(cc[0] + q, cg.G[0]);
        if (cc[0] + q >= cg.G[0]) x[0] -= L[0];
      }
      if (D == 3) {
        const int w = 2 * cg.K[1] + 1, q1 = q - (cg.K[1] + 1);
        const int r0 = cc[0] + (q1 < 0 ? 0 : q1 / w + 1), r1 = cc[1] + (q1 < 0 ? q : q1 % w - cg.K[1]);
        row = wrap(r0, cg.G[0]) * cg.G[1] + wrap(r1, cg.G[1]);
        if (r0 >= cg.G[0]) x[0] -= L[0];
        if (r1 >= cg.G[1]) x[1] -= L[1];
        if (r1 < 0) x[1] += L[1];
      }
      const int lo = q == 0 ? 0 : cg.K[D - 1];
      CellSpan sp = cell_span(end, row, cg.G[D - 1], cc[D - 1], lo, cg.K[D - 1]);
      if (q == 0) {   // the rest of its own cell first
        sp.n1 -= i + 1 - sp.a;
        sp.a = i + 1;
      }
      const int len = live ? sp.n1 + sp.n2 : 0, gap = sp.b - sp.a - sp.n1;
      const float x2 = cc[D - 1] < lo ? x[D - 1] + L[D - 1] : x[D - 1] - L[D - 1];   // of the second span
      int k0 = 0, most = __reduce_max_sync(0xffffffffu, len);
      if (SLICED) {
        k0 = most * sl / slices;
        most = most * (sl + 1) / slices;
      }
      auto at = [&](int k) { return k < len ? sp.a + k + (k >= sp.n1 ? gap : 0) : 0; };
      auto screen = [&](int k, int j) {
        float r2 = 0.f;
#pragma unroll
        for (int c = 0; c < D; ++c) {
          const float v = pf[j * D + c] - (c == D - 1 && k >= sp.n1 ? x2 : x[c]);
          r2 = fmaf(v, v, r2);
        }
        return r2;
      };
      auto push = [&](bool in, int j) {
        const unsigned m = __ballot_sync(0xffffffffu, in);
        if (in) queue[have + __popc(m & below)] = (unsigned)i << 16 | (unsigned)j;
        have += __popc(m);
        if (have >= 32) {
          __syncwarp();
          count(queue[wl]);
          have -= 32;
          const unsigned rest = queue[32 + wl];
          __syncwarp();
          if (wl < have) queue[wl] = rest;
        }
      };
      if (direct) {
#pragma unroll 4
        for (int k = k0; k < most; ++k) {
          const int j = at(k);
          const float r2 = fmaxf(screen(k, j), cg.least);
          const float u = fmaf(r2 * rsqrtf(r2), g.inv_w, shift);   // bin - 1/2
          const float n = u + 0x1.8p23f;                           // its nearest integer
          const int b = __float_as_int(n) - 0x4b400000;
          const bool edge = fabsf(u - (n - 0x1.8p23f)) >= half;
          const bool in = k < len && r2 <= lim;
          if (in && !edge && (unsigned)b < (unsigned)g.n_bins) atomicAdd(bins + b, 1u);
          if (__any_sync(0xffffffffu, in && edge)) push(in && edge, j);
        }
      } else {
#pragma unroll 4
        for (int k = k0; k < most; ++k) {
          const int j = at(k);
          push(k < len && screen(k, j) <= lim, j);
        }
      }
    }
  }
  __syncwarp();
  if (wl < have) count(queue[wl]);
  if (!local) return;
  __syncthreads();
  for (int b = threadIdx.x; b < g.n_bins; b += kCellThreads)
    if (bins[b]) atomicAdd(counts + b, (unsigned long long)bins[b]);
}

// Nearest neighbours: the 3^D cells around a particle, then 5^D if the best
// could be beaten from outside, then everything.
template <int D>
__global__ void __launch_bounds__(kCellThreads)
    k_nearest_cells(const double* __restrict__ s, PairGeom g, CellGrid grid, double* __restrict__ out) {
  extern __shared__ double sm[];   // positions, cell ends, rows
  double* ps = sm;
  int* end = reinterpret_cast<int*>(ps + (size_t)g.n * D);
  int* idx = end + grid.cells;
  const CellGrid cg = cell_sort<D>(s + (size_t)blockIdx.y * g.n * D, g.n, grid, ps, end, idx);
  double Bd[D], side = INFINITY;
  int gmin = 1 << 30;
#pragma unroll
  for (int c = 0; c < D; ++c) {
    Bd[c] = g.B[c * D + c];
    side = fmin(side, fabs(Bd[c]) / cg.G[c] * (1.0 - kCellMargin));
    gmin = min(gmin, cg.G[c]);
  }
  const int i1 = cell_range(cg, end, g.n, blockIdx.x + 1);
  for (int i = cell_range(cg, end, g.n, blockIdx.x) + threadIdx.x; i < i1; i += kCellThreads) {
    double si[D];
#pragma unroll
    for (int c = 0; c < D; ++c) si[c] = ps[i * D + c];
    double best = min_image_r2<D>(si, si, g, true);   // its own nearest image
    int cc[3] = {0, 0, 0};
    if (cg.cells > 1) cell_of<D>(si, cg.G, cc);
    auto visit = [&](int j) {
      const double r2 = diag_r2<D, true>(si, ps + j * D, Bd);
      if (j != i) best = fmin(best, r2);
    };
    bool done = false;
    for (int K = 1; K <= 2 && !done && gmin >= 2 * K + 1; ++K) {
      const int w = 2 * K + 1, rows = D == 1 ? 1 : D == 2 ? w : w * w;
      for (int q = 0; q < rows; ++q) {
        int row = 0;
        if (D == 2) row = wrap(cc[0] + q - K, cg.G[0]);
        if (D == 3) row = wrap(cc[0] + q / w - K, cg.G[0]) * cg.G[1] + wrap(cc[1] + q % w - K, cg.G[1]);
        const CellSpan sp = cell_span(end, row, cg.G[D - 1], cc[D - 1], K, K);
        for (int k = 0; k < sp.n1; ++k) visit(sp.a + k);
        for (int k = 0; k < sp.n2; ++k) visit(sp.b + k);
      }
      const double reach = K * side;
      done = best <= reach * reach * (1.0 - kCellMargin);
    }
    if (!done)
      for (int j = 0; j < g.n; ++j) {
        const double r2 = diag_r2<D>(si, ps + j * D, Bd);
        if (j != i) best = fmin(best, r2);
      }
    out[(size_t)blockIdx.y * g.n + idx[i]] = sqrt(best);
  }
}

// Cell grid with cells of about `side`; reach > 0: K covers it, else K = 1. False
// if the stencil covers too much of the box or the configuration is too large
// or too small.
bool cell_grid(const PairGeom& g, int d, double side, double reach, double most, CellGrid* c) {
  *c = CellGrid{{1, 1, 1}, {0, 0, 0}, 1, 0.f, 0.f, 0.f, 1.f};
  double part = 1.0, longest = 0.0;
  if (!(side > 0.0) || g.n > 0xffff) return false;
  for (int a = 0; a < d; ++a) {
    const double L = std::fabs(g.B[a * d + a]);
    const double n = std::floor(L / side);
    if (!(n >= 3.0 && L > 1e-12 && L < 1e12)) return false;
    longest = std::max(longest, L);
    c->G[a] = (int)std::min<double>(n, kMaxAxisCells);
    const double k = reach > 0.0 ? std::ceil(reach * c->G[a] / (L * (1.0 - kCellMargin))) : 1.0;
    if (!(2.0 * k + 1.0 <= c->G[a])) return false;
    c->K[a] = (int)k;
    part *= (2.0 * k + 1.0) / c->G[a];
    if ((double)c->cells * c->G[a] > kMaxCells) return false;
    c->cells *= c->G[a];
  }
  const double r = reach + 1e-6 * longest;
  c->lim = (float)(r * r * (1.0 + 1e-6));
  c->least = (float)(kCellLeast * longest * kCellLeast * longest);
  c->part = (float)part;
  return part <= most;
}

// CTAs per configuration of a histogram on cells: 96 particles each, fewer (32 at
// least) while that leaves SMs without one, more when the batch alone fills the GPU
// (one / 16 configurations of d=2 N=1000, range 0.28 L: 96 particles 24.9 / 31.4 us,
// 32 particles 20.6 / 37.7).
int hist_chunks(int n, int batch) {
  const int few = (n + kCellSplit - 1) / kCellSplit, most = (n + 31) / 32;
  const int chunks = std::min(most, std::max(few, 148 / batch));
  return std::max(1, std::min(chunks, (kCellCtas + batch - 1) / batch));
}

// Whether a histogram takes cells: an estimate of both forms' time in us, fitted to
// ranges of 5 to 45% of the box, 64 to 9000 particles and 1 to 256 configurations.
// All pairs: a cost per pair of the tiles and per pair in range. Cells: the CTAs'
// sorts, then the stencil's pairs at the rate of the CTAs that have cells of their
// own, at most the GPU's. One configuration of d=2 N=6000, range 0.05 / 0.2 / 0.28 /
// 0.4 L: all pairs 37 / 42 / 46 / 56 us, cells 23 / 45 / 67 / 173; 256 of N=1000: 200 /
// 234 / 264 / 332 against 38 / 93 / 149 / 312; 64 of d=3 N=500, 0.05 / 0.2: 32 / 34
// against 32 / 60.
bool cells_pay(int n, int batch, int d, const CellGrid& c, double range, double vol, size_t smem) {
  const double pairs = 0.5 * n * n * batch;
  const double ball = d == 1 ? 2.0 * range : d == 2 ? M_PI * range * range : 4.0 / 3.0 * M_PI * range * range * range;
  const double in = std::min(1.0, ball / vol);
  const double tiles = (n + kPairTile - 1) / kPairTile;
  const double tested = 0.5 * tiles * (tiles + 1) * kPairTile * kPairTile * batch;
  const double all = std::max(24.0 + 16.0 * in,
                              8.0 + tested * (d == 1 ? 1.15e-6 : d == 2 ? 1.3e-6 : 1.6e-6) + pairs * in * 2.1e-6);
  const int ctas = hist_chunks(n, batch);
  const double fit = std::max<double>(1.0, std::min<double>(4.0, std::floor(227.0 * 1024 / (smem + 6 * 1024))));
  const double per_sm = std::min(fit, ctas * (double)batch / 148);
  const double busy = (double)std::min(ctas, c.cells) * batch;
  const double rate = std::min(4e5, (d == 1 ? 1300.0 : d == 2 ? 2000.0 : 800.0) * busy);
  return 0.9 * (10.0 + per_sm * (4.0 + 2e-3 * n) + pairs * c.part / rate) < all;
}

bool is_diagonal(const PairGeom& g, int d) {
  for (int r = 0; r < d; ++r)
    for (int c = 0; c < d; ++c)
      if (r != c && g.B[r * d + c] != 0.0) return false;
  return true;
}

template <int D>
void launch_hist(bool diag, dim3 grid, size_t smem, cudaStream_t st, const double* s,
                 const PairGeom& g, const double* t, unsigned long long* c, int tiles) {
  if (diag) k_pair_hist<D, true><<<grid, kPairTile, smem, st>>>(s, g, t, c, tiles);
  else k_pair_hist<D, false><<<grid, kPairTile, smem, st>>>(s, g, t, c, tiles);
}
template <int D>
cudaError_t launch_hist_cells(dim3 grid, size_t smem, cudaStream_t st, const double* s, const PairGeom& g,
                              const CellGrid& c, const double* t, unsigned long long* out) {
  // two warps or more for every 32 particles, and SMs with warps to spare (256
  // configurations of d=2 N=300, three CTAs an SM: 97 us sliced, 91 not)
  const bool sliced = (size_t)g.n <= (size_t)grid.x * (kCellThreads / 2) && grid.x * grid.y <= 2 * 148;
  const auto kernel = sliced ? k_pair_hist_cells<D, true> : k_pair_hist_cells<D, false>;
  static OncePerDevice once;
  const cudaError_t e = once.run([] {
    const cudaError_t a = cudaFuncSetAttribute(k_pair_hist_cells<D, true>,
                                               cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kCellSmem);
    return a != cudaSuccess ? a
                            : cudaFuncSetAttribute(k_pair_hist_cells<D, false>,
                                                   cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kCellSmem);
  });
  if (e == cudaSuccess) kernel<<<grid, kCellThreads, smem, st>>>(s, g, c, t, out);
  return e;
}
template <int D>
cudaError_t launch_nearest_cells(dim3 grid, size_t smem, cudaStream_t st, const double* s,
                                 const PairGeom& g, const CellGrid& c, double* out) {
  static OncePerDevice once;   // on every call it is 0.7 of 18 us
  const cudaError_t e = once.run([] {
    return cudaFuncSetAttribute(k_nearest_cells<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kCellSmem);
  });
  if (e == cudaSuccess) k_nearest_cells<D><<<grid, kCellThreads, smem, st>>>(s, g, c, out);
  return e;
}
template <int D>
void launch_nearest(bool diag, dim3 grid, cudaStream_t st, const double* s, const PairGeom& g,
                    double* out) {
  if (diag) k_nearest<D, true><<<grid, kPairTile, 0, st>>>(s, g, out);
  else k_nearest<D, false><<<grid, kPairTile, 0, st>>>(s, g, out);
}

int pair_args(int device, int batch, int n, int d, const double* s, const double* basis,
              PairGeom* g) {
  if (d < 1 || d > 3) return fail(CCO_ERR_ARG, "d must be 1, 2 or 3, got %d", d);
  if (batch < 1 || n < 1) return fail(CCO_ERR_ARG, "need batch >= 1 and n >= 1");
  if (batch > 65535) return fail(CCO_ERR_ARG, "batch %d above 65535: split it", batch);
  if (!s || !basis) return fail(CCO_ERR_ARG, "null positions or basis");
  int ndev = 0;
  if (cco_device_count(&ndev) != CCO_OK) return CCO_ERR_NODEVICE;
  if (device < 0 || device >= ndev) return fail(CCO_ERR_ARG, "device %d out of range", device);
  *g = PairGeom{};
  for (int k = 0; k < d * d; ++k) {
    if (!std::isfinite(basis[k])) return fail(CCO_ERR_ARG, "non-finite basis entry %d", k);
    g->B[k] = basis[k];
  }
  g->n = n;
  return CCO_OK;
}

}  // namespace
}  // namespace cco

using namespace cco;

extern "C" {

int cco_pair_histogram(int device, void* stream, int batch, int n, int d, const double* s,
                       const double* basis, int n_edges, const double* edges, int64_t* counts) {
  PairGeom g;
  const int rc = pair_args(device, batch, n, d, s, basis, &g);
  if (rc != CCO_OK) return rc;
  if (n_edges < 2 || !edges || !counts) return fail(CCO_ERR_ARG, "need >= 2 edges and a counts array");
  for (int k = 0; k < n_edges; ++k) {
    if (!std::isfinite(edges[k]) || edges[k] < 0.0)
      return fail(CCO_ERR_ARG, "edges must be finite and non-negative");
    if (k > 0 && !(edges[k] > edges[k - 1])) return fail(CCO_ERR_ARG, "edges must be strictly increasing");
  }
  g.n_bins = n_edges - 1;
  const bool host_thresholds = g.n_bins < kSmemEdges;
  std::vector<double> ht(edges, edges + n_edges);
  if (host_thresholds)
    for (int k = 0; k < n_edges; ++k) ht[k] = r2_threshold(edges[k], k == g.n_bins);
  // evenly spaced edges (within half a bin): the guess is off by a few bins at most
  const double width = (edges[g.n_bins] - edges[0]) / g.n_bins;
  bool even = width > 1e-30 && edges[g.n_bins] < 1e18 && edges[g.n_bins] < 1e5 * width;
  for (int k = 0; k < n_edges && even; ++k)
    even = std::fabs(edges[k] - (edges[0] + k * width)) <= 0.5 * width;
  if (even) {
    g.e0 = (float)edges[0];
    g.inv_w = (float)(1.0 / width);
  }
  DeviceGuard guard(device);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  double* d_t = nullptr;
  CCO_CUDA(upload(&d_t, ht, st));
  if (!host_thresholds) k_thresholds<<<(n_edges + 127) / 128, 128, 0, st>>>(d_t, n_edges);
  CCO_CUDA(cudaMemsetAsync(counts, 0, sizeof(int64_t) * g.n_bins, st));
  const bool diag = is_diagonal(g, d);
  auto* c = reinterpret_cast<unsigned long long*>(counts);
  const size_t bin_smem = (g.n_bins < kSmemEdges ? sizeof(double) * n_edges : 0) +
                          (g.n_bins <= kSmemBins ? sizeof(unsigned int) * g.n_bins : 0);
  double vol = 1.0;
  for (int a = 0; a < d; ++a) vol *= std::fabs(g.B[a * d + a]);
  double side = std::max(edges[g.n_bins] / (d == 1 ? kHistReach1 : kHistReach) * (1.0 + 4.0 * kCellMargin),
                         std::pow(kHistFill * vol / n, 1.0 / d));
  if (d == 1) side = std::max(side, vol / kHistCells1);
  // FP32 bins: what rounding and the shortest distance can move a pair by, and the
  // edges against the even ones
  double dev = 0.0, longest = 0.0;
  for (int k = 0; k < n_edges; ++k) dev = std::max(dev, std::fabs(edges[k] - (edges[0] + k * width)));
  for (int a = 0; a < d; ++a) longest = std::max(longest, std::fabs(g.B[a * d + a]));
  const double eps = 1.01 * ((1e-6 + kCellLeast) * longest + 1e-6 * edges[g.n_bins] + dev) / width;
  CellGrid cg;
  const size_t pos_smem = sizeof(double) * n * d + sizeof(float) * ((n + 1) / 2 * 2) * d;
  const size_t cell_smem = pos_smem + bin_smem + sizeof(int) * kMaxCells;
  if (diag && n >= kCellMin && cell_smem <= kCellSmem &&
      cell_grid(g, d, side, edges[g.n_bins], d == 1 ? kHistMost1 : kHistMost, &cg) &&
      cells_pay(n, batch, d, cg, edges[g.n_bins], vol, pos_smem + bin_smem + sizeof(int) * cg.cells)) {
    const dim3 grid(hist_chunks(n, batch), batch);
    const size_t smem = pos_smem + bin_smem + sizeof(int) * cg.cells;
    if (even && g.n_bins <= kSmemBins && eps < 0.1) cg.eps = (float)eps;
    CCO_CUDA(d == 1   ? launch_hist_cells<1>(grid, smem, st, s, g, cg, d_t, c)
             : d == 2 ? launch_hist_cells<2>(grid, smem, st, s, g, cg, d_t, c)
                      : launch_hist_cells<3>(grid, smem, st, s, g, cg, d_t, c));
    CCO_CUDA(cudaGetLastError());
    CCO_CUDA(cudaFreeAsync(d_t, st));
    return CCO_OK;
  }
  const int tiles = (n + kPairTile - 1) / kPairTile;
  const long long units = (long long)tiles * (tiles + 1) / 2;
  // a CTA's range: enough CTAs to fill the GPU a few times, few flushes of the bins
  long long ctas = std::min<long long>(units, (kPairCtas + batch - 1) / batch);
  ctas = std::max(ctas, (units + kMaxUnits - 1) / kMaxUnits);
  const dim3 grid((unsigned)ctas, batch);
  const size_t smem = bin_smem;
  if (d == 1) launch_hist<1>(diag, grid, smem, st, s, g, d_t, c, tiles);
  else if (d == 2) launch_hist<2>(diag, grid, smem, st, s, g, d_t, c, tiles);
  else launch_hist<3>(diag, grid, smem, st, s, g, d_t, c, tiles);
  CCO_CUDA(cudaGetLastError());
  CCO_CUDA(cudaFreeAsync(d_t, st));
  return CCO_OK;
}

int cco_nearest_neighbor(int device, void* stream, int batch, int n, int d, const double* s,
                         const double* basis, double* out) {
  PairGeom g;
  const int rc = pair_args(device, batch, n, d, s, basis, &g);
  if (rc != CCO_OK) return rc;
  if (!out) return fail(CCO_ERR_ARG, "null output");
  DeviceGuard guard(device);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const bool diag = is_diagonal(g, d);
  double vol = 1.0;
  for (int a = 0; a < d; ++a) vol *= std::fabs(g.B[a * d + a]);
  CellGrid cg;
  const size_t cell_smem = (sizeof(double) * d + sizeof(int)) * n + sizeof(int) * kMaxCells;
  if (diag && n >= kCellMin && cell_smem <= kCellSmem &&
      cell_grid(g, d, std::pow(kNearFill * vol / n, 1.0 / d), 0.0, kNearMost, &cg)) {
    const int chunks = (n + kCellSplit - 1) / kCellSplit;
    const dim3 grid(std::max(1, std::min(chunks, (kCellCtas + batch - 1) / batch)), batch);
    const size_t smem = (sizeof(double) * d + sizeof(int)) * n + sizeof(int) * cg.cells;
    CCO_CUDA(d == 1   ? launch_nearest_cells<1>(grid, smem, st, s, g, cg, out)
             : d == 2 ? launch_nearest_cells<2>(grid, smem, st, s, g, cg, out)
                      : launch_nearest_cells<3>(grid, smem, st, s, g, cg, out));
    CCO_CUDA(cudaGetLastError());
    return CCO_OK;
  }
  const dim3 grid((n + kPairTile - 1) / kPairTile, batch);
  if (d == 1) launch_nearest<1>(diag, grid, st, s, g, out);
  else if (d == 2) launch_nearest<2>(diag, grid, st, s, g, out);
  else launch_nearest<3>(diag, grid, st, s, g, out);
  CCO_CUDA(cudaGetLastError());
  return CCO_OK;
}

}  // extern "C"
