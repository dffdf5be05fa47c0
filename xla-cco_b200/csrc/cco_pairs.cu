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
// issue (FP64: 6 operations per axis and pair). Screening pairs by FP32 distances
// of fixed-point differences first ran 272 and 242 us (conversions) and was not kept.
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

// r2 of the zero shift on a diagonal basis.
template <int D>
__device__ __forceinline__ double diag_r2(const double* si, const double* sj, const double* Bd) {
  double r2 = 0.0;
#pragma unroll
  for (int c = 0; c < D; ++c) {
    const double t = __dadd_rn(sj[c], -si[c]);
    const double v = __dmul_rn(__dadd_rn(t, -rint(t)), Bd[c]);
    r2 = __dadd_rn(r2, __dmul_rn(v, v));
  }
  return r2;
}

// np.histogram bin of a pair with t[0] <= r2 < t[n_bins] (t[k]: the threshold
// of edge k; t[n_bins]: of the first r past the last edge, which belongs to the
// last bin): the largest k with t[k] <= r2.
__device__ __forceinline__ int bin_of(double r2, const double* t, const PairGeom& g) {
  if (g.inv_w > 0.f) {
    int k = (int)((sqrtf((float)r2) - g.e0) * g.inv_w);
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
#pragma unroll 4
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
#pragma unroll 4
    for (int jj = 0; jj < nj; ++jj) {
      const double r2 = DIAG ? diag_r2<D>(si, col + jj * D, Bd)
                             : min_image_r2<D>(si, col + jj * D, g, false);
      if (jj != self) best = fmin(best, r2);
    }
  }
  if (i < g.n) out[(size_t)blockIdx.y * g.n + i] = sqrt(best);
}

// The smallest double t >= 0 with sqrt(t) >= e (e >= 0), or > e with `past`.
double r2_threshold(double e, bool past) {
  auto in = [&](double t) { return past ? std::sqrt(t) > e : std::sqrt(t) >= e; };
  double t = e * e;
  while (!in(t) && std::isfinite(t)) t = std::nextafter(t, INFINITY);
  while (t > 0.0 && in(std::nextafter(t, 0.0))) t = std::nextafter(t, 0.0);
  return t;
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
  std::vector<double> ht(n_edges);
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
  CCO_CUDA(cudaMemsetAsync(counts, 0, sizeof(int64_t) * g.n_bins, st));
  const int tiles = (n + kPairTile - 1) / kPairTile;
  const long long units = (long long)tiles * (tiles + 1) / 2;
  // a CTA's range: enough CTAs to fill the GPU a few times, few flushes of the bins
  long long ctas = std::min<long long>(units, (kPairCtas + batch - 1) / batch);
  ctas = std::max(ctas, (units + kMaxUnits - 1) / kMaxUnits);
  const dim3 grid((unsigned)ctas, batch);
  const size_t smem = (g.n_bins < kSmemEdges ? sizeof(double) * n_edges : 0) +
                      (g.n_bins <= kSmemBins ? sizeof(unsigned int) * g.n_bins : 0);
  auto* c = reinterpret_cast<unsigned long long*>(counts);
  const bool diag = is_diagonal(g, d);
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
  const dim3 grid((n + kPairTile - 1) / kPairTile, batch);
  const bool diag = is_diagonal(g, d);
  if (d == 1) launch_nearest<1>(diag, grid, st, s, g, out);
  else if (d == 2) launch_nearest<2>(diag, grid, st, s, g, out);
  else launch_nearest<3>(diag, grid, st, s, g, out);
  CCO_CUDA(cudaGetLastError());
  return CCO_OK;
}

}  // extern "C"
