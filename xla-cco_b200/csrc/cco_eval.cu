// Stealthy energy, gradient and collective density on sm_100a (FP64).
//
// Reference math (src/xla_cco/energy.py:45-50,195-225,301-324):
//   rho_k  = sum_j exp(2 pi i n_k . s_j)
//   Phi    = (1/V) sum_k w_k |rho_k|^2
//   dPhi/ds_j = (2 (2 pi) / V) sum_k w_k (Im rho_k cos th_kj - Re rho_k sin th_kj) n_k
//
// B200 formulation. The k-set is stored as runs of consecutive last-axis n
// with a fixed prefix (n_0..n_{d-2}); along a run the phase advances by one
// complex multiply, exp(i th_{k+1,j}) = exp(i th_kj) z_j, z_j = exp(2 pi i
// s_{j,d-1}). A segment start takes its phase from per-particle tables in
// shared memory: z_a^|n| = prod_l T_a,l[digit_l(|n|)]. Table entries come
// from FP64 sincospi of the exact integer exponent (the product e s reduced
// without rounding, sincos_2pi_ms), re-seeded every 8 entries
// with products in between, so a phase carries O(10 eps) error on top of the
// <= segment-length products along a run - inside the reference's eps |theta|
// trig error. No theta matrix ever reaches HBM: traffic per evaluation is s
// in, g out and the M-row density, so both passes are FP64-pipe bound.
//
// Dense k-sets run both FP64 passes on the matrix pipe instead (k_grid1 and
// k_grid2, cco_grid.cuh); the recurrences below serve sparse k-sets (more than
// two grid slots per row) and FP32 lanes.
//
//   pass 1 (k_pass1): CTA = (configuration, 64-particle tile), 128 threads.
//     A thread owns a segment of <= 8 rows and streams the tile's particles
//     four at a time (four independent phase chains), accumulating 8 complex
//     sums in registers: no cross-thread reduction. Small k-sets split the
//     particles into slices summed in a fixed order. Output: one partial
//     density row per tile.
//   reduce  (k_reduce): sums the tile rows in tile order (deterministic),
//     forms rho, w rho and Phi (fixed-order block sum).
//   pass 2 (k_pass2): CTA = (configuration, 128-particle tile), one particle
//     per thread; the CTA walks the segments two at a time (two independent
//     chains per thread; density reads are warp-uniform broadcasts, fetched
//     two rows ahead). Per row: one complex multiply, the coefficient
//     w(Im rho cos - Re rho sin) and two accumulations; prefix axes are
//     weighted once per segment.
#include <algorithm>
#include <vector>
#include <cstdio>
#include <cstdlib>

#include "cco_eval_bodies.cuh"
#include "cco_grid.cuh"
#include "cco_internal.cuh"

namespace cco {

namespace {

constexpr int kGridSms = 148;                      // SMs of a B200


// An FP64 lane that is still to be evaluated.
__device__ __forceinline__ bool grid_lane_runs(const EvalPlan& plan, const EvalLane& ln) {
  return lane_active(ln.status) && !(plan.dyn_prec && lane_prec(ln) == PREC_FP32);
}

// Grid form: the phases the tables start from.
__global__ void __launch_bounds__(kRootChunk) k_grid_roots(EvalPlan plan) {
  chain_wait<CHAIN_FEW>();
  const EvalLane& ln = plan.lanes[blockIdx.y];
  if (!grid_lane_runs(plan, ln)) return;
  const ProbDev& P = plan.probs[ln.prob];
  const int w = blockIdx.x * kRootChunk + threadIdx.x;
  if (!P.grid || w >= P.groots * P.N) return;
  if (P.d == 1) grid_roots<1>(P, ln, w);
  else if (P.d == 2) grid_roots<2>(P, ln, w);
  else grid_roots<3>(P, ln, w);
}

// Grid form (cco_grid.cuh), pass 1: one kernel per (dimension, class), each
// holding the accumulators of 2 or 3 tiles per warp. Persistent: four CTAs of
// four warps per SM walk the items.
template <int D, int CLS>
__global__ void __launch_bounds__(kGridThreads, kGridCtas) k_grid1(EvalPlan plan) {
  extern __shared__ double2 smem[];
  __shared__ GridStage stage;
  constexpr bool LINES = CLS == kGridLines, ROOTS = CLS > 0 && !LINES;
  constexpr int NT = CLS == 2 ? 3 : LINES ? 1 : 2;
  const EvalItem* items = plan.itemsG + plan.q_offG[D - 1][CLS];
  const int n = plan.q_offG[D - 1][CLS + 1] - plan.q_offG[D - 1][CLS];
  chain_wait<CHAIN_LATE>();
  for (int i = blockIdx.x; i < n; i += gridDim.x) {
    const EvalItem it = items[i];
    const EvalLane ln = plan.lanes[it.lane];
    if (!grid_lane_runs(plan, ln)) continue;   // FP32 lanes: k_pass1
    const ProbDev& P = plan.probs[ln.prob];
    grid_pass1<D, ROOTS, NT, LINES>(P, ln, it.tile / P.ngblk, it.tile % P.ngblk, stage, smem);
  }
}

int grid_ctas(int items) { return std::min(items, kGridCtas * kGridSms); }

template <int D, int CLS>
void launch_grid1_class(const EvalPlan& plan, cudaStream_t s) {
  const int n = plan.q_offG[D - 1][CLS + 1] - plan.q_offG[D - 1][CLS];
  if (n > 0) launch_chained(plan.chain, k_grid1<D, CLS>, grid_ctas(n), kGridThreads, plan.smemG, s, plan);
}
template <int D>
void launch_grid1(const EvalPlan& plan, cudaStream_t s) {
  launch_grid1_class<D, 0>(plan, s);
  launch_grid1_class<D, 1>(plan, s);
  launch_grid1_class<D, 2>(plan, s);
  if constexpr (D > 1) launch_grid1_class<D, kGridLines>(plan, s);
}

// One kernel per dimension D and arithmetic keeps each kernel's code small:
// the instruction cache holds one body instead of all of them. F32 = false
// evaluates the FP64 lanes of a launch, F32 = true its FP32 lanes (a plan with
// FP32 lanes launches both). An FP64 lane therefore always runs the same
// kernel, in a mixed-precision run and in a plain one, and gets the same bits.
template <int D, bool F32>
__global__ void __launch_bounds__(kPass1Threads, 4) k_pass1(EvalPlan plan) {
  extern __shared__ double2 smem[];
  __shared__ ProbDev sp;
  chain_wait();
  const EvalItem it = plan.items1[plan.d_off1[D - 1] + blockIdx.x];
  const EvalLane ln = plan.lanes[it.lane];
  if (!lane_active(ln.status)) return;
  if ((lane_prec(ln) == PREC_FP32) != F32) return;   // the other kernel's lane
  if (threadIdx.x == 0) sp = plan.probs[ln.prob];
  __syncthreads();
  if (F32) {
    pass1_body_f32<D>(sp, ln, it.tile, smem);
  } else if (!sp.grid) {   // grid problems: k_grid1
    const int C = pass1_chunks(sp, plan.chunks1);
    pass1_body<D>(sp, ln, it.tile / C, smem, it.tile % C, C);
  }
}

// Chunk energies of a grid-form lane: after the pass-2 weights.
__device__ __forceinline__ double* grid_energies(const ProbDev& P, const EvalLane& ln) {
  return reinterpret_cast<double*>(
      ln.rhow + (P.grid == 2 ? (size_t)P.M : (size_t)P.gslots * (P.d == 1 ? 2 : 4)));
}

// Reduction (grid: chunks x lanes): rho_k = sum over tiles of the pass-1
// partials in tile order, the weighted density for pass 2, and this chunk's
// part of sum w |rho|^2, stored over the chunk's first partial (which only
// this block reads).
__global__ void __launch_bounds__(kReduceChunk) k_reduce(EvalPlan plan) {
  __shared__ double red[32];
  chain_wait<CHAIN_FEW>();
  const EvalLane ln = plan.lanes[blockIdx.y];
  if (!lane_active(ln.status)) return;
  const ProbDev& P = plan.probs[ln.prob];
  if (P.grid && lane_prec(ln) == PREC_FP64) {
    if ((int)(blockIdx.x * kReduceChunk) >= P.gslots) return;
    const int slot = blockIdx.x * kReduceChunk + threadIdx.x;
    double e = 0.0;
    if (slot < P.gslots) {
      if (P.d == 1) e = grid_reduce_slot<true>(P, ln, slot);
      else e = grid_reduce_slot<false>(P, ln, slot);
    }
    e = block_sum(e, red);
    if (threadIdx.x == 0) grid_energies(P, ln)[blockIdx.x] = e;
    return;
  }
  const int M = P.M, nt = P.ntile1;
  const int k0 = blockIdx.x * kReduceChunk;
  if (k0 >= M) return;
  const int k = k0 + threadIdx.x;
  double e = 0.0;
  if (k < M) {
    const double2* __restrict__ col = ln.part + k;
    double2 t = col[0];
    int q = 1;
    // sixteen tile rows in flight per step, added in tile order (the same sums
    // as one row at a time; a lone lane of many tiles is latency-bound here)
    for (; q + 16 <= nt; q += 16) {
      double2 o[16];
#pragma unroll
      for (int u = 0; u < 16; ++u) o[u] = col[(size_t)(q + u) * M];
#pragma unroll
      for (int u = 0; u < 16; ++u) {
        t.x += o[u].x;
        t.y += o[u].y;
      }
    }
    for (; q < nt; ++q) {
      const double2 o = col[(size_t)q * M];
      t.x += o.x;
      t.y += o.y;
    }
    ln.rho[k] = t;
    const double wk = P.w_run[k];
    if (lane_prec(ln) == PREC_FP32)
      reinterpret_cast<float2*>(ln.rhow)[k] = make_float2((float)(wk * t.x), (float)(wk * t.y));
    else
      ln.rhow[k] = make_double2(wk * t.x, wk * t.y);
    e = wk * (t.x * t.x + t.y * t.y);
  }
  e = block_sum(e, red);
  if (threadIdx.x == 0) ln.part[k0] = make_double2(e, 0.0);
}

// Energy of one lane (one warp): the chunk energies summed in a fixed order.
__device__ __forceinline__ void lane_energy(const EvalPlan& plan, const EvalLane& ln) {
  const ProbDev& P = plan.probs[ln.prob];
  const int wl = threadIdx.x & 31;
  double e = 0.0;
  if (P.grid && lane_prec(ln) == PREC_FP64) {
    const double* ec = grid_energies(P, ln);
    const int nc = reduce_chunks(P.gslots);
    for (int c = wl; c < nc; c += 32) e += ec[c];
  } else {
    const int nc = reduce_chunks(P.M);
    for (int c = wl; c < nc; c += 32) e += ln.part[(size_t)c * kReduceChunk].x;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
  if (wl == 0) *ln.f = e / P.vol;
}

// Energy-only evaluations (no pass 2): one warp per lane. With the gradient,
// the first warp of each lane's first pass-2 tile sums it instead (one launch
// fewer per evaluation, the same sum).
__global__ void k_energy(EvalPlan plan) {
  chain_wait();
  const EvalLane ln = plan.lanes[blockIdx.x];
  if (!lane_active(ln.status)) return;
  lane_energy(plan, ln);
}

// Grid form, pass 2.
template <int D, bool ROOTS>
__global__ void __launch_bounds__(kGridThreads, kGridCtas) k_grid2(EvalPlan plan) {
  extern __shared__ double2 smem[];
  __shared__ GridStage stage;
  const EvalItem* items = plan.itemsH + plan.h_off[D - 1][ROOTS];
  const int n = plan.h_off[D - 1][ROOTS + 1] - plan.h_off[D - 1][ROOTS];
  chain_wait<CHAIN_LATE>();
  for (int i = blockIdx.x; i < n; i += gridDim.x) {
    const EvalItem it = items[i];
    const EvalLane ln = plan.lanes[it.lane];
    if (!grid_lane_runs(plan, ln)) continue;   // FP32 lanes: k_pass2
    if (it.tile == 0 && threadIdx.x < 32) lane_energy(plan, ln);
    if (ln.g) grid_pass2<D, ROOTS>(plan.probs[ln.prob], ln, it.tile, stage, smem);
  }
}

template <int D, bool F32>
__global__ void __launch_bounds__(kPass2Threads, 4) k_pass2(EvalPlan plan) {
  extern __shared__ double2 smem[];
  __shared__ ProbDev sp;
  chain_wait();
  const EvalItem it = plan.items2[plan.d_off2[D - 1] + blockIdx.x];
  const EvalLane ln = plan.lanes[it.lane];
  if (!lane_active(ln.status)) return;
  if ((lane_prec(ln) == PREC_FP32) != F32) return;   // the other kernel's lane
  if (!F32 && plan.probs[ln.prob].grid == 1) return;      // grid problems: k_grid2
  if (it.tile == 0 && threadIdx.x < 32) lane_energy(plan, ln);
  if (ln.g == nullptr) return;
  if (threadIdx.x == 0) sp = plan.probs[ln.prob];
  __syncthreads();
  if (D == 1 && !F32) {
    if ((size_t)sp.M * sizeof(double2) <= kPass2RhoStage1D)
      pass2_body_1d<true>(sp, ln, it.tile, plan.split2, smem);
    else
      pass2_body_1d<false>(sp, ln, it.tile, plan.split2, smem);
    return;
  }
  const bool staged = (size_t)sp.M * sizeof(double2) <= kPass2RhoStage;
  if (F32) {
    if (staged)
      pass2_body_f32<D, true>(sp, ln, it.tile, plan.split2, smem);
    else
      pass2_body_f32<D, false>(sp, ln, it.tile, plan.split2, smem);
    return;
  }
  if (staged)
    pass2_body<D, true>(sp, ln, it.tile, plan.split2, smem);
  else
    pass2_body<D, false>(sp, ln, it.tile, plan.split2, smem);
}

__global__ void k_rho_scatter(const double2* __restrict__ rho, const int* __restrict__ run2ref,
                              int M, int batch, size_t lane_stride, double* re, double* im) {
  const size_t total = (size_t)M * batch;
  for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < total;
       t += (size_t)gridDim.x * blockDim.x) {
    const int b = (int)(t / M), k = (int)(t - (size_t)b * M);
    const double2 v = rho[(size_t)b * lane_stride + k];
    const size_t o = (size_t)b * M + run2ref[k];
    if (re) re[o] = v.x;
    if (im) im[o] = v.y;
  }
}

__global__ void k_rho_rows(const double2* __restrict__ rho, const int* __restrict__ row_of,
                           int total, int M, double n, double* re, double* im) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x, b = blockIdx.y;
  if (c >= total) return;
  const int k = row_of[c];
  const double2 v = k >= 0 ? rho[(size_t)b * M + k] : make_double2(n, 0.0);
  if (re) re[(size_t)b * total + c] = v.x;
  if (im) im[(size_t)b * total + c] = v.y;
}

// One thread per row walks the batch, eight densities in flight, so the sums
// are a sequential scan of the configurations. One pass over the densities
// where separate array operations took three launches per configuration.
__global__ void k_structure_sums(const double2* __restrict__ rho, const int* __restrict__ run2ref,
                                 int M, double n, int batch, double* tot, double* tot2) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= M) return;
  const int o = run2ref[k];
  double t = tot[o], t2 = tot2[o];
  for (int b0 = 0; b0 < batch; b0 += 8) {
    double2 v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (b0 + u < batch) v[u] = rho[(size_t)(b0 + u) * M + k];
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (b0 + u < batch) {
        const double sk = __dadd_rn(__dmul_rn(v[u].x, v[u].x), __dmul_rn(v[u].y, v[u].y)) / n;
        t = __dadd_rn(t, sk);
        t2 = __dadd_rn(t2, __dmul_rn(sk, sk));
      }
  }
  tot[o] = t;
  tot2[o] = t2;
}

}  // namespace

int pass1_slices(int nseg, int nj) {
  int ns = 1;
  while (2 * ns * nseg <= kPass1Threads && 2 * ns <= nj) ns *= 2;
  return ns;
}

size_t eval_smem1(const ProbDev& p) {
  const int ns = pass1_slices(p.nseg1, kPass1Tile);
  const size_t red = ns > 1 ? (size_t)ns * p.nseg1 * kSeg1Len : 0;
  return ((size_t)p.t1.nrows * kPass1Stride + red) * sizeof(double2);
}

size_t eval_smemG(const ProbDev& p) {
  return p.grid ? (size_t)kGridChunk * p.gts * sizeof(double2) : 0;
}

size_t eval_smemH(const ProbDev& p) {
  return p.grid ? (size_t)kGridTile2 * p.gts * sizeof(double2) : 0;
}

size_t eval_smem2(const ProbDev& p, int split, bool f32) {
  if (p.d == 1 && !f32) {   // pass2_body_1d: the staged density and the slice combine
    const size_t rho = (size_t)p.M * sizeof(double2);
    const size_t comb = split > 1 ? (size_t)kPass2Tile * sizeof(double) : 0;
    return (rho <= kPass2RhoStage1D ? rho : 0) + comb;
  }
  const size_t rho = (size_t)p.M * sizeof(double2);
  const size_t comb = split > 1 ? (size_t)kPass2Tile * p.d * sizeof(double) : 0;
  return (size_t)p.t2.nrows * (kPass2Tile / split) * sizeof(double2) +
         (rho <= kPass2RhoStage ? rho : 0) + comb;
}

int pass2_tiles(const ProbDev& p, int split) {
  const int tw = kPass2Tile / split;
  return (p.N + tw - 1) / tw;
}

int pass2_split(long long tiles_at_split1) {
  if (const char* env = getenv("CCO_PASS2_SPLIT")) {
    const int s = atoi(env);
    if (s == 1 || s == 2 || s == 4 || s == 8) return s;
  }
  int split = 1;
  while (split < 8 && tiles_at_split1 * split < kPass2TargetCtas) split *= 2;
  return split;
}

namespace {

template <int D, bool F32>
cudaError_t configure_d() {
  cudaError_t e = cudaFuncSetAttribute(k_pass1<D, F32>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024 - 1024);
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(k_pass2<D, F32>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              227 * 1024 - 1024);
}

template <int D>
cudaError_t configure_grid() {
  constexpr int most = kGridTile2 * kGridMaxEntries * sizeof(double2);
  cudaError_t e = cudaSuccess;
  auto opt_in = [&](const void* k) {
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
  };
  opt_in((const void*)k_grid1<D, 0>);
  opt_in((const void*)k_grid1<D, 1>);
  opt_in((const void*)k_grid1<D, 2>);
  if constexpr (D > 1) opt_in((const void*)k_grid1<D, kGridLines>);
  opt_in((const void*)k_grid2<D, false>);
  opt_in((const void*)k_grid2<D, true>);
  return e;
}

template <int D, bool ROOTS>
void launch_grid2(const EvalPlan& plan, cudaStream_t s) {
  const int n = plan.h_off[D - 1][ROOTS + 1] - plan.h_off[D - 1][ROOTS];
  if (n > 0) launch_chained(plan.chain, k_grid2<D, ROOTS>, grid_ctas(n), kGridThreads, plan.smemH, s, plan);
}

template <int D, bool F32>
void launch_d(const EvalPlan& plan, bool pass2, cudaStream_t stream) {
  if (!pass2) {
    const int n = plan.d_off1[D] - plan.d_off1[D - 1];
    if (n > 0) launch_chained(plan.chain, k_pass1<D, F32>, n, kPass1Threads, plan.smem1, stream, plan);
  } else {
    const int n = plan.d_off2[D] - plan.d_off2[D - 1];
    if (n > 0)
      launch_chained(plan.chain, k_pass2<D, F32>, n, kPass2Threads, F32 ? plan.smem2_f32 : plan.smem2, stream, plan);
  }
}

}  // namespace

cudaError_t eval_configure() {
  static OncePerDevice once;
  return once.run([] {
    cudaError_t e = configure_grid<1>();
    if (e == cudaSuccess) e = configure_grid<2>();
    if (e == cudaSuccess) e = configure_grid<3>();
    if (e == cudaSuccess) e = configure_d<1, false>();
    if (e == cudaSuccess) e = configure_d<2, false>();
    if (e == cudaSuccess) e = configure_d<3, false>();
    if (e == cudaSuccess) e = configure_d<1, true>();
    if (e == cudaSuccess) e = configure_d<2, true>();
    if (e == cudaSuccess) e = configure_d<3, true>();
    return e;
  });
}

namespace {

// The pass kernels of dimension D (per-segment and grid forms). FP64 lanes run
// the F32 = false kernels whatever the plan; a plan that may hold FP32 lanes
// (dyn_prec) launches the F32 = true kernels as well.
template <int D>
void launch_dim(const EvalPlan& plan, bool pass2, cudaStream_t s) {
  launch_d<D, false>(plan, pass2, s);
  if (plan.dyn_prec) launch_d<D, true>(plan, pass2, s);
  if (pass2) {
    launch_grid2<D, false>(plan, s);
    launch_grid2<D, true>(plan, s);
  } else {
    launch_grid1<D>(plan, s);
  }
}
void launch_dim(const EvalPlan& plan, bool pass2, int D, cudaStream_t s) {
  if (D == 1) launch_dim<1>(plan, pass2, s);
  else if (D == 2) launch_dim<2>(plan, pass2, s);
  else launch_dim<3>(plan, pass2, s);
}

// The nodes that the next operation captured on a stream depends on.
cudaError_t capture_front(cudaStream_t s, std::vector<cudaGraphNode_t>* front) {
  cudaStreamCaptureStatus status;
  const cudaGraphNode_t* deps = nullptr;
  size_t n = 0;
  const cudaError_t e = cudaStreamGetCaptureInfo(s, &status, nullptr, nullptr, &deps, &n);
  if (e == cudaSuccess) front->assign(deps, deps + n);
  return e;
}

// One pass over every dimension present: in order on `stream`, or, while a tick
// graph is captured (fork), every dimension's kernels as a chain of nodes of
// their own, from what came before and joined before what follows.
cudaError_t launch_pass_all(const EvalPlan& plan, bool pass2, cudaStream_t stream, bool fork) {
  std::vector<cudaGraphNode_t> base, at, ends;
  cudaError_t e = fork ? capture_front(stream, &base) : cudaSuccess;
  for (int D = 1; D <= 3 && e == cudaSuccess; ++D) {
    if (fork)
      e = cudaStreamUpdateCaptureDependencies(stream, base.data(), base.size(),
                                              cudaStreamSetCaptureDependencies);
    if (e == cudaSuccess) launch_dim(plan, pass2, D, stream);
    if (fork && e == cudaSuccess) e = capture_front(stream, &at);
    if (fork && at != base) ends.insert(ends.end(), at.begin(), at.end());
  }
  if (e == cudaSuccess && !ends.empty())
    e = cudaStreamUpdateCaptureDependencies(stream, ends.data(), ends.size(),
                                            cudaStreamSetCaptureDependencies);
  return e == cudaSuccess ? cudaGetLastError() : e;
}

}  // namespace

cudaError_t eval_launch(const EvalPlan& plan, cudaStream_t stream, bool fork) {
  if (plan.n_grid > 0)
    launch_chained(plan.chain, k_grid_roots, dim3(plan.root_chunks, plan.n_lanes), kRootChunk, 0, stream, plan);
  cudaError_t e = launch_pass_all(plan, false, stream, fork);
  if (e != cudaSuccess) return e;
  if (plan.n_lanes > 0) {
    launch_chained(plan.chain, k_reduce, dim3(plan.red_chunks, plan.n_lanes), kReduceChunk, 0, stream, plan);
    if (!plan.want_grad) launch_chained(plan.chain, k_energy, plan.n_lanes, 32, 0, stream, plan);
  }
  if (plan.want_grad) {
    e = launch_pass_all(plan, true, stream, fork);
    if (e != cudaSuccess) return e;
  }
  return cudaGetLastError();
}

cudaError_t rho_rows(const double2* rho_run, const int* row_of, int total, int M, int N, int batch,
                     double* re, double* im, cudaStream_t stream) {
  for (int lo = 0; lo < batch; lo += 65535) {
    const int b = std::min(batch - lo, 65535);
    k_rho_rows<<<dim3((total + 127) / 128, b), 128, 0, stream>>>(
        rho_run + (size_t)lo * M, row_of, total, M, (double)N, re ? re + (size_t)lo * total : nullptr,
        im ? im + (size_t)lo * total : nullptr);
  }
  return cudaGetLastError();
}

cudaError_t structure_sums(const double2* rho_run, const int* run2ref, int M, int N, int batch,
                           double* tot, double* tot2, cudaStream_t stream) {
  k_structure_sums<<<(M + 127) / 128, 128, 0, stream>>>(rho_run, run2ref, M, (double)N, batch, tot,
                                                        tot2);
  return cudaGetLastError();
}

cudaError_t rho_scatter(const double2* rho_run, const int* run2ref, int M, int batch,
                        size_t lane_stride, double* re, double* im, cudaStream_t stream) {
  const size_t total = (size_t)M * batch;
  int blocks = (int)((total + 255) / 256);
  if (blocks > 4096) blocks = 4096;
  if (blocks < 1) blocks = 1;
  k_rho_scatter<<<blocks, 256, 0, stream>>>(rho_run, run2ref, M, batch, lane_stride, re, im);
  return cudaGetLastError();
}

}  // namespace cco
