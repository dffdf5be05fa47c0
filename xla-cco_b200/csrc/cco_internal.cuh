// Internal declarations shared by the CUDA translation units of libcco.
//
// HBM layout of one problem (built once by cco_problem_create):
//   seg1[nseg1], seg2[nseg2]  32-byte segment headers (runs of consecutive
//                             last-axis n, split at <= 8 / <= 256 rows)
//   w_run[M]                  weights in run order
//   run2ref[M]                run-order row -> caller row
// Per evaluated configuration (lane):
//   s[N][d] in, phi out, g[N][d] out, rho[M] / rhow[M] (complex, run order),
//   part[ntile1][M] pass-1 partial densities (one row per particle tile).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <mutex>

#include "cco.h"

namespace cco {

constexpr int kSeg1Len = 8;     // pass-1 segment length (register accumulators)
constexpr int kSeg2Len = 256;   // pass-2 segment length (phase re-seed interval)
constexpr int kPass1Threads = 128;
constexpr int kPass1Tile = 64;  // particles per pass-1 CTA
constexpr int kPass1Stride = kPass1Tile + 1;  // padded table row (bank spread)
constexpr int kPass2Threads = 128;
constexpr int kPass2Tile = kPass2Threads;     // one particle per pass-2 thread
constexpr int kMaxLevels = 3;
constexpr size_t kPass1TableBudget = 56 * 1024;   // bytes of pass-1 tables per CTA
constexpr size_t kPass2TableBudget = 44 * 1024;   // bytes of pass-2 tables per CTA
constexpr size_t kPass2RhoStage = 24 * 1024;      // density staged in pass-2 smem up to this
constexpr size_t kPass2RhoStage1D = 64 * 1024;    // the same for 1-D problems (no phase tables)

// One segment: rows kstart .. kstart+len-1 (run order) share the prefix
// n_0..n_{d-2}; the last axis runs n_{d-1} = n[d-1] + i.
// dig[a] packs the absolute table rows of the digits of |n_a| (start value
// for the last axis) in that pass's table layout: level l in bits 8l..8l+7,
// sign (n_a < 0) in bit 24.
struct SegHdr {
  int dig[3];
  int kstart;
  int n[3];
  int len;
};
static_assert(sizeof(SegHdr) == 32, "segment header is two 16-byte loads");

// Tensor-core form of both FP64 passes over the folded grid of the k-set
// (cco_grid.cuh). A run is a prefix and the last-axis range [a, b] of its rows
// (k-set rows kstart ..); a strip is 8 runs of similar folded length with nq
// quads of 4 columns from its block's lo on; a block is up to 4 strips and
// kGridCols columns whose phase tables a CTA builds together. A slot is one
// (quad, lane) cell; slots are numbered strip by strip, quad by quad.
constexpr int kGridStrips = 4;     // strips of a block
constexpr int kGridChunk = 64;     // particles of a pass-1 stage
constexpr int kGridTile2 = 64;     // particles of a pass-2 CTA
constexpr int kGridThreads = 128;
constexpr int kGridCtas = 4;       // CTAs per SM (registers and shared memory)
constexpr int kGridMaxEntries = 55;   // table entries per particle: 64 particles, four CTAs per SM
constexpr int kGridRootsMin = 4;  // blocks from which a kernel forms the phase roots
// pass-1 kernels by tiles of 8 x 8 cells per warp and where the roots come from:
// <= 2 (formed in the passes), <= 2, <= 3 (from the roots kernel); line grids
constexpr int kGridClasses = 4;
constexpr int kGridLines = 3;      // their class
constexpr int kGridMaxTiles = 12;  // tiles of a block
struct GridRun {
  int n0, n1, a, b, kstart, pad_;   // prefix (1-D: n0 = q), last-axis range [a, b]
};
struct GridStrip {
  int run0, nrun, nq, slot0;
  int col0, pad_;                    // table offset of its first column
};
// Line grids (sparse k-sets made of multiples i v of primitive vectors v): each
// strip has columns and prefixes of its own, i = q step + c along its line v.
struct GridLine {
  int n[3], step, q0, ncol;          // rows q0 .. q0 + 7, columns 0 .. ncol - 1
};
struct GridBlock {
  int strip0, nstrip, lo, ncol;      // columns lo .. lo + ncol - 1 (ncol a multiple of 8)
  int m0, c0, m1, c1;                // prefix windows [m, m + c) of its runs, per axis
  int ntile, pad_[3];                // its 8 x 8-cell tiles
};
struct GridRow {                     // run r of strip i at 8 i + r: table offsets, prefix
  int o0, o1, n0, n1;
};
struct GridQuad {
  int run0, nrun, c0, pad_;          // the strip's runs, the quad's first column
};

// Per-particle phase tables of one pass: row r holds z_a^(e * base^l) for one
// (axis a, level l, entry e); level 0 always holds z^0 .. z^(base-1).
struct TabLayout {
  int nlev[3];
  int base[3];
  int nent[3][kMaxLevels];
  int row[3][kMaxLevels];
  int nrows;
  int zrow;   // row of z^1 of the last axis
};

// Device-resident problem descriptor.
struct ProbDev {
  int d, N, M, nseg1, nseg2;
  TabLayout t1, t2;          // pass-1 / pass-2 table layouts
  int ntile1, ntile2;        // particle tiles of pass 1 / pass 2 (pass 2 at split 1)
  int sl2;                   // logical slices of the pass-2 segment pairs (power of 2, <= 8)
  int grid;                  // 1: FP64 lanes run the tensor-core form below, 2: pass 1 only, on lines
  int ngblk, gcls;           // its blocks; pass-1 kernel class
  int gts;                   // table entries per particle (odd)
  int gstep;                 // 1-D: prefix exponents are gstep n0 (1 otherwise)
  int groff[3], groots;      // roots area: first word / N of each virtual axis, words / N (0: none)
  int gslots;                // slots (a multiple of 32)
  int gtile, gntile;         // particles per pass-1 tile, tiles
  int grhow;                 // double2 words of the rhow area (chunk energies after the weights)
  const GridBlock* gblk;
  const GridStrip* gstrip;
  const GridRun* grun;
  const GridQuad* gquad;
  const GridRow* grow;
  const GridLine* gline;     // line grids: per strip; and per slot its rows n = +c, -c (-1: none)
  const int2* gslotk;
  int rmax[3];               // largest |n| per axis
  int compact;               // descent lanes run k_persist_compact (2: and keep their phases)
  const double4* krow;       // run-order rows (n_0, n_1, n_2, w)
  double vol;                // V
  double gpref;              // 2 (2 pi) / V
  const SegHdr* seg1;
  const SegHdr* seg2;        // sorted by length (pairs processed together)
  const double* w_run;
  const int* run2ref;
};

// One configuration evaluated by a launch.
struct EvalLane {
  const double* s;        // [N][d]
  double* f;              // [1]
  double* g;              // [N][d] or null
  double2* rho;           // [M] run order
  double2* rhow;          // pass-2 input: [M] weighted density, or the grid form's weights
  double2* part;          // [ntile1][M], or [gntile][gslots][2] (grid form)
  double2* roots;         // [groots][N] phase roots and seeds (grid form)
  const int64_t* status;  // evaluate iff null or *status == RUNNING
  const int32_t* prec;    // arithmetic of this evaluation: *prec, or `fixed_prec` when null
  int prob;
  int fixed_prec;         // PREC_FP64 or PREC_FP32
};

// Evaluation arithmetic of a lane. PREC_FP32: phase tables seeded in FP64
// and stored in FP32, phase recurrences, pass-1 accumulation (compensated)
// and the back-projection in FP32; the tile reduction, rho, w rho and Phi in
// FP64; pass-2 segment sums folded into FP64 gradients.
enum : int32_t { PREC_FP64 = 0, PREC_FP32 = 1 };
__device__ __forceinline__ int lane_prec(const EvalLane& ln) {
  return ln.prec ? *ln.prec : ln.fixed_prec;
}

struct EvalItem {
  int lane;
  int tile;
};

// ---------------------------------------------------------------- phases
// sin and cos of 2 pi m s for an integer-valued m and any s. The product m s
// is formed without rounding (p + e == m s, e by fma) and its nearest integer
// removed exactly before sincospi, so the phase keeps full precision however
// large |m s| is. Passing the rounded product instead puts |m s| eps of
// absolute error into the argument: 1.4e-12 rad at |m s| ~ 4000, which
// makes Phi ~ M (1.4e-12)^2 ~ 1e-20 the roundoff floor of a wide 1-D k-set.
__device__ __forceinline__ void sincos_2pi_ms(double m, double s, double* sn, double* cs) {
  const double p = m * s;
  const double e = fma(m, s, -p);
  sincospi(2.0 * ((p - rint(p)) + e), sn, cs);
}

// The same for n . s = sum_a n_a s_a (integer-valued n_a): exact products,
// compensated sum, nearest integer removed before sincospi.
template <int D>
__device__ __forceinline__ void sincos_2pi_dot(const double* n, const double* s, double* sn,
                                               double* cs) {
  double hi = 0.0, lo = 0.0;
#pragma unroll
  for (int a = 0; a < D; ++a) {
    const double p = n[a] * s[a];
    const double e = fma(n[a], s[a], -p);
    const double t = hi + p;
    const double z = t - hi;
    lo += ((hi - (t - z)) + (p - z)) + e;
    hi = t;
  }
  sincospi(2.0 * ((hi - rint(hi)) + lo), sn, cs);
}

// ---------------------------------------------------------------- complex
__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

// z^0 of a phase z as a table entry: 1, but NaN for a NaN z, so that a particle
// with a non-finite coordinate makes every row NaN (n . s is, also where n_a = 0).
__device__ __forceinline__ double2 zeroth_power(double2 z) {
  return make_double2(fma(0.0, z.x, 1.0), 0.0);
}

__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

__device__ __forceinline__ bool lane_active(const int64_t* status) {
  return status == nullptr || *status == CCO_STATUS_RUNNING;
}

// Deterministic block sum (fixed shuffle tree, then fixed warp order).
// `red` holds >= 32 doubles; every thread gets the total.
__device__ __forceinline__ double block_sum(double v, double* red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nw = (blockDim.x + 31) >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();
  if (lane == 0) red[warp] = v;
  __syncthreads();
  double t = 0.0;
  for (int w = 0; w < nw; ++w) t += red[w];
  return t;
}

// ---------------------------------------------------------------- launches
// Chained launches. The kernels of an evaluation or a tick follow one another on a
// stream, each needing all of its predecessor. launch_chained lets a kernel be
// set up, and its CTAs come in, while the predecessor's last ones still run; every
// CTA of it calls chain_wait first (a grid whose CTAs left without it would let
// its own successor run beside the predecessor), which returns when the
// predecessor has finished and its writes are visible. CHAIN_EARLY: the successor's
// CTAs may come in from then on; the grid kernels, which fill the GPU, leave
// that to their end (CHAIN_LATE; let in early they cost the two passes 2%). Used where a call
// is one evaluation (256 lanes of d=2 N=1000 166 -> 160 us, one of N=20000 288 -> 281,
// one of d=1 N=7777 with its synchronisation 82 -> 77, a Hessian 129 -> 123) and by
// the tick graphs of a lone lane (d=2 N=1000 to the ground state 41.7 -> 39.0 ms);
// graphs of more lanes lose more to the edges than they gain (64 MD lanes, 40
// steps: 5.17 -> 5.38 ms; 25 of d=3 N=1492: 6.1 -> 6.4 ms).
//
// The reduction and the phase roots do so only up to kChainCtas CTAs (one per SM): of
// more, the successor's CTAs would pile up on the SMs that are left first, and a pass of
// few CTAs per SM runs as long as its fullest SM (gradient of 256 lanes of d=1 N=36, 2003
// rows, after their reduction 383 -> 320 us; one lane of d=1 N=7777 after its roots 50.9
// -> 47.1). The minimizers' kernels always do: looking at their grids cost a tick 1.5 us.
constexpr unsigned kChainCtas = 148;
enum ChainLet { CHAIN_LATE, CHAIN_EARLY, CHAIN_FEW };
template <ChainLet LET = CHAIN_EARLY>
__device__ __forceinline__ void chain_wait() {
  cudaGridDependencySynchronize();
  if (LET == CHAIN_EARLY || (LET == CHAIN_FEW && gridDim.x * gridDim.y <= kChainCtas))
    cudaTriggerProgrammaticLaunchCompletion();
}

template <class... P, class... A>
void launch_chained(bool chain, void (*kernel)(P...), dim3 grid, int threads, size_t smem, cudaStream_t stream,
                    const A&... args) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = &at;
  cfg.numAttrs = chain ? 1 : 0;
  cudaLaunchKernelEx(&cfg, kernel, P(args)...);   // the error is read by cudaGetLastError
}

// Kernel attributes belong to a device: `set` (host code that opts kernels in to
// large dynamic shared memory) runs once on each device it is asked for on.
class OncePerDevice {
  std::mutex mu_;
  uint64_t done_ = 0;

 public:
  template <class F>
  cudaError_t run(F set) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const uint64_t bit = dev >= 0 && dev < 64 ? 1ull << dev : 0;   // others: every time
    std::lock_guard<std::mutex> lk(mu_);
    if (done_ & bit) return cudaSuccess;
    e = set();
    if (e == cudaSuccess) done_ |= bit;
    return e;
  }
};

// Launches of an evaluation: (phase roots,) partial densities, reduction +
// energy, gradient. Items index (lane, tile); lanes whose status is not RUNNING exit.
struct EvalPlan {
  bool chain = false;       // launch_chained: the kernels as a chain
  const ProbDev* probs;     // device
  const EvalLane* lanes;    // device
  const EvalItem* items1;   // device, grouped by d: d = D items at [d_off1[D-1], d_off1[D])
  const EvalItem* items2;   // device, grouped the same way (d_off2)
  int n_lanes, n_items1, n_items2;
  int d_off1[4], d_off2[4];
  // grid form: pass-1 items (lane, tile * ngblk + block) and pass-2 items (lane,
  // tile), grouped by d; within dimension D the pass-1 items of kernel class c
  // are [q_offG[D - 1][c], q_offG[D - 1][c + 1])
  const EvalItem* itemsG;
  const EvalItem* itemsH;
  int q_offG[3][kGridClasses + 1];
  int h_off[3][3];          // pass-2 items likewise: roots formed in the pass, from the kernel
  int n_grid, root_chunks; // lanes with roots; chunks of their roots (largest)
  size_t smemG, smemH;     // dynamic shared memory
  int dyn_prec;             // 1: lanes may be FP32 (the FP32 pass kernels launch too), 0: FP64 only
  int max_d;                // largest d in the plan (template dispatch)
  int red_chunks;           // chunks of the reduction (reduce_chunks, largest in the plan)
  int split2;               // pass-2 threads per particle (1, 2, 4 or 8)
  int chunks1;              // pass-1 segment chunks per tile (FP64 per-segment form; 1 = none)
  size_t smem1, smem2;      // dynamic shared memory of pass 1 / pass 2 (FP64 kernels)
  size_t smem2_f32;         // pass 2, FP32 kernels
  bool want_grad;
};

// A launch with few pass-1 tiles (a lone wide lane: one CTA per SM at most)
// splits each tile's segments over up to 8 CTAs. Only problems with at least
// 2 kPass1ChunkSegs segments are split, where one thread already owns one
// segment (no in-CTA particle slices), so every segment's sum is computed
// exactly as unsplit: the chunking changes where the work runs, not the bits.
// A tile is cut into no more chunks than it takes to give each thread of a
// 128-thread CTA one segment (ceil(nseg / 128)).
constexpr int kPass1ChunkSegs = 128;
__host__ __device__ __forceinline__ int pass1_chunks(const ProbDev& p, int plan_chunks) {
  if (p.nseg1 < 2 * kPass1ChunkSegs) return 1;
  const int most = (p.nseg1 + kPass1ChunkSegs - 1) / kPass1ChunkSegs;
  return plan_chunks < most ? plan_chunks : most;
}

// The reduction of the pass-1 partials runs one block per kReduceChunk
// k-vectors of a lane; a second kernel sums the chunks' energies in a fixed
// order, so the energy's rounding depends on M alone.
constexpr int kRootChunk = 256;   // roots per block of the roots kernel
constexpr int kReduceChunk = 256;
__host__ __device__ __forceinline__ int reduce_chunks(int M) {
  return (M + kReduceChunk - 1) / kReduceChunk;
}
// Scratch of one evaluated configuration, in double2 words: rho [M], the rhow
// area, the pass-1 partials (the larger of the forms the problem may run) and
// the grid form's roots.
__host__ __device__ __forceinline__ size_t eval_rhow_words(const ProbDev& p) {
  const size_t m = (size_t)p.M, g = p.grid ? (size_t)p.grhow : 0;
  return m > g ? m : g;
}
__host__ __device__ __forceinline__ size_t eval_part_words(const ProbDev& p) {
  const size_t seg = (size_t)p.ntile1 * p.M;
  const size_t g = p.grid ? 2 * (size_t)p.gntile * p.gslots : 0;
  return seg > g ? seg : g;
}
__host__ __device__ __forceinline__ size_t eval_roots_words(const ProbDev& p) {
  return p.grid ? (size_t)p.groots * p.N : 0;
}
__host__ __device__ __forceinline__ size_t eval_scratch_words(const ProbDev& p) {
  return (size_t)p.M + eval_rhow_words(p) + eval_part_words(p) + eval_roots_words(p);
}

// fork: `stream` is being captured into a tick graph; the dimensions of a pass
// become parallel nodes.
cudaError_t eval_launch(const EvalPlan& plan, cudaStream_t stream, bool fork = false);
// Kernels one eval_launch of a plan issues: per dimension the per-segment and
// grid pass kernels that have items, plus the reduction (and the energy kernel
// when there is no pass 2).
inline int eval_kernels(const EvalPlan& p) {
  int n = p.n_lanes > 0 ? (p.want_grad ? 1 : 2) : 0;   // reduce (+ energy without pass 2)
  n += p.n_grid > 0;                                   // roots
  const int per = p.dyn_prec ? 2 : 1;   // FP64 and FP32 pass kernels
  for (int D = 1; D <= 3; ++D) {
    n += per * (p.d_off1[D] > p.d_off1[D - 1]);
    for (int c = 0; c < kGridClasses; ++c) n += p.q_offG[D - 1][c + 1] > p.q_offG[D - 1][c];
    if (p.want_grad)
      n += per * (p.d_off2[D] > p.d_off2[D - 1]) + (p.h_off[D - 1][1] > p.h_off[D - 1][0]) +
           (p.h_off[D - 1][2] > p.h_off[D - 1][1]);
  }
  return n;
}
size_t eval_smem1(const ProbDev& p);
size_t eval_smemG(const ProbDev& p);   // grid pass 1 (0 when the problem has no grid)
size_t eval_smemH(const ProbDev& p);   // grid pass 2
// Pass-2 dynamic shared memory at `split` for the FP64 kernels, or with
// f32 for the FP32 ones (which keep phase tables for 1-D problems too).
size_t eval_smem2(const ProbDev& p, int split, bool f32 = false);
// Pass-2 tiles of one configuration when `split` threads share a particle.
int pass2_tiles(const ProbDev& p, int split);
// Threads per particle in pass 2 for a launch whose configurations have
// `tiles_at_split1` tiles in total at split 1: the smallest power of two
// (<= 8) that gives kPass2TargetCtas CTAs (CCO_PASS2_SPLIT overrides).
// It changes how work is spread, never the arithmetic.
constexpr long long kPass2TargetCtas = 148 * 3;
int pass2_split(long long tiles_at_split1);
cudaError_t eval_configure();   // the current device: opt-in to large dynamic shared memory

// The run-order densities in a padded layout: column c holds row row_of[c], or
// (N, 0) where that is -1.
cudaError_t rho_rows(const double2* rho_run, const int* row_of, int total, int M, int N, int batch,
                     double* re, double* im, cudaStream_t stream);
// tot[k] += |rho_k|^2 / N and tot2[k] += its square over the batch, in batch
// order, k in the caller's row order.
cudaError_t structure_sums(const double2* rho_run, const int* run2ref, int M, int N, int batch,
                           double* tot, double* tot2, cudaStream_t stream);

// Copy the run-order density of lane i out in the caller's row order.
cudaError_t rho_scatter(const double2* rho_run, const int* run2ref, int M,
                        int batch, size_t lane_stride, double* re, double* im,
                        cudaStream_t stream);

}  // namespace cco
