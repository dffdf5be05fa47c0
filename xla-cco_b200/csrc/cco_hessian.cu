// cco_hessian.cu - closed-form Hessian of the stealthy energy on the device.
//
//   d2 Phi / ds_ja ds_lb = pref sum_k w_k n_ka n_kb [cos(th_kj - th_kl)
//                           - delta_jl (Re rho_k cos th_kj + Im rho_k sin th_kj)]
//   th_kj = 2 pi n_k . s_j,  pref = 2 (2 pi)^2 / V        (src/xla_cco/energy.py:272-299)
//
// Three kernels per k-chunk (one chunk unless the phases pass kPhaseBytes):
//   k_hess_phase  the phases exp(i th_kj) of the chunk, once per (k, particle),
//                 from the argument n . s reduced exactly (fma products,
//                 compensated sum, nearest integer removed) before sincospi;
//   k_hess_diag   the delta_jl sums of the chunk (a warp per particle; rho comes
//                 from the evaluation kernels);
//   k_hess_tiles  cos(th_j - th_l) = c_j c_l + s_j s_l makes block (a, b) a real
//                 matrix product of depth 2 M with weights q_kab = w_k n_ka n_kb
//                 (a <= b), run on the FP64 matrix pipe (DMMA m8n8k4). A CTA owns
//                 32 particles x 32 particles at or above the diagonal and all
//                 component pairs; a warp 16 x 16 of them.
// The product costs N^2 M (d (d + 1) / 2) FMAs (half of the matrix), against
// which everything else is small; the tile goes through shared memory so that it
// and its mirror are written row by row, and an element and its mirror come from
// the same sum (the matrix is exactly symmetric).
//
// d=2 N=700 M=560: before, one sincospi per (k, particle, tile pair) and FP64
// FMAs took 240 us and a thread per particle walking all k 238 us; now 4 us for
// the phases, 8 for the diagonal and 88 for the tiles, whose DMMAs alone need
// 57 us on the SMs that hold two of the 253 CTAs.
#include <cuda_runtime.h>

#include <algorithm>

#include "cco_host.cuh"
#include "cco_internal.cuh"

namespace cco {
namespace {

constexpr int kHessTile = 32;      // particles per tile side
constexpr int kHessK = 16;         // k rows per shared-memory chunk (two chunks held)
constexpr int kHessThreads = 128;
constexpr int kHessStride = kHessTile + 2;   // 16-byte words: fragment reads hit 8 banks
constexpr size_t kPhaseBytes = (size_t)256 << 20;   // phases held at a time

// Component pair c (a <= b) of dimension D, in row order of the upper triangle.
template <int D>
__device__ __forceinline__ void hess_ab(int c, int& a, int& b) {
  if (D == 1) {
    a = b = 0;
  } else if (D == 2) {
    a = c == 2 ? 1 : 0;
    b = c == 0 ? 0 : 1;
  } else {
    a = c < 3 ? 0 : c < 5 ? 1 : 2;
    b = c < 3 ? c : c < 5 ? c - 2 : 2;
  }
}

// Linear index over the upper triangle of T x T tile pairs -> (J, L), L >= J.
__device__ __forceinline__ void tile_pair(int t, int T, int& J, int& L) {
  J = 0;
  while (t >= T - J) {
    t -= T - J;
    ++J;
  }
  L = J + t;
}

// ph[lane][k - k0][j] = exp(i th_kj)
template <int D>
__global__ void k_hess_phase(const double* __restrict__ s, const double4* __restrict__ krow, int N,
                             int k0, int kn, double2* __restrict__ ph) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x, lane = blockIdx.z;
  if (j >= N) return;
  double sj[D];
#pragma unroll
  for (int a = 0; a < D; ++a) sj[a] = s[((size_t)lane * N + j) * D + a];
  for (int k = blockIdx.y; k < kn; k += gridDim.y) {
    const double4 r = krow[k0 + k];
    const double nv[3] = {r.x, r.y, r.z};
    double sn, cs;
    sincos_2pi_dot<D>(nv, sj, &sn, &cs);
    ph[((size_t)lane * kn + k) * N + j] = make_double2(cs, sn);
  }
}

// dg[lane][j][c] = sum over the chunk of q_kab (Re rho_k cos th_kj + Im rho_k sin th_kj)
template <int D>
__global__ void k_hess_diag(const double2* __restrict__ ph, const double4* __restrict__ krow,
                            const double2* __restrict__ rho, int N, int M, int k0, int kn,
                            double* __restrict__ dg) {
  constexpr int NC = D * (D + 1) / 2;
  const int j = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = blockIdx.y;
  if (j >= N) return;
  double acc[NC];
#pragma unroll
  for (int c = 0; c < NC; ++c) acc[c] = 0.0;
  for (int k = threadIdx.x & 31; k < kn; k += 32) {
    const double4 r = krow[k0 + k];
    const double2 z = ph[((size_t)lane * kn + k) * N + j];
    const double2 rh = rho[(size_t)lane * M + k0 + k];
    const double core = r.w * fma(rh.x, z.x, rh.y * z.y);
    const double nv[3] = {r.x, r.y, r.z};
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      int a, b;
      hess_ab<D>(c, a, b);
      acc[c] = fma(core * nv[a], nv[b], acc[c]);
    }
  }
#pragma unroll
  for (int c = 0; c < NC; ++c) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], o);
    if ((threadIdx.x & 31) == 0) dg[((size_t)lane * N + j) * NC + c] = acc[c];
  }
}

__device__ __forceinline__ void dmma(double (&d)[2], double a, double b) {
  asm volatile(
      "mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
      : "+d"(d[0]), "+d"(d[1])
      : "d"(a), "d"(b));
}

template <int D>
constexpr size_t hess_smem() {
  const size_t nc = D * (D + 1) / 2;
  const size_t chunk =
      2 * (2 * (size_t)kHessK * kHessStride * sizeof(double2) + kHessK * nc * sizeof(double));
  const size_t side = (size_t)kHessTile * D, tile = side * (side + 1) * sizeof(double);
  return chunk > tile ? chunk : tile;
}

template <int D>
__global__ void __launch_bounds__(kHessThreads)
k_hess_tiles(const double2* __restrict__ ph, const double4* __restrict__ krow,
             const double* __restrict__ dg, int N, int k0, int kn, double pref, bool first,
             double* __restrict__ H) {
  constexpr int NC = D * (D + 1) / 2, TS = kHessTile, SIDE = TS * D;
  extern __shared__ double2 sm[];
  double2* z2 = sm;   // [2][j, l][kHessK][kHessStride]
  constexpr int ZW = kHessK * kHessStride;
  double* q2 = reinterpret_cast<double*>(sm + 4 * ZW);   // [2][kHessK][NC]
  const int T = (N + TS - 1) / TS;
  int J, L;
  tile_pair(blockIdx.x, T, J, L);
  const int lane = blockIdx.y;
  const double2* pl = ph + (size_t)lane * kn * N;
  const int warp = threadIdx.x >> 5, wl = threadIdx.x & 31, t = wl & 3, r = wl >> 2;
  const int jw = 16 * (warp >> 1), lw = 16 * (warp & 1);
  double acc[NC][2][2][2];
#pragma unroll
  for (int c = 0; c < NC; ++c)
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
      for (int v = 0; v < 2; ++v) acc[c][u][v][0] = acc[c][u][v][1] = 0.0;
  // a chunk's phases travel through registers: the next chunk's are loaded while
  // this one's products run (95 -> 88 us on d=2 N=700), one barrier per chunk
  constexpr int NL = kHessK * TS / kHessThreads;
  double2 nj[NL], nl[NL];
  auto load = [&](int kc) {
#pragma unroll
    for (int i = 0; i < NL; ++i) {
      const int e = threadIdx.x + i * kHessThreads, k = e / TS, p = e - k * TS;
      const bool in = kc + k < kn;   // rows past the chunk are zero
      const size_t row = (size_t)(kc + k) * N;
      const int j = J * TS + p, l = L * TS + p;
      nj[i] = in && j < N ? pl[row + j] : make_double2(0.0, 0.0);
      nl[i] = in && l < N ? pl[row + l] : make_double2(0.0, 0.0);
    }
  };
  auto store = [&](int buf, int kc) {
    double2 *zj = z2 + 2 * buf * ZW, *zl = zj + ZW;
#pragma unroll
    for (int i = 0; i < NL; ++i) {
      const int e = threadIdx.x + i * kHessThreads, k = e / TS, p = e - k * TS;
      zj[k * kHessStride + p] = nj[i];
      zl[k * kHessStride + p] = nl[i];
    }
    for (int e = threadIdx.x; e < kHessK * NC; e += kHessThreads) {
      const int k = e / NC, c = e - k * NC;
      double v = 0.0;
      if (kc + k < kn) {
        const double4 w = krow[k0 + kc + k];
        const double nv[3] = {w.x, w.y, w.z};
        int a, b;
        hess_ab<D>(c, a, b);
        v = w.w * nv[a] * nv[b];
      }
      q2[buf * kHessK * NC + e] = v;
    }
  };
  load(0);
  store(0, 0);
  __syncthreads();
  for (int kc = 0, buf = 0; kc < kn; kc += kHessK, buf ^= 1) {
    const bool more = kc + kHessK < kn;
    if (more) load(kc + kHessK);
    const double2 *zj = z2 + 2 * buf * ZW, *zl = zj + ZW;
    const double* q = q2 + buf * kHessK * NC;
#pragma unroll 2
    for (int k = 0; k < kHessK; k += 4) {
      double2 a[2], b[2];
#pragma unroll
      for (int u = 0; u < 2; ++u) a[u] = zj[(k + t) * kHessStride + jw + 8 * u + r];
#pragma unroll
      for (int v = 0; v < 2; ++v) b[v] = zl[(k + t) * kHessStride + lw + 8 * v + r];
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        const double qc = q[(k + t) * NC + c];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const double ax = qc * a[u].x, ay = qc * a[u].y;
#pragma unroll
          for (int v = 0; v < 2; ++v) {
            dmma(acc[c][u][v], ax, b[v].x);
            dmma(acc[c][u][v], ay, b[v].y);
          }
        }
      }
    }
    if (more) store(buf ^ 1, kc + kHessK);
    __syncthreads();
  }
  // the tile, scaled and with its share of the diagonal term, into shared memory
  double* tile = reinterpret_cast<double*>(sm);   // [SIDE][SIDE + 1]
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    int a, b;
    hess_ab<D>(c, a, b);
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
      for (int v = 0; v < 2; ++v)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int pj = jw + 8 * u + r, p2 = lw + 8 * v + 2 * t + h;
          double x = pref * acc[c][u][v][h];
          if (J == L && pj == p2 && J * TS + pj < N)
            x -= pref * dg[((size_t)lane * N + J * TS + pj) * NC + c];
          tile[(pj * D + a) * (SIDE + 1) + p2 * D + b] = x;
          if (a != b) tile[(pj * D + b) * (SIDE + 1) + p2 * D + a] = x;
        }
  }
  __syncthreads();
  const size_t nd = (size_t)N * D;
  double* Hl = H + (size_t)lane * nd * nd;
  const int rows = min(SIDE, (N - J * TS) * D), cols = min(SIDE, (N - L * TS) * D);
  // a diagonal tile's lower half is the mirror of its upper half (blocks of equal
  // particles are symmetric as written)
  for (int e = threadIdx.x; e < SIDE * SIDE; e += kHessThreads) {
    const int y = e / SIDE, x = e - y * SIDE;
    if (y >= rows || x >= cols) continue;
    const bool up = J != L || x / D >= y / D;
    const double v = up ? tile[y * (SIDE + 1) + x] : tile[x * (SIDE + 1) + y];
    double* o = Hl + (size_t)(J * SIDE + y) * nd + L * SIDE + x;
    *o = first ? v : *o + v;
  }
  if (J == L) return;
  for (int e = threadIdx.x; e < SIDE * SIDE; e += kHessThreads) {
    const int x = e / SIDE, y = e - x * SIDE;   // row x of the mirror tile
    if (y >= rows || x >= cols) continue;
    const double v = tile[y * (SIDE + 1) + x];
    double* o = Hl + (size_t)(L * SIDE + x) * nd + J * SIDE + y;
    *o = first ? v : *o + v;
  }
}

template <int D>
cudaError_t launch_hessian(const cco_problem* p, cudaStream_t st, int batch, const double* s,
                           const double2* rho, double* H) {
  constexpr int NC = D * (D + 1) / 2;
  const int N = p->N, M = p->M;
  const int T = (N + kHessTile - 1) / kHessTile;
  const size_t nd = (size_t)N * D;
  const double pref = 2.0 * (2.0 * M_PI) * (2.0 * M_PI) / p->host.vol;
  static OncePerDevice once;
  const cudaError_t opt = once.run([] {
    return cudaFuncSetAttribute(k_hess_tiles<D>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)hess_smem<D>());
  });
  if (opt != cudaSuccess) return opt;
  // lanes, then k rows, at a time: phases within kPhaseBytes
  const size_t per_k = (size_t)N * sizeof(double2);
  const int kn_max = (int)std::max<size_t>(1, std::min<size_t>(M, kPhaseBytes / per_k));
  const int lanes = (int)std::max<size_t>(1, std::min<size_t>(batch, kPhaseBytes / (per_k * kn_max)));
  double2* ph = nullptr;
  double* dg = nullptr;
  cudaError_t e = pool_alloc(&ph, per_k * kn_max * lanes, st);
  if (e == cudaSuccess) e = pool_alloc(&dg, sizeof(double) * NC * N * lanes, st);
  for (int lo = 0; lo < batch && e == cudaSuccess; lo += lanes) {
    const int b = std::min(lanes, batch - lo);
    for (int k0 = 0; k0 < M && e == cudaSuccess; k0 += kn_max) {
      const int kn = std::min(kn_max, M - k0);
      const double* sl = s + (size_t)lo * nd;
      k_hess_phase<D><<<dim3((N + 127) / 128, std::min(kn, 256), b), 128, 0, st>>>(sl, p->krow, N, k0,
                                                                               kn, ph);
      k_hess_diag<D><<<dim3((N + 3) / 4, b), 128, 0, st>>>(ph, p->krow, rho + (size_t)lo * M, N, M, k0,
                                                           kn, dg);
      k_hess_tiles<D><<<dim3((unsigned)(T * (T + 1) / 2), b), kHessThreads, hess_smem<D>(), st>>>(
          ph, p->krow, dg, N, k0, kn, pref, k0 == 0, H + (size_t)lo * nd * nd);
      e = cudaGetLastError();
    }
  }
  if (ph) cudaFreeAsync(ph, st);
  if (dg) cudaFreeAsync(dg, st);
  return e;
}

}  // namespace

cudaError_t hessian_launch(const cco_problem* p, cudaStream_t st, int batch, const double* s,
                           const double2* rho_run, double* H) {
  if (p->d == 1) return launch_hessian<1>(p, st, batch, s, rho_run, H);
  if (p->d == 2) return launch_hessian<2>(p, st, batch, s, rho_run, H);
  return launch_hessian<3>(p, st, batch, s, rho_run, H);
}

}  // namespace cco
