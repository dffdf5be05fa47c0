// cco_persist.cu - persistent relaxation of small problems: one CTA runs one
// lane's whole descent, evaluation and update, in a single launch.
//
// A tick of the graph driver (cco_relax.cu) is five to eight dependent kernel
// launches; for a problem of a few thousand (k, particle) pairs - the
// reference README's d=3 N=100 chi=0.05 relax has 1300 - their launch
// latency is the whole cost of an iteration. Here a CTA owns one lane and loops
// with block barriers between the stages and no host round trip. Lanes that fit
// shared memory altogether run k_persist_compact (512 threads, below); the others
// k_persist_descent (128 threads, the evaluation bodies' size): pass 1 over the
// lane's particle tiles (per-segment form), the tile-order reduction to rho,
// w rho and Phi, pass 2 over its tiles, and the descent update. Lanes never wait on
// one another, so there is no inter-CTA synchronization; the loop ends when
// the lane's status leaves RUNNING or after the same tick bound as the graph
// driver (then the launch reports an overrun, the host CCO_ERR_ROUNDS).
//
// Which path a lane takes depends on its problem alone (persist_eligible), so
// a lane relaxed alone and in any batch takes the same path and gives the
// same bits.
#include <cuda_runtime.h>

#include "cco_eval_bodies.cuh"
#include "cco_host.cuh"
#include "cco_internal.cuh"
#include "cco_opt_bodies.cuh"

namespace cco {

namespace {

constexpr int kPersistThreads = 128;   // kPass1Threads = kPass2Threads

// rho_k = sum over tiles of the pass-1 rows in tile order, w rho and Phi
// (one lane, the whole CTA; fixed-order block sum).
__device__ void persist_reduce(const ProbDev& P, const EvalLane& ln, double* red) {
  const int M = P.M, nt = P.ntile1;
  double e = 0.0;
  for (int k = threadIdx.x; k < M; k += blockDim.x) {
    double2 t = ln.part[k];
    for (int q = 1; q < nt; ++q) {
      const double2 o = ln.part[(size_t)q * M + k];
      t.x += o.x;
      t.y += o.y;
    }
    ln.rho[k] = t;
    const double wk = P.w_run[k];
    ln.rhow[k] = make_double2(wk * t.x, wk * t.y);
    e += wk * (t.x * t.x + t.y * t.y);
  }
  e = block_sum(e, red);
  if (threadIdx.x == 0) *ln.f = e / P.vol;
}

// Energy, gradient and density of the lane's probe positions (FP64).
template <int D>
__device__ void persist_eval(const ProbDev& P, const EvalLane& ln, double2* smem, double* red) {
  for (int t = 0; t < P.ntile1; ++t) {
    pass1_body<D>(P, ln, t, smem);
    __syncthreads();
  }
  persist_reduce(P, ln, red);
  __syncthreads();
  const int nt2 = (P.N + kPass2Tile - 1) / kPass2Tile;
  for (int t = 0; t < nt2; ++t) {
    if constexpr (D == 1) {
      if ((size_t)P.M * sizeof(double2) <= kPass2RhoStage1D) pass2_body_1d<true>(P, ln, t, 1, smem);
      else pass2_body_1d<false>(P, ln, t, 1, smem);
    } else {
      if ((size_t)P.M * sizeof(double2) <= kPass2RhoStage) pass2_body<D, true>(P, ln, t, 1, smem);
      else pass2_body<D, false>(P, ln, t, 1, smem);
    }
    __syncthreads();
  }
}

// CTA i relaxes lane i of the table (lanes of another dimension leave at once).
template <int D>
__global__ void __launch_bounds__(kPersistThreads) k_persist_descent(DescentArgs a, EvalPlan plan,
                                                                     int64_t max_ticks,
                                                                     int* overrun) {
  extern __shared__ double2 smem[];
  __shared__ ProbDev sp;
  __shared__ double red[32];
  const int lane = blockIdx.x;
  const EvalLane ln = plan.lanes[lane];
  if (threadIdx.x == 0) sp = plan.probs[ln.prob];
  __syncthreads();
  if (sp.d != D || sp.compact) return;
  const LaneRef R = a.lanes[lane];
  for (int64_t t = 0;; ++t) {
    if (*rec_status(R.rec) != CCO_STATUS_RUNNING) break;   // written before the last barrier
    if (t >= max_ticks) {
      if (threadIdx.x == 0) atomicExch(overrun, 1);
      break;
    }
    persist_eval<D>(sp, ln, smem, red);
    __syncthreads();
    descent_update_lane(a, lane);
    __syncthreads();
  }
}

// ------------------------------------------------------------ compact lanes
// A lane whose positions, gradients and per-particle axis tables fit shared
// memory runs there altogether, 512 threads, four barriers per iteration:
//   tables   z_a^0 .. z_a^R of the probe positions, a thread per (particle,
//            axis, 8 entries): one FP64 sincospi of the exactly reduced argument,
//            then products;
//   density  a warp per row (up to four rows interleaved), lanes over the
//            particles, the phase a product of d table entries, shuffle sums;
//   gradient 2^t neighbouring threads per particle, each every 2^t-th row,
//            shuffle sums (the density's phases are kept for it where they
//            fit); |g|^2 and the exact zero test on the way; one warp also
//            sums the energy;
//   update   the descent rule, every thread on the same scalars (no broadcast).
// At d=3 N=100 M=13 the general form above spent 12.7 us per iteration on two
// table builds, two particle tiles one after the other, trips through global
// memory and ~25 barriers; this form takes 3.6 us, a chain of latencies (sincospi,
// shuffles, barriers) that neither the 1300 pairs nor memory bound.
// (With more lanes than SMs fewer threads take a lane, see launch_compact; sums are
// then formed as the 512 form them.)
constexpr int kCompactThreads = 512;
constexpr int kPersistSms = 148;   // SMs of a B200

// Every thread's copy of the descent state of a lane.
struct CompactState {
  double f, step, norm;
  int64_t it, n_evals, rec;
  bool nonzero;
};

template <int D, int T>
__global__ void __launch_bounds__(T) k_persist_compact(DescentArgs a, EvalPlan plan, int64_t max_ticks,
                                                       int* overrun) {
  extern __shared__ double2 smem[];
  __shared__ ProbDev P;
  __shared__ double red[kCompactThreads / 32], f_s;
  const int lane = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, wl = tid & 31;
  constexpr int NWARP = T / 32, VWARP = kCompactThreads / 32;
  const EvalLane ln = plan.lanes[lane];
  if (tid == 0) P = plan.probs[ln.prob];
  __syncthreads();
  if (P.d != D || !P.compact) return;
  const LaneRef R = a.lanes[lane];
  const DsView v = ds_view(R.rec, R.ld);
  if (v.st->status != CCO_STATUS_RUNNING) return;
  const int N = P.N, M = P.M, nd = N * D;
  // shared memory: tables [entries][N], rows, w rho, energies; s, g, ps, pg
  int base[D], entries = 0;
#pragma unroll
  for (int c = 0; c < D; ++c) {
    base[c] = entries;
    entries += P.rmax[c] + 1;
  }
  double2* tab = smem;
  double2* rw = tab + (size_t)entries * N;
  double4* row = reinterpret_cast<double4*>(rw + M + (M & 1));
  int4* ro = reinterpret_cast<int4*>(row + M);   // table offsets per axis (~o: conjugate)
  double* ek = reinterpret_cast<double*>(ro + M);
  double *s = ek + M, *g = s + nd, *ps = g + nd, *pg = ps + nd;
  // the density's phases, kept for the gradient when they fit as well
  const bool keep = P.compact == 2;
  const int pst = N | 1;
  double2* ph = reinterpret_cast<double2*>(ek + ((M + 4 * nd + 1) & ~1));
  for (int k = tid; k < M; k += T) {
    const double4 r = P.krow[k];
    const double nv[3] = {r.x, r.y, r.z};
    int o[3] = {0, 0, 0};
#pragma unroll
    for (int c = 0; c < D; ++c) {
      const int n = (int)nv[c], at = (base[c] + abs(n)) * N;
      o[c] = n < 0 ? ~at : at;
    }
    row[k] = r;
    ro[k] = make_int4(o[0], o[1], o[2], 0);
  }
  for (int e = tid; e < nd; e += T) {
    s[e] = v.s[e];
    g[e] = v.g[e];
    ps[e] = v.ps[e];
  }
  // table units: (axis, 8 entries) of every particle
  int units[D], nunit = 0;
#pragma unroll
  for (int c = 0; c < D; ++c) nunit += units[c] = (P.rmax[c] + 8) >> 3;
  int tpp = 1;   // threads per particle in the gradient
  while (tpp < 16 && 2 * tpp * N <= kCompactThreads && 2 * tpp <= M) tpp *= 2;
  CompactState S{v.st->f, v.st->step, v.st->norm, v.st->it, v.st->n_evals,
                 a.traj_count ? a.traj_count[R.idx] : 0, v.st->nonzero != 0};
  bool init = v.st->phase == PH_INIT;
  int64_t status = CCO_STATUS_RUNNING;
  auto phase = [&](const int4& r, int j) {
    const int o[3] = {r.x, r.y, r.z};
    double2 p;
#pragma unroll
    for (int c = 0; c < D; ++c) {
      double2 z = tab[(o[c] < 0 ? ~o[c] : o[c]) + j];
      if (o[c] < 0) z.y = -z.y;
      p = c == 0 ? z : cmul(p, z);
    }
    return p;
  };
  __syncthreads();
  for (int64_t t = 0;; ++t) {
    if (t >= max_ticks) {
      if (tid == 0) atomicExch(overrun, 1);
      break;
    }
    // tables
    for (int w = tid; w < nunit * N; w += T) {
      const int j = w % N;
      int u = w / N, c = 0;
#pragma unroll
      for (int q = 0; q + 1 < D; ++q)
        if (c == q && u >= units[q]) {
          u -= units[q];
          c = q + 1;
        }
      const double x = ps[j * D + c];
      const int e0 = 8 * u, e1 = min(e0 + 8, P.rmax[c] + 1);
      double2 z, p;
      sincos_2pi_ms(1.0, x, &z.y, &z.x);
      p = zeroth_power(z);
      if (e0 > 0) sincos_2pi_ms((double)e0, x, &p.y, &p.x);
      for (int e = e0; e < e1; ++e) {
        tab[(size_t)(base[c] + e) * N + j] = p;
        p = cmul(p, z);
      }
    }
    __syncthreads();
    // density
    for (int k0 = warp; k0 < M; k0 += 4 * NWARP) {
      double2 acc[4];
      int4 r[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        acc[q] = make_double2(0.0, 0.0);
        r[q] = ro[min(k0 + q * NWARP, M - 1)];
      }
      const int nq = min(4, (M - 1 - k0) / NWARP + 1);
      for (int j = wl; j < N; j += 32)
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (q < nq) {
            const double2 z = phase(r[q], j);
            if (keep) ph[(size_t)(k0 + q * NWARP) * pst + j] = z;
            acc[q].x += z.x;
            acc[q].y += z.y;
          }
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (q < nq) {
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) {
            acc[q].x += __shfl_xor_sync(0xffffffffu, acc[q].x, o);
            acc[q].y += __shfl_xor_sync(0xffffffffu, acc[q].y, o);
          }
          if (wl == 0) {
            const double w = row[k0 + q * NWARP].w;
            rw[k0 + q * NWARP] = make_double2(w * acc[q].x, w * acc[q].y);
            ek[k0 + q * NWARP] = w * (acc[q].x * acc[q].x + acc[q].y * acc[q].y);
          }
        }
    }
    __syncthreads();
    // gradient, |g|^2, energy: as kCompactThreads threads do it, whatever T (the
    // warps take the 16 warps' parts one after the other)
    int nz = 0;
    const int per = kCompactThreads / tpp, q = tid & (tpp - 1);
#pragma unroll 1
    for (int i = 0; i < VWARP / NWARP; ++i) {
      const int vw = warp + i * NWARP;
      double ss = 0.0;
      for (int j0 = 0; j0 < N; j0 += per) {
        const int j = j0 + (32 * vw + wl) / tpp;
        double G[D];
#pragma unroll
        for (int c = 0; c < D; ++c) G[c] = 0.0;
        if (j < N)
          for (int k = q; k < M; k += tpp) {
            const double4 r = row[k];
            const double2 z = keep ? ph[(size_t)k * pst + j] : phase(ro[k], j), w = rw[k];
            const double h = w.y * z.x - w.x * z.y;
            const double nv[3] = {r.x, r.y, r.z};
#pragma unroll
            for (int c = 0; c < D; ++c) G[c] += nv[c] * h;
          }
        for (int o = tpp >> 1; o > 0; o >>= 1)
#pragma unroll
          for (int c = 0; c < D; ++c) G[c] += __shfl_xor_sync(0xffffffffu, G[c], o);
        if (j < N && q == 0) {
#pragma unroll
          for (int c = 0; c < D; ++c) {
            const double x = P.gpref * G[c];
            pg[j * D + c] = x;
            ss += x * x;
            nz |= x != 0.0;
          }
        }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
      if (wl == 0) red[vw] = ss;
    }
    if (warp == NWARP - 1) {
      double e = 0.0;
      for (int k = wl; k < M; k += 32) e += ek[k];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
      if (wl == 0) f_s = e / P.vol;
    }
    nz = __syncthreads_or(nz);
    // the descent rule (descent.py:121-175), every thread on the same numbers
    double ss = 0.0;
#pragma unroll
    for (int w = 0; w < VWARP; ++w) ss += red[w];
    const double f2 = f_s;
    bool take = true;
    if (!init) {
      const double df = S.f - f2, df2 = S.step * S.norm;
      // reject iff |df - df2| / df2 > rel_tol (NaN accepts); the division only
      // where the products are too close to tell
      const double x = fabs(df - df2), y = a.rel_tol * df2;
      if (df2 > 1e-280 && a.rel_tol > 1e-20 && x > y * (1.0 + 1e-15) && x < 1e280) take = false;
      else if (df2 > 1e-280 && a.rel_tol > 1e-20 && x < y * (1.0 - 1e-15)) take = true;
      else take = !(x / df2 > a.rel_tol);
      S.step = take ? S.step * a.grow : S.step * a.shrink;
      S.it += 1;
      S.n_evals += 2;
    }
    init = false;
    if (take) {
      S.f = f2;
      S.norm = sqrt(ss);
      S.nonzero = nz != 0;
    }
    status = descent_status(S.f, S.nonzero, S.step, S.it, a);
    const bool rec = a.traj_count && S.it % a.rec_every == 0 && S.rec < a.rec_cap;
    for (int e = tid; e < nd; e += T) {
      if (take) {
        s[e] = S.it == 0 ? s[e] : ps[e];
        g[e] = pg[e];
      }
      if (rec) a.traj_s[R.toff + (size_t)S.rec * nd + e] = wrap01(s[e]);
      if (status == CCO_STATUS_RUNNING) {
        const double gn = S.norm > 0.0 ? __ddiv_rn(g[e], S.norm) : 0.0 * g[e];
        ps[e] = __dsub_rn(s[e], __dmul_rn(gn, S.step));
      }
    }
    if (rec) {
      if (tid == 0) {
        a.traj_e[R.idx * a.rec_cap + S.rec] = S.f;
        a.traj_step[R.idx * a.rec_cap + S.rec] = S.step;
        a.traj_it[R.idx * a.rec_cap + S.rec] = S.it;
      }
      S.rec += 1;
    }
    if (status != CCO_STATUS_RUNNING) break;
    __syncthreads();
  }
  __syncthreads();
  for (int e = tid; e < nd; e += T) {
    v.s[e] = s[e];
    v.g[e] = g[e];
    v.ps[e] = ps[e];
  }
  if (tid == 0) {
    DsState* st = v.st;
    st->phase = init ? PH_INIT : PH_ITER;
    st->f = S.f;
    st->step = S.step;
    st->norm = S.norm;
    st->nonzero = S.nonzero;
    st->it = S.it;
    st->n_evals = S.n_evals;
    st->status = status;
    if (status != CCO_STATUS_RUNNING) st->t1 = gtimer();
    if (a.traj_count) a.traj_count[R.idx] = S.rec;
  }
}

}  // namespace

bool persist_eligible(const cco_problem* p) {
  const double flops = (double)p->N * p->M * (p->d == 1 ? 7.0 : p->d == 2 ? 21.0 : 35.0);
  return flops <= kPersistMaxFlops && persist_smem(p) <= kPersistMaxSmem;
}

size_t compact_smem(const ProbDev& p) {
  size_t entries = 0;
  for (int a = 0; a < p.d; ++a) entries += p.rmax[a] + 1;
  const size_t N = p.N, M = p.M, nd = N * p.d;
  return 16 * (entries * N + M + (M & 1)) + 48 * M + 8 * (M + 4 * nd + 1);
}

size_t compact_phase_smem(const ProbDev& p) {
  return 16 * (size_t)p.M * (p.N | 1);
}

size_t persist_smem(const cco_problem* p) {
  if (p->host.compact)
    return compact_smem(p->host) + (p->host.compact == 2 ? compact_phase_smem(p->host) : 0);
  return std::max(p->smem1, eval_smem2(p->host, 1));
}

namespace {

template <int D, int T>
void launch_compact(const DescentArgs& a, const EvalPlan& plan, size_t smem, int64_t max_ticks,
                    int* d_overrun, cudaStream_t st) {
  k_persist_compact<D, T><<<a.B, T, smem, st>>>(a, plan, max_ticks, d_overrun);
}

// Rounds of CTAs that a.B lanes take with T threads each, times what an iteration
// costs next to 512 threads.
template <int D, int T>
double compact_cost(const DescentArgs& a, size_t smem) {
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_persist_compact<D, T>, T, smem) !=
          cudaSuccess || per_sm < 1)
    return 1e300;
  const int rounds = (a.B + kPersistSms * per_sm - 1) / (kPersistSms * per_sm);
  return rounds * (T == 512 ? 1.0 : T == 256 ? 1.25 : 1.9);
}

// A lane gives the same bits with any number of threads. 512 are the fastest for one
// lane per SM (relaxations of 100 evaluations with 512 / 256 / 128 threads, 5 lanes: d=3
// N=100 278 / 351 / 462 us, d=1 N=60 301 / 326 / 467); more lanes run in fewer rounds
// with smaller CTAs where shared memory lets several share an SM (1500 lanes: 2255 /
// 1924 / 1552 and 2006 / 1171 / 1268 us; the general form 3342 and 1456).
template <int D>
void launch_compact(const DescentArgs& a, const EvalPlan& plan, size_t smem, int64_t max_ticks,
                    int* d_overrun, cudaStream_t st) {
  const double c512 = a.B <= kPersistSms ? 0.0 : compact_cost<D, 512>(a, smem);
  const double c256 = c512 == 0.0 ? 1.0 : compact_cost<D, 256>(a, smem);
  const double c128 = c512 == 0.0 ? 1.0 : compact_cost<D, 128>(a, smem);
  if (c512 <= c256 && c512 <= c128) launch_compact<D, 512>(a, plan, smem, max_ticks, d_overrun, st);
  else if (c256 <= c128) launch_compact<D, 256>(a, plan, smem, max_ticks, d_overrun, st);
  else launch_compact<D, 128>(a, plan, smem, max_ticks, d_overrun, st);
}

}  // namespace

cudaError_t persist_descent(const DescentArgs& a, const EvalPlan& plan, size_t smem, int dims,
                            int64_t max_ticks, int* d_overrun, cudaStream_t st) {
  static OncePerDevice once;
  const cudaError_t configured = once.run([] {
    cudaError_t e = cudaSuccess;
    for (const void* k : {(const void*)k_persist_descent<1>, (const void*)k_persist_descent<2>,
                          (const void*)k_persist_descent<3>, (const void*)k_persist_compact<1, 512>,
                          (const void*)k_persist_compact<2, 512>, (const void*)k_persist_compact<3, 512>,
                          (const void*)k_persist_compact<1, 256>, (const void*)k_persist_compact<2, 256>,
                          (const void*)k_persist_compact<3, 256>, (const void*)k_persist_compact<1, 128>,
                          (const void*)k_persist_compact<2, 128>, (const void*)k_persist_compact<3, 128>})
      if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kPersistMaxSmem);
    return e;
  });
  if (configured != cudaSuccess) return configured;
  if (dims & 8) launch_compact<1>(a, plan, smem, max_ticks, d_overrun, st);
  if (dims & 16) launch_compact<2>(a, plan, smem, max_ticks, d_overrun, st);
  if (dims & 32) launch_compact<3>(a, plan, smem, max_ticks, d_overrun, st);
  if (dims & 1) k_persist_descent<1><<<a.B, kPersistThreads, smem, st>>>(a, plan, max_ticks, d_overrun);
  if (dims & 2) k_persist_descent<2><<<a.B, kPersistThreads, smem, st>>>(a, plan, max_ticks, d_overrun);
  if (dims & 4) k_persist_descent<3><<<a.B, kPersistThreads, smem, st>>>(a, plan, max_ticks, d_overrun);
  return cudaGetLastError();
}

}  // namespace cco
