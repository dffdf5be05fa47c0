// Tensor-core form of the FP64 evaluation: both passes as small FP64 matrix
// products (DMMA, mma.sync m8n8k4) over a folded grid of the k-set.
//
// Grid. A k-set row is (prefix, last-axis n). Rows sharing a prefix form a
// run; the last axis is folded to columns c = |n|, so a cell (run r, column c)
// holds the two k-set rows n = +c and n = -c. A 1-D k-set n = 1..M is given
// runs of its own: n = q S + c with S = 2 C + 1 and |c| <= C, prefix phase
// z^(q S). With A_r = a + i b the run's prefix phase of a particle and
// z^c = u + i v its last-axis power:
//   density   P1 = sum a u, P2 = sum b v, P3 = sum a v, P4 = sum b u give
//             rho(+c) = (P1 - P2) + i (P3 + P4), rho(-c) = (P1 + P2) + i (P4 - P3)
//   gradient  T_r = sum_c conj(w rho(+c)) z^c + conj(w rho(-c)) conj(z^c) and
//             T'_r, the same with weights +-c, are real products of a weight
//             matrix with (u, v); the gradient is -sum_r n_r Im(A_r T_r) per
//             prefix axis and -sum_r Im(A_r T'_r) along the last axis.
// That is 2 FMAs per (k-set row, particle) for the density and 4 for the
// gradient, against 6 and 8 FP64 instructions of the phase recurrences
// (cco_eval_bodies.cuh), and they run on the FP64 matrix pipe: it has the FMA
// pipe's peak (37.0 against 33.9 TFLOP/s measured on register-only loops), but
// one instruction does 256 FMAs from two operand registers per thread, so
// issue slots and shared-memory reads stop being the limit.
//
// Measured against the recurrence kernels it replaced (evaluations with
// gradient): 256 lanes of d=2 N=1000 M=802 285 -> 186 us, 64 lanes of d=3
// N=4000 M=5413 2765 -> 1432 us, one lane of d=2 N=20000 M=18000 600 -> 309 us,
// one of d=1 N=7777 M=3732 109 -> 64 us; forces up to 1.6 times closer to
// the exact sums. Bound: the FP64 pipe, which the tables share.
//
// Tiling. Runs are sorted by folded length in strips of 8; a strip's columns
// are 4-column quads. A slot (quad, lane) is one cell: lane = 4 row + t holds
// run grid_perm(row) of the strip and column 4 quad + t. Partials and the
// pass-2 weights are stored slot by slot, which makes both coalesced and is
// the order the matrix fragments want. Up to 4 strips and 48 columns form a
// block, whose phase tables a CTA builds together in shared memory.
//
// Bank conflicts. A particle's table entries are contiguous and particles are
// an odd number of entries apart. Fragment reads then touch 8 distinct 16-byte
// banks per quarter warp because row (or column) r of a fragment is run
// (particle, column) grid_perm(r): the two rows of a quarter are 4 apart.
#pragma once

#include "cco_internal.cuh"

namespace cco {

namespace {

__device__ __forceinline__ int grid_perm(int r) { return (r >> 1) + 4 * (r & 1); }

// D += A B, A 8x4 (row = lane / 4, k = lane % 4), B 4x8 (k = lane % 4,
// column = lane / 4), D 8x8 (row = lane / 4, columns 2 (lane % 4) + {0, 1}).
__device__ __forceinline__ void dmma(double (&d)[2], double a, double b) {
  asm volatile(
      "mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
      : "+d"(d[0]), "+d"(d[1])
      : "d"(a), "d"(b));
}

// dst[e] = exp(2 pi i step (m + e) s), e < cnt: FP64 sincospi of the exactly
// reduced argument at the first entry, products with exp(2 pi i step s) after
// it. A dead particle (past the tile's end) gets `fillv` instead.
__device__ __forceinline__ void grid_powers(double2* dst, int m, int cnt, int step, double s,
                                            bool live, double fillv) {
  if (!live) {
    for (int e = 0; e < cnt; ++e) dst[e] = make_double2(fillv, 0.0);
    return;
  }
  double sn, cs;
  sincos_2pi_ms((double)step, s, &sn, &cs);
  const double2 z = make_double2(cs, sn);
  double2 p = make_double2(1.0, 0.0);
  if (m == 1) {
    p = z;
  } else if (m != 0) {
    sincos_2pi_ms((double)((long long)step * m), s, &sn, &cs);
    p = make_double2(cs, sn);
  }
  for (int e = 0; e < cnt; ++e) {
    dst[e] = p;
    p = cmul(p, z);
  }
}

// Phase tables of a block for TP particles from j0 on: per particle (row of
// P.gts entries) the columns lo .. lo + ncol - 1, then the prefix windows of
// axis 0 and (d = 3) axis 1. A unit is up to 16 entries of one table of one
// particle; a warp's threads share the unit and differ in the particle.
template <int D, int TP>
__device__ __forceinline__ void grid_tables(const ProbDev& P, const GridBlock& B,
                                            const double* __restrict__ s, int j0, int nj,
                                            double2* tab) {
  const int uz = (B.ncol + 15) >> 4, u0 = (B.c0 + 15) >> 4, u1 = D == 3 ? (B.c1 + 15) >> 4 : 0;
  const int total = (uz + u0 + u1) * TP;
  for (int w = threadIdx.x; w < total; w += blockDim.x) {
    const int j = w & (TP - 1), u = w / TP;
    const bool live = j < nj;
    const double* sj = s + (size_t)(j0 + (live ? j : 0)) * D;
    double2* row = tab + (size_t)j * P.gts;
    if (u < uz) {
      const int L = (B.ncol + uz - 1) / uz, e0 = u * L;
      grid_powers(row + e0, B.lo + e0, min(L, B.ncol - e0), 1, sj[D - 1], live, 1.0);
    } else if (u < uz + u0) {
      const int q = u - uz, L = (B.c0 + u0 - 1) / u0, e0 = q * L;
      // dead particles drop out of every product through a zero prefix
      grid_powers(row + B.ncol + e0, B.m0 + e0, min(L, B.c0 - e0), P.gstep, sj[0], live, 0.0);
    } else if constexpr (D == 3) {
      const int q = u - uz - u0, L = (B.c1 + u1 - 1) / u1, e0 = q * L;
      grid_powers(row + B.ncol + B.c0 + e0, B.m1 + e0, min(L, B.c1 - e0), 1, sj[1], live, 1.0);
    }
  }
}

// Table offsets of run `r` of a block (its prefix phase is the product).
template <int D>
__device__ __forceinline__ void run_offsets(const GridBlock& B, const GridRun& g, int& o0, int& o1) {
  o0 = B.ncol + g.n0 - B.m0;
  o1 = D == 3 ? B.ncol + B.c0 + g.n1 - B.m1 : 0;
}
template <int D>
__device__ __forceinline__ double2 run_phase(const double2* row, int o0, int o1) {
  const double2 a = row[o0];
  if (D == 3) return cmul(a, row[o1]);
  return a;
}

// Pass 1 of one (lane, particle tile, block): a warp owns a strip, 4 DMMAs per
// 8 columns and 4 particles. NT: column tiles of 8 a warp may hold.
template <int D, int NT>
__device__ __forceinline__ void grid_pass1_body(const ProbDev& P, const EvalLane& ln, int tile,
                                                int blk, int rot, double2* tab) {
  constexpr int KC = kGridChunk;
  const GridBlock B = P.gblk[blk];
  const int jt0 = tile * P.gtile, jt1 = min(P.N, jt0 + P.gtile);
  const int lane = threadIdx.x & 31, t = lane & 3, pr = grid_perm(lane >> 2);
  // warps take strips in rotation over the CTAs, so that a block of fewer than
  // four strips does not leave the same quarter of every SM idle
  const int sidx = ((threadIdx.x >> 5) + rot) & 3;
  GridStrip S{};
  int o0 = 0, o1 = 0;
  if (sidx < B.nstrip) {
    S = P.gstrip[B.strip0 + sidx];
    run_offsets<D>(B, P.grun[S.run0 + min(pr, S.nrun - 1)], o0, o1);
  }
  const int nt = (S.nq + 1) >> 1;
  double p1[NT][2], p2[NT][2], p3[NT][2], p4[NT][2];
#pragma unroll
  for (int i = 0; i < NT; ++i)
#pragma unroll
    for (int c = 0; c < 2; ++c) p1[i][c] = p2[i][c] = p3[i][c] = p4[i][c] = 0.0;
  for (int j0 = jt0; j0 < jt1; j0 += KC) {
    __syncthreads();   // the previous chunk's products are done
    grid_tables<D, KC>(P, B, ln.s, j0, jt1 - j0, tab);
    __syncthreads();
    if (nt > 0) {
      const double2* row = tab + (size_t)t * P.gts;
      const int dead = min(KC, (jt1 - j0 + 3) & ~3);
      for (int j = 0; j < dead; j += 4, row += 4 * P.gts) {
        const double2 a = run_phase<D>(row, o0, o1);
#pragma unroll
        for (int i = 0; i < NT; ++i) {
          if (i < nt) {
            const double2 z = row[8 * i + pr];
            dmma(p1[i], a.x, z.x);
            dmma(p2[i], a.y, z.y);
            dmma(p3[i], a.x, z.y);
            dmma(p4[i], a.y, z.x);
          }
        }
      }
    }
  }
  if (nt == 0) return;
  // lane holds the cells (run pr, columns 8 i + t and 8 i + t + 4): one slot of
  // each of the tile's two quads
  double2* out = ln.part + 2 * ((size_t)tile * P.gslots + S.slot0 + lane);
#pragma unroll
  for (int i = 0; i < NT; ++i) {
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const int q = 2 * i + c;
      if (q < S.nq) {
        out[64 * q] = make_double2(p1[i][c] - p2[i][c], p3[i][c] + p4[i][c]);
        out[64 * q + 1] = make_double2(p1[i][c] + p2[i][c], p4[i][c] - p3[i][c]);
      }
    }
  }
}

// Reduction of one slot: rho of its two k-set rows summed over the tiles in
// tile order, the slot's part of sum w |rho|^2 and its pass-2 weights (zero
// where the grid has no k-set row).
template <bool ONE_D>
__device__ __forceinline__ double grid_reduce_slot(const ProbDev& P, const EvalLane& ln, int slot) {
  const GridQuad Q = P.gquad[slot >> 5];
  const int lane = slot & 31, r = grid_perm(lane >> 2), c = Q.c0 + (lane & 3);
  int kp = -1, km = -1, n0 = 0;
  if (r < Q.nrun) {
    const GridRun g = P.grun[Q.run0 + r];
    n0 = g.n0;
    if (c >= g.a && c <= g.b) kp = g.kstart + c - g.a;
    if (c > 0 && -c >= g.a && -c <= g.b) km = g.kstart - c - g.a;
  }
  double2 tp = make_double2(0.0, 0.0), tm = tp;
  double e = 0.0;
  if (kp >= 0 || km >= 0) {
    const double2* __restrict__ col = ln.part + 2 * (size_t)slot;
    const size_t stride = 2 * (size_t)P.gslots;
    const int nt = P.gntile;
    int q = 0;
    for (; q + 8 <= nt; q += 8) {   // eight tile rows in flight, added in tile order
      double2 x[8], y[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        x[u] = col[(q + u) * stride];
        y[u] = col[(q + u) * stride + 1];
      }
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        tp.x += x[u].x;
        tp.y += x[u].y;
        tm.x += y[u].x;
        tm.y += y[u].y;
      }
    }
    for (; q < nt; ++q) {
      const double2 x = col[q * stride], y = col[q * stride + 1];
      tp.x += x.x;
      tp.y += x.y;
      tm.x += y.x;
      tm.y += y.y;
    }
    if (kp >= 0) {
      ln.rho[kp] = tp;
      const double w = P.w_run[kp];
      e += w * (tp.x * tp.x + tp.y * tp.y);
      tp = make_double2(w * tp.x, w * tp.y);
    } else {
      tp = make_double2(0.0, 0.0);
    }
    if (km >= 0) {
      ln.rho[km] = tm;
      const double w = P.w_run[km];
      e += w * (tm.x * tm.x + tm.y * tm.y);
      tm = make_double2(w * tm.x, w * tm.y);
    } else {
      tm = make_double2(0.0, 0.0);
    }
  }
  // -conj(w rho): T = sum_c -(conj(p+) z^c + conj(p-) conj(z^c)), u and v parts
  const double2 re_t = make_double2(-(tp.x + tm.x), tm.y - tp.y);
  const double2 im_t = make_double2(tp.y + tm.y, tm.x - tp.x);
  const double2 re_d = make_double2(tm.x - tp.x, -(tp.y + tm.y));
  const double2 im_d = make_double2(tp.y - tm.y, -(tp.x + tm.x));
  constexpr int NW = ONE_D ? 2 : 4;
  double2* w = ln.rhow + (size_t)(slot >> 5) * (32 * NW) + lane;
  const double cd = (double)c;
  if (ONE_D) {
    // one axis: the weights n = q S + c of both kinds in one sum
    const double m = (double)n0 * P.gstep;
    w[0] = make_double2(m * re_t.x + cd * re_d.x, m * re_t.y + cd * re_d.y);
    w[32] = make_double2(m * im_t.x + cd * im_d.x, m * im_t.y + cd * im_d.y);
  } else {
    w[0] = re_t;
    w[32] = im_t;
    w[64] = make_double2(cd * re_d.x, cd * re_d.y);
    w[96] = make_double2(cd * im_d.x, cd * im_d.y);
  }
  return e;
}

// Pass 2 of one (lane, 64-particle tile): a warp owns 16 particles (two
// fragment columns of 8) and walks every strip of every block: per quad and
// 8 particles 8 DMMAs (4 in 1-D) from 4 (2) coalesced 16-byte weight loads and
// one table read, then the strip's rows are weighted by their prefix phases.
template <int D>
__device__ __forceinline__ void grid_pass2_body(const ProbDev& P, const EvalLane& ln, int tile,
                                                double2* tab) {
  constexpr int TP = kGridTile2, NW = D == 1 ? 2 : 4, NP = 2;
  const int j0 = tile * TP, nj = min(TP, P.N - j0);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, t = lane & 3;
  const int pr = grid_perm(lane >> 2);
  double G[NP][2][D];
#pragma unroll
  for (int p = 0; p < NP; ++p)
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
      for (int x = 0; x < D; ++x) G[p][c][x] = 0.0;
  const double2* wtab = tab + (size_t)(warp * 16) * P.gts;
  for (int b = 0; b < P.ngblk; ++b) {
    const GridBlock B = P.gblk[b];
    __syncthreads();
    grid_tables<D, TP>(P, B, ln.s, j0, nj, tab);
    __syncthreads();
    for (int si = 0; si < B.nstrip; ++si) {
      const GridStrip S = P.gstrip[B.strip0 + si];
      double acc[NW][NP][2];
#pragma unroll
      for (int w = 0; w < NW; ++w)
#pragma unroll
        for (int p = 0; p < NP; ++p) acc[w][p][0] = acc[w][p][1] = 0.0;
      const double2* __restrict__ wq = ln.rhow + (size_t)(S.slot0 >> 5) * (32 * NW) + lane;
      const double2* zr = wtab + (size_t)pr * P.gts + t;
      double2 w[NW];
#pragma unroll
      for (int x = 0; x < NW; ++x) w[x] = wq[32 * x];
      for (int q = 0; q < S.nq; ++q) {
        double2 wn[NW];
        wq += 32 * NW;
        if (q + 1 < S.nq) {
#pragma unroll
          for (int x = 0; x < NW; ++x) wn[x] = wq[32 * x];
        }
#pragma unroll
        for (int p = 0; p < NP; ++p) {
          const double2 z = zr[(size_t)(8 * p) * P.gts + 4 * q];
#pragma unroll
          for (int x = 0; x < NW; ++x) dmma(acc[x][p], w[x].x, z.x);
#pragma unroll
          for (int x = 0; x < NW; ++x) dmma(acc[x][p], w[x].y, z.y);
        }
#pragma unroll
        for (int x = 0; x < NW; ++x) w[x] = wn[x];
      }
      // lane holds T, T' of run pr for particles t and t + 4 of each eight
      const GridRun g = P.grun[S.run0 + min(pr, S.nrun - 1)];
      int o0, o1;
      run_offsets<D>(B, g, o0, o1);
#pragma unroll
      for (int p = 0; p < NP; ++p)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const double2 a = run_phase<D>(wtab + (size_t)(8 * p + 4 * c + t) * P.gts, o0, o1);
          const double h = a.x * acc[1][p][c] + a.y * acc[0][p][c];
          if (D == 1) {
            G[p][c][0] += h;
          } else {
            G[p][c][0] += (double)g.n0 * h;
            if (D == 3) G[p][c][1] += (double)g.n1 * h;
            G[p][c][D - 1] += a.x * acc[3][p][c] + a.y * acc[2][p][c];
          }
        }
    }
  }
  // sum over the strip rows (lanes 4 apart); lanes 0..3 hold the particles
#pragma unroll
  for (int p = 0; p < NP; ++p)
#pragma unroll
    for (int c = 0; c < 2; ++c) {
#pragma unroll
      for (int x = 0; x < D; ++x) {
        double v = G[p][c][x];
        v += __shfl_xor_sync(0xffffffffu, v, 4);
        v += __shfl_xor_sync(0xffffffffu, v, 8);
        v += __shfl_xor_sync(0xffffffffu, v, 16);
        G[p][c][x] = v;
      }
      const int j = warp * 16 + 8 * p + 4 * c + t;
      if (lane < 4 && j < nj) {
        double* gj = ln.g + (size_t)(j0 + j) * D;
#pragma unroll
        for (int x = 0; x < D; ++x) gj[x] = P.gpref * G[p][c][x];
      }
    }
}

}  // namespace

}  // namespace cco
