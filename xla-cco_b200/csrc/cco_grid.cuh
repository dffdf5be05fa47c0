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
// gradient): 256 lanes of d=2 N=1000 M=802 285 -> 165 us, 64 lanes of d=3
// N=4000 M=5413 2765 -> 1187 us, one lane of d=2 N=20000 M=18000 600 -> 288 us,
// one of d=1 N=7777 M=3732 108 -> 56 us; forces up to 2.8 times closer to the
// exact sums. Bound: the FP64 pipe (DMMA 62% active on the 256 lanes; the two
// passes' DMMAs alone take 87 us there, a fifth of them on padded cells, and
// what the table fills, the weight loads (33.2 against 36.8 TFLOP/s in a loop
// of their own) and a kernel's start and end add comes on top: neither a
// producer / consumer split of the warps, nor loading items and weights further
// ahead, nor offsetting the CTAs of an SM made them overlap better).
//
// Tiling. Runs are sorted by folded length in strips of 8; a strip's columns
// are 4-column quads. A slot (quad, lane) is one cell: lane = 4 row + t holds
// run grid_perm(row) of the strip and column 4 quad + t. Partials and the
// pass-2 weights are stored slot by slot, which makes both coalesced and is
// the order the matrix fragments want. Up to 4 strips and 32 columns form a
// block, whose phase tables a CTA builds together in shared memory: at most 55
// entries per particle, so that four CTAs with 64 particles' tables share an SM
// (wider blocks, one or two CTAs per SM, ran N=20000 in 416 instead of 296 us).
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

// Phases that the tables of an evaluation start from. Problems of kGridRootsMin
// blocks or more, or of more than 8 tiles a block, have a kernel form them once
// per particle (k_grid_roots): per virtual axis v (prefix 0, prefix 1, columns) the
// root exp(2 pi i step s) and the seeds exp(2 pi i 16 q step s), q = 1 .., by
// FP64 sincospi of the exactly reduced argument; word (P.groff[v] + q) N + j of
// the lane's roots area. Forming them in the passes, once per block, took 350 of
// 550 FP64 instructions per particle and pass on an 802-row set; with 10 blocks
// (64 lanes of d=3 N=4000) taking them out cut the passes from 1260 to 1130 us
// for a 9 us kernel. With few blocks the kernel costs what it saves (one block,
// 256 lanes of N=1000: passes -8 us, kernel +9 us) and a lone small evaluation
// one launch more, so there the passes form them.
template <int D>
__device__ __forceinline__ void grid_roots(const ProbDev& P, const EvalLane& ln, int w) {
  const int N = P.N, e = w / N, j = w - e * N;
  const int v = e >= P.groff[2] ? 2 : e >= P.groff[1] ? 1 : 0;
  const int q = e - P.groff[v];
  const double s = ln.s[(size_t)j * D + (v == 2 ? D - 1 : v)];
  const int step = v == 0 ? P.gstep : 1;
  double sn, cs;
  sincos_2pi_ms((double)(q == 0 ? step : 16 * q * step), s, &sn, &cs);
  ln.roots[w] = make_double2(cs, sn);
}

// A unit of a block's phase tables: the entries of one virtual axis whose
// exponents share their multiple of 16. Entry i of the unit is exponent 16 q + i;
// [i0, i1) are inside the block's window and go to row words off + i.
struct GridUnit {
  int v, q, i0, i1, off;
};
__device__ __forceinline__ int grid_floor16(int m) { return m >> 4; }
__device__ __forceinline__ GridUnit grid_unit(const GridBlock& B, int u, int uz, int u0) {
  int v, m, cnt, first;
  if (u < uz) {
    v = 2; m = B.lo; cnt = B.ncol; first = 0;
  } else if (u < uz + u0) {
    u -= uz;
    v = 0; m = B.m0; cnt = B.c0; first = B.ncol;
  } else {
    u -= uz + u0;
    v = 1; m = B.m1; cnt = B.c1; first = B.ncol + B.c0;
  }
  GridUnit U;
  U.v = v;
  U.q = grid_floor16(m) + u;
  U.i0 = max(0, m - 16 * U.q);
  U.i1 = min(16, m + cnt - 16 * U.q);
  U.off = first + 16 * U.q - m;
  return U;
}
__device__ __forceinline__ int grid_units(int m, int cnt) {
  return cnt > 0 ? grid_floor16(m + cnt - 1) - grid_floor16(m) + 1 : 0;
}

// Two units' first phases (exponents 16 q) and roots for particle j.
template <int D, bool ROOTS>
__device__ __forceinline__ void grid_seeds(const ProbDev& P, const EvalLane& ln, const GridUnit& A,
                                           const GridUnit& C, int j, double2& za, double2& a0,
                                           double2& zc, double2& c0) {
  if constexpr (ROOTS) {
    const double2* ra = ln.roots + (size_t)P.groff[A.v] * P.N + j;
    const double2* rc = ln.roots + (size_t)P.groff[C.v] * P.N + j;
    za = ra[0];
    zc = rc[0];
    a0 = A.q != 0 ? ra[(size_t)abs(A.q) * P.N] : zeroth_power(za);
    c0 = C.q != 0 ? rc[(size_t)abs(C.q) * P.N] : zeroth_power(zc);
    if (A.q < 0) a0.y = -a0.y;
    if (C.q < 0) c0.y = -c0.y;
  } else {
    const double* sj = ln.s + (size_t)j * D;
    const double sa = sj[A.v == 2 ? D - 1 : A.v], sc = sj[C.v == 2 ? D - 1 : C.v];
    const int ka = A.v == 0 ? P.gstep : 1, kc = C.v == 0 ? P.gstep : 1;
    sincos_2pi_ms((double)ka, sa, &za.y, &za.x);
    sincos_2pi_ms((double)kc, sc, &zc.y, &zc.x);
    a0 = zeroth_power(za);
    c0 = zeroth_power(zc);
    if (A.q != 0 || C.q != 0) {   // warp-uniform
      sincos_2pi_ms((double)(16 * A.q * ka), sa, &a0.y, &a0.x);
      sincos_2pi_ms((double)(16 * C.q * kc), sc, &c0.y, &c0.x);
    }
  }
}

// Phase tables of a block for TP particles from j0 on: per particle (row of
// P.gts entries) the columns lo .. lo + ncol - 1, then the prefix windows of
// axis 0 and (d = 3) axis 1. Each unit goes on from its seed by products with
// the root, even and odd entries apart (at most 8 products of the root's
// square). A thread forms two units of one particle at a time: four independent
// chains, since a chain's latency (its operations queue behind other warps'
// DMMAs) is what a stage waits for. A warp's threads share the units and differ
// in the particle. Dead particles (past the tile's end) get a zero axis-0
// prefix and drop out of every product.
template <int D, bool ROOTS, int TP>
__device__ __forceinline__ void grid_tables(const ProbDev& P, const GridBlock& B,
                                            const EvalLane& ln, int j0, int nj,
                                            int thread, double2* tab) {
  const int uz = grid_units(B.lo, B.ncol), u0 = grid_units(B.m0, B.c0);
  const int units = uz + u0 + (D == 3 ? grid_units(B.m1, B.c1) : 0);
  const int pairs = (units + 1) >> 1, gts = P.gts;
  for (int w = thread; w < pairs * TP; w += kGridThreads) {
    const int j = w & (TP - 1), u = w / TP;
    const bool live = j < nj;
    const int jj = j0 + (live ? j : 0);
    const GridUnit A = grid_unit(B, u, uz, u0);
    GridUnit C = A;
    if (u + pairs < units) C = grid_unit(B, u + pairs, uz, u0);
    else C.i1 = 0;
    double2 za, zc, a0, c0;
    grid_seeds<D, ROOTS>(P, ln, A, C, jj, za, a0, zc, c0);
    if (!live && A.v == 0) a0 = make_double2(0.0, 0.0);
    if (!live && C.v == 0) c0 = make_double2(0.0, 0.0);
    double2 a1 = cmul(a0, za), c1 = cmul(c0, zc);
    za = cmul(za, za);
    zc = cmul(zc, zc);
    double2 *da = tab + j * gts + A.off, *dc = tab + j * gts + C.off;
    const int most = max(A.i1, C.i1);
    for (int i = 0; i < most; i += 2) {
      if (i >= A.i0 && i < A.i1) da[i] = a0;
      if (i + 1 >= A.i0 && i + 1 < A.i1) da[i + 1] = a1;
      if (i >= C.i0 && i < C.i1) dc[i] = c0;
      if (i + 1 >= C.i0 && i + 1 < C.i1) dc[i + 1] = c1;
      a0 = cmul(a0, za);
      a1 = cmul(a1, za);
      c0 = cmul(c0, zc);
      c1 = cmul(c1, zc);
    }
  }
}

// Tables of a block of a line grid: strip by strip the powers of the line's
// phase z = exp(2 pi i v . s) for its columns and of z^step from row q0 on, a
// thread per (strip, particle), both chains even and odd apart.
template <int D, int TP>
__device__ __forceinline__ void grid_line_tables(const ProbDev& P, const GridBlock& B,
                                                 const EvalLane& ln, int j0, int nj, int thread,
                                                 double2* tab) {
  const int gts = P.gts;
  for (int w = thread; w < B.nstrip * TP; w += kGridThreads) {
    const int j = w & (TP - 1), st = B.strip0 + w / TP;
    const GridLine L = P.gline[st];
    const bool live = j < nj;
    const double* sj = ln.s + (size_t)(j0 + (live ? j : 0)) * D;
    double n1[D], nS[D], nQ[D];
#pragma unroll
    for (int a = 0; a < D; ++a) {
      n1[a] = (double)L.n[a];
      nS[a] = (double)(L.n[a] * L.step);
      nQ[a] = (double)(L.n[a] * L.step * L.q0);
    }
    double2 z, y, r0 = make_double2(1.0, 0.0);
    sincos_2pi_dot<D>(n1, sj, &z.y, &z.x);
    double2 c0 = zeroth_power(z);
    sincos_2pi_dot<D>(nS, sj, &y.y, &y.x);
    if (L.q0 != 0) sincos_2pi_dot<D>(nQ, sj, &r0.y, &r0.x);
    if (!live) r0 = make_double2(0.0, 0.0);
    double2 c1 = z, r1 = cmul(r0, y);
    z = cmul(z, z);
    y = cmul(y, y);
    double2* dc = tab + j * gts + P.gstrip[st].col0;
    double2* dr = dc + L.ncol;
    for (int e = 0; e < L.ncol; e += 2) {   // ncol is a multiple of 8
      dc[e] = c0;
      dc[e + 1] = c1;
      c0 = cmul(c0, z);
      c1 = cmul(c1, z);
      if (e < 8) {
        dr[e] = r0;
        dr[e + 1] = r1;
        r0 = cmul(r0, y);
        r1 = cmul(r1, y);
      }
    }
  }
}

// Prefix phase of a run from its table offsets (one particle's row).
template <int D>
__device__ __forceinline__ double2 run_phase(const double2* row, int o0, int o1) {
  const double2 a = row[o0];
  if (D == 3) return cmul(a, row[o1]);
  return a;
}

// CTA barrier that warps may meet in different branches (bar.sync counts
// arrivals, wherever they come from).
__device__ __forceinline__ void bar_cta() { asm volatile("bar.sync 0;" ::: "memory"); }

// What a stage's block and item are (loaded once per CTA).
struct GridStage {
  double2* buf;   // pass 1: the partials, pass 2: the weights
  double* g;
  double gpref;
  int tile, N, gtile, gts, gslots, ngblk, nstrip, ntile;
  GridStrip strip[kGridStrips];
  GridRow row[8 * kGridStrips];
};
__device__ __forceinline__ void grid_describe(GridStage& S, const ProbDev& P, const GridBlock& B,
                                              double2* buf, double* g, int tile) {
  const int t = threadIdx.x;
  if (t < 8 * B.nstrip) S.row[t] = P.grow[8 * B.strip0 + t];
  if (t >= 32 && t < 32 + B.nstrip) S.strip[t - 32] = P.gstrip[B.strip0 + t - 32];
  if (t == 64) {
    S.buf = buf;
    S.g = g;
    S.gpref = P.gpref;
    S.tile = tile;
    S.N = P.N;
    S.gtile = P.gtile;
    S.gts = P.gts;
    S.gslots = P.gslots;
    S.ngblk = P.ngblk;
    S.nstrip = B.nstrip;
    S.ntile = B.ntile;
  }
}

// Pass 1 products of one item by a warp that owns the CNT tiles lo .. lo + CNT
// - 1 of the block: 4 DMMAs per tile and 4 particles. SAME: the tiles are of
// one strip and share the prefix phase. CNT = 0: the warp only fills.
template <int D, bool ROOTS, int CNT, bool SAME, bool LINES>
__device__ __forceinline__ void grid_pass1_item(const ProbDev& P, const GridBlock& B,
                                                const EvalLane& ln, const GridStage& S, int lo,
                                                double2* tab) {
  constexpr int NA = SAME ? 1 : CNT, NC = CNT > 0 ? CNT : 1;
  const int lane = threadIdx.x & 31, t = lane & 3, pr = grid_perm(lane >> 2);
  const int jt0 = S.tile * S.gtile, jt1 = min(S.N, jt0 + S.gtile), gts = S.gts;
  // tile i: run offsets of the lane's row, column, slot (doubled, plus one if
  // the tile's second quad exists)
  int o0[NC], o1[NC], col[NC], slot[NC];
  double p1[NC][2], p2[NC][2], p3[NC][2], p4[NC][2];
  int at = 0, si = 0, nq = S.strip[0].nq;
#pragma unroll
  for (int i = 0; i < CNT; ++i) {
    while (lo + i - at >= ((nq + 1) >> 1)) {
      at += (nq + 1) >> 1;
      nq = S.strip[++si].nq;
    }
    const int c = lo + i - at;
    o0[i] = S.row[8 * si + pr].o0;
    o1[i] = S.row[8 * si + pr].o1;
    col[i] = S.strip[si].col0 + 8 * c + pr;
    slot[i] = 2 * (S.strip[si].slot0 + 64 * c) + (2 * c + 1 < nq ? 1 : 0);
#pragma unroll
    for (int h = 0; h < 2; ++h) p1[i][h] = p2[i][h] = p3[i][h] = p4[i][h] = 0.0;
  }
  for (int j0 = jt0;;) {
    if (CNT > 0) {
      const double2* row = tab + t * gts;
      const int nj = min(kGridChunk, (jt1 - j0 + 3) & ~3);
#pragma unroll 2
      for (int j = 0; j < nj; j += 4, row += 4 * gts) {
        double2 a[NC], z[NC];
#pragma unroll
        for (int i = 0; i < CNT; ++i) z[i] = row[col[i]];
#pragma unroll
        for (int i = 0; i < NA; ++i) a[i] = run_phase<D>(row, o0[i], o1[i]);
#pragma unroll
        for (int i = 0; i < CNT; ++i) {
          const double2 ai = a[SAME ? 0 : i];
          dmma(p1[i], ai.x, z[i].x);
          dmma(p2[i], ai.y, z[i].y);
          dmma(p3[i], ai.x, z[i].y);
          dmma(p4[i], ai.y, z[i].x);
        }
      }
    }
    j0 += kGridChunk;
    if (j0 >= jt1) break;
    bar_cta();
    if constexpr (LINES) grid_line_tables<D, kGridChunk>(P, B, ln, j0, jt1 - j0, threadIdx.x, tab);
    else grid_tables<D, ROOTS, kGridChunk>(P, B, ln, j0, jt1 - j0, threadIdx.x, tab);
    bar_cta();
  }
  // lane holds the cells (run pr, columns t and t + 4 of a tile): a slot of each
  // of the tile's two quads
  double2* const out = S.buf + 2 * ((size_t)S.tile * S.gslots + lane);
#pragma unroll
  for (int i = 0; i < CNT; ++i) {
    double2* o = out + (slot[i] & ~1);
    o[0] = make_double2(p1[i][0] - p2[i][0], p3[i][0] + p4[i][0]);
    o[1] = make_double2(p1[i][0] + p2[i][0], p4[i][0] - p3[i][0]);
    if (slot[i] & 1) {
      o[64] = make_double2(p1[i][1] - p2[i][1], p3[i][1] + p4[i][1]);
      o[65] = make_double2(p1[i][1] + p2[i][1], p4[i][1] - p3[i][1]);
    }
  }
}

// Pass 1 of one item (lane, tile, block): the block's 8 x 8-cell tiles in strip
// order are cut into four equal ranges, one per warp (at most NT tiles), so
// that uneven strips do not leave warps idle.
template <int D, bool ROOTS, int NT, bool LINES>
__device__ __forceinline__ void grid_pass1(const ProbDev& P, const EvalLane& ln, int tile, int blk,
                                           GridStage& S, double2* tab) {
  const GridBlock B = P.gblk[blk];
  const int jt0 = tile * P.gtile;
  grid_describe(S, P, B, ln.part, nullptr, tile);
  if constexpr (LINES)
    grid_line_tables<D, kGridChunk>(P, B, ln, jt0, min(P.N - jt0, P.gtile), threadIdx.x, tab);
  else
    grid_tables<D, ROOTS, kGridChunk>(P, B, ln, jt0, min(P.N - jt0, P.gtile), threadIdx.x, tab);
  bar_cta();
  const int warp = threadIdx.x >> 5;
  const int lo = B.ntile * warp >> 2, hi = B.ntile * (warp + 1) >> 2;
  int at = 0, si = 0;   // the strip of tile lo: whether tile hi - 1 is of it
  while (lo >= at + ((S.strip[si].nq + 1) >> 1)) at += (S.strip[si++].nq + 1) >> 1;
  const bool same = hi <= at + ((S.strip[si].nq + 1) >> 1);
#define CCO_GRID_CASE(CNT)                                                                     \
  if (CNT <= NT && hi - lo == CNT) {                                                           \
    if (same) grid_pass1_item<D, ROOTS, CNT <= NT ? CNT : 0, true, LINES>(P, B, ln, S, lo, tab);   \
    else grid_pass1_item<D, ROOTS, CNT <= NT ? CNT : 0, false, LINES>(P, B, ln, S, lo, tab);       \
  }
  CCO_GRID_CASE(0)
  CCO_GRID_CASE(1)
  CCO_GRID_CASE(2)
  CCO_GRID_CASE(3)
#undef CCO_GRID_CASE
  bar_cta();   // the tables and the description are free again
}

// Reduction of one slot: rho of its two k-set rows summed over the tiles in
// tile order, the slot's part of sum w |rho|^2 and its pass-2 weights (zero
// where the grid has no k-set row).
template <bool ONE_D>
__device__ __forceinline__ double grid_reduce_slot(const ProbDev& P, const EvalLane& ln, int slot) {
  const bool lines = P.grid == 2;
  GridQuad Q{};
  if (!lines) Q = P.gquad[slot >> 5];
  const int lane = slot & 31, r = grid_perm(lane >> 2), c = Q.c0 + (lane & 3);
  int kp = -1, km = -1, n0 = 0;
  if (lines) {
    const int2 k = P.gslotk[slot];
    kp = k.x;
    km = k.y;
  } else if (r < Q.nrun) {
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
  if (lines) {   // the weighted density of the recurrence pass 2
    if (kp >= 0) ln.rhow[kp] = tp;
    if (km >= 0) ln.rhow[km] = tm;
    return e;
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

// Sum over a strip's rows (lanes 4 apart) of 8 values: halves are exchanged and
// added three times, so row r ends with the total of value r (7 shuffles where
// summing every value everywhere takes 24).
__device__ __forceinline__ double grid_row_sum(const double (&v)[8], int row) {
  double a[4], b[2];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const bool up = row & 4;
    const double mine = up ? v[i + 4] : v[i], other = up ? v[i] : v[i + 4];
    a[i] = mine + __shfl_xor_sync(0xffffffffu, other, 16);
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const bool up = row & 2;
    const double mine = up ? a[i + 2] : a[i], other = up ? a[i] : a[i + 2];
    b[i] = mine + __shfl_xor_sync(0xffffffffu, other, 8);
  }
  const bool up = row & 1;
  const double mine = up ? b[1] : b[0], other = up ? b[0] : b[1];
  return mine + __shfl_xor_sync(0xffffffffu, other, 4);
}

// Pass 2 of one item (lane, 64-particle tile): a warp owns 16 particles (two
// fragment columns of 8) and walks every strip of every block: per quad and 8
// particles 8 DMMAs (4 in 1-D) from 4 (2) coalesced 16-byte weight loads, one
// quad ahead, and one table read; then the strip's rows are weighted by their
// prefix phases. The weights of all quads are one stream.
template <int D, bool ROOTS>
__device__ __forceinline__ void grid_pass2(const ProbDev& P, const EvalLane& ln, int tile,
                                           GridStage& S, double2* tab) {
  constexpr int NW = D == 1 ? 2 : 4, NP = 2;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, t = lane & 3, r8 = lane >> 2;
  const int pr = grid_perm(r8);
  const int j0 = tile * kGridTile2, nj = min(kGridTile2, P.N - j0), gts = P.gts, nb = P.ngblk;
  const double2* __restrict__ wq = ln.rhow + lane;
  const double2* const wlast = wq + (size_t)((P.gslots >> 5) - 1) * (32 * NW);
  double2 w[NW];
#pragma unroll
  for (int x = 0; x < NW; ++x) w[x] = wq[32 * x];
  if (wq < wlast) wq += 32 * NW;
  double G[D][NP][2];
#pragma unroll
  for (int x = 0; x < D; ++x)
#pragma unroll
    for (int p = 0; p < NP; ++p) G[x][p][0] = G[x][p][1] = 0.0;
  const double2* wtab = tab + warp * 16 * gts;
  for (int b = 0; b < nb; ++b) {
    const GridBlock B = P.gblk[b];
    grid_describe(S, P, B, nullptr, nullptr, tile);
    grid_tables<D, ROOTS, kGridTile2>(P, B, ln, j0, nj, threadIdx.x, tab);
    __syncthreads();
    for (int si = 0; si < B.nstrip; ++si) {
      const int nq = S.strip[si].nq;
      const GridRow R = S.row[8 * si + pr];
      double acc[NW][NP][2];
#pragma unroll
      for (int x = 0; x < NW; ++x)
#pragma unroll
        for (int p = 0; p < NP; ++p) acc[x][p][0] = acc[x][p][1] = 0.0;
      const double2* zr = wtab + pr * gts + t;
      for (int q = 0; q < nq; ++q, zr += 4) {
        double2 wn[NW], z[NP];
#pragma unroll
        for (int p = 0; p < NP; ++p) z[p] = zr[8 * p * gts];
#pragma unroll
        for (int x = 0; x < NW; ++x) wn[x] = wq[32 * x];   // past the end: the last quad again
        if (wq < wlast) wq += 32 * NW;
#pragma unroll
        for (int p = 0; p < NP; ++p)
#pragma unroll
          for (int x = 0; x < NW; ++x) dmma(acc[x][p], w[x].x, z[p].x);
#pragma unroll
        for (int p = 0; p < NP; ++p)
#pragma unroll
          for (int x = 0; x < NW; ++x) dmma(acc[x][p], w[x].y, z[p].y);
#pragma unroll
        for (int x = 0; x < NW; ++x) w[x] = wn[x];
      }
      // lane holds T, T' of run pr for particles t and t + 4 of each eight
#pragma unroll
      for (int p = 0; p < NP; ++p)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const double2 a = run_phase<D>(wtab + (8 * p + 4 * c + t) * gts, R.o0, R.o1);
          const double h = a.x * acc[1][p][c] + a.y * acc[0][p][c];
          if (D == 1) {
            G[0][p][c] += h;
          } else {
            G[0][p][c] += (double)R.n0 * h;
            if (D == 3) G[1][p][c] += (double)R.n1 * h;
            G[D - 1][p][c] += a.x * acc[3][p][c] + a.y * acc[2][p][c];
          }
        }
    }
    __syncthreads();   // the tables and the description are free again
  }
  // value 4 x + 2 p + c of the row sums is axis x of particle 8 p + 4 c + t
#pragma unroll
  for (int h = 0; h < D; h += 2) {
    double v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int x = h + (i >> 2);
      v[i] = x < D ? G[x < D ? x : 0][(i >> 1) & 1][i & 1] : 0.0;
    }
    const double tot = grid_row_sum(v, r8);
    const int x = h + (r8 >> 2), j = warp * 16 + 8 * ((r8 >> 1) & 1) + 4 * (r8 & 1) + t;
    if (x < D && j < nj) ln.g[(size_t)(j0 + j) * D + x] = P.gpref * tot;
  }
}

}  // namespace

}  // namespace cco
