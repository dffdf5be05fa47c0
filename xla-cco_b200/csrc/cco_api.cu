// C ABI of libcco: problems, evaluation and the batched relax drivers.
#include <algorithm>
#include <array>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <numeric>
#include <string>
#include <vector>

#include "cco_host.cuh"
#include "cco_internal.cuh"
#include "cco_opt.cuh"

using namespace cco;

namespace {
thread_local std::string g_last_error;
constexpr int kMaxPoolDevices = 64;
std::mutex g_pool_mu;
cudaMemPool_t g_pool[kMaxPoolDevices] = {};
}  // namespace

namespace cco {

int fail(int code, const char* fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof(buf), fmt, ap);
  va_end(ap);
  g_last_error = buf;
  return code;
}

int cuda_fail(cudaError_t e, const char* what) {
  if (e == cudaErrorMemoryAllocation) return fail(CCO_ERR_OOM, "%s: %s", what, cudaGetErrorString(e));
  return fail(CCO_ERR_DEVICE, "%s: %s", what, cudaGetErrorString(e));
}

// One pool per device that keeps its memory (release threshold = max): a
// relaxation's lane records are reused by the next call instead of being
// unmapped at every synchronize, as the default pool (threshold 0) would do.
cudaError_t device_pool(cudaMemPool_t* out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= kMaxPoolDevices) return cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> lk(g_pool_mu);
  if (!g_pool[dev]) {
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.handleTypes = cudaMemHandleTypeNone;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    cudaMemPool_t pool;
    e = cudaMemPoolCreate(&pool, &props);
    if (e != cudaSuccess) return e;
    uint64_t keep = UINT64_MAX;
    e = cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
    if (e != cudaSuccess) return e;
    g_pool[dev] = pool;
  }
  *out = g_pool[dev];
  return cudaSuccess;
}

}  // namespace cco


namespace {

// ----------------------------------------------------------- problem build
// Digit layout of one axis for |n| <= R with `nlev` levels: base b with
// b^nlev > R; level 0 holds z^0..z^(b-1) (the run axis needs z^1, so b >= 2
// there), the top level holds R / b^(nlev-1) + 1 entries.
void set_axis(TabLayout& T, int a, int R, int nlev, bool run_axis) {
  const int nv = R + 1;
  int b = 1;
  if (nlev == 1) {
    b = std::max(nv, run_axis ? 2 : 1);
  } else {
    b = std::max(2, (int)std::floor(std::pow((double)nv, 1.0 / nlev)));
    auto pw = [&](int x) { long long r = 1; for (int l = 0; l < nlev; ++l) r *= x; return r; };
    while (pw(b) < nv) ++b;
  }
  T.nlev[a] = nlev;
  T.base[a] = b;
  long long scale = 1;
  for (int l = 0; l < kMaxLevels; ++l) {
    if (l >= nlev) T.nent[a][l] = 0;
    else if (l == nlev - 1) T.nent[a][l] = (int)(R / scale) + 1;
    else T.nent[a][l] = b;
    if (l == 0 && nlev == 1) T.nent[a][0] = b;
    scale *= b;
  }
}

void assign_rows(TabLayout& T, int d) {
  int row = 0;
  for (int a = 0; a < 3; ++a)
    for (int l = 0; l < kMaxLevels; ++l) {
      T.row[a][l] = row;
      if (a < d && l < T.nlev[a]) row += T.nent[a][l];
    }
  T.nrows = row;
  T.zrow = T.row[d - 1][0] + 1;
}

// Fewest table lookups whose rows fit `max_rows`: start with one level per
// axis (one load per lookup) and add a level to the axis with the most rows
// until the table fits (or every axis has kMaxLevels levels).
TabLayout make_layout(const int* R, int d, int max_rows) {
  TabLayout T{};
  int lev[3] = {1, 1, 1};
  for (;;) {
    for (int a = 0; a < d; ++a) set_axis(T, a, R[a], lev[a], a == d - 1);
    assign_rows(T, d);
    if (T.nrows <= max_rows) break;
    int best = -1, most = 0;
    for (int a = 0; a < d; ++a) {
      int rows = 0;
      for (int l = 0; l < lev[a]; ++l) rows += T.nent[a][l];
      if (lev[a] < kMaxLevels && rows > most) { most = rows; best = a; }
    }
    if (best < 0) break;
    ++lev[best];
  }
  return T;
}

// Folded last-axis range of a run: columns c = |n| from fold_lo to fold_hi.
int fold_lo(const GridRun& g) {
  return (g.a <= 0 && g.b >= 0) ? 0 : std::min(std::abs(g.a), std::abs(g.b));
}
int fold_hi(const GridRun& g) { return std::max(std::abs(g.a), std::abs(g.b)); }

void sort_by_fold(std::vector<GridRun>& runs) {
  std::stable_sort(runs.begin(), runs.end(), [](const GridRun& x, const GridRun& y) {
    return fold_hi(x) - fold_lo(x) > fold_hi(y) - fold_lo(y);
  });
}

// The density class of cco_problem_pass1_form, which is also part of the scratch
// cco_energy_grad_noalloc has always asked for: the (24-run x 16 cq-column) blocks of a
// k-set of d >= 2 whose blocks hold at least half (d = 3: all) as many rows as
// cells, cells counted per 6 runs; 0 for sparser ones and in 1-D.
int folded_blocks(std::vector<GridRun> runs, int d, int m) {
  if (d < 2 || runs.empty()) return 0;
  sort_by_fold(runs);
  double best = 0.0;
  int blocks = 0;
  for (int cols = 16; cols <= 48; cols += 16) {
    double cells = 0.0;
    int nb = 0;
    for (size_t r0 = 0; r0 < runs.size(); r0 += 24) {
      const int nrun = (int)std::min<size_t>(24, runs.size() - r0);
      int lo = 1 << 30, hi = 0;
      for (int r = 0; r < nrun; ++r) {
        lo = std::min(lo, fold_lo(runs[r0 + r]));
        hi = std::max(hi, fold_hi(runs[r0 + r]));
      }
      const int win = (hi - lo) / cols + 1;
      cells += (double)((nrun + 5) / 6 * 6) * cols * win;
      nb += win;
    }
    if (cols == 16 || cells <= best) {
      best = cells;
      blocks = nb;
    }
  }
  return (double)m >= (d == 3 ? 1.0 : 0.5) * best ? blocks : 0;
}

// The grid of a k-set (cco_grid.cuh): runs, strips of 8, blocks, quads.
struct GridPlan {
  std::vector<GridRun> runs;
  std::vector<GridStrip> strips;
  std::vector<GridBlock> blocks;
  std::vector<GridQuad> quads;
  std::vector<GridRow> rows;
  std::vector<GridLine> lines;   // line grids
  std::vector<int2> slotk;
  int entries = 0;   // widest block's table entries
  int tiles = 0;     // most 8 x 8-cell tiles of a block
};

// by_length: strips of runs of the same number of quads (fewest padded cells);
// otherwise in prefix order (narrowest prefix windows: large or skewed sets).
// Either way the inner axis runs back and forth, so that a strip that crosses
// into the next outer value stays at the same end of the inner one.
void grid_layout(std::vector<GridRun> runs, int d, int max_cols, int max_strips, bool by_length,
                 GridPlan* out) {
  *out = GridPlan{};
  std::stable_sort(runs.begin(), runs.end(), [by_length](const GridRun& x, const GridRun& y) {
    const int u = by_length ? fold_hi(x) / 4 : 0, v = by_length ? fold_hi(y) / 4 : 0;
    if (u != v) return u > v;
    if (by_length)
      return x.n1 != y.n1 ? x.n1 < y.n1 : (x.n1 & 1) ? x.n0 > y.n0 : x.n0 < y.n0;
    return x.n0 != y.n0 ? x.n0 < y.n0 : (x.n0 & 1) ? x.n1 > y.n1 : x.n1 < y.n1;
  });
  out->runs = runs;
  const int nr = (int)runs.size(), ns = (nr + 7) / 8;
  const int nbr = (ns + max_strips - 1) / max_strips;   // block rows, of even height
  for (int br = 0; br < nbr; ++br) {
    const int s0 = (int)((long long)ns * br / nbr), s1 = (int)((long long)ns * (br + 1) / nbr);
    int lo = 1 << 30, hi = 0;
    for (int r = 8 * s0; r < std::min(nr, 8 * s1); ++r) {
      lo = std::min(lo, fold_lo(runs[r]));
      hi = std::max(hi, fold_hi(runs[r]));
    }
    const int range = hi - lo + 1, nw = (range + max_cols - 1) / max_cols;
    const int width = ((range + nw - 1) / nw + 7) / 8 * 8;
    std::vector<int> wins;   // first columns of the windows
    if (nw <= 64) {
      for (int w = lo; w <= hi; w += width) wins.push_back(w);
    } else {   // those with columns of a run: far-apart runs leave most of them empty
      for (int r = 8 * s0; r < std::min(nr, 8 * s1); ++r)
        for (int w = (fold_lo(runs[r]) - lo) / width; w <= (fold_hi(runs[r]) - lo) / width; ++w)
          wins.push_back(lo + w * width);
      std::sort(wins.begin(), wins.end());
      wins.erase(std::unique(wins.begin(), wins.end()), wins.end());
    }
    for (const int w : wins) {
      GridBlock b{};
      b.strip0 = (int)out->strips.size();
      b.lo = w;
      b.m0 = b.m1 = 1 << 30;
      int M0 = -(1 << 30), M1 = -(1 << 30);
      for (int s = s0; s < s1; ++s) {
        GridStrip g{};
        g.run0 = 8 * s;
        g.nrun = std::min(8, nr - 8 * s);
        int top = -1;
        for (int r = g.run0; r < g.run0 + g.nrun; ++r)
          if (fold_hi(runs[r]) >= w && fold_lo(runs[r]) < w + width)
            top = std::max(top, std::min(fold_hi(runs[r]) - w, width - 1));
        if (top < 0) continue;
        g.nq = top / 4 + 1;
        g.slot0 = 32 * (int)out->quads.size();
        for (int q = 0; q < g.nq; ++q) out->quads.push_back(GridQuad{g.run0, g.nrun, w + 4 * q, 0});
        out->strips.push_back(g);
        b.nstrip += 1;
        b.ntile += (g.nq + 1) / 2;
        b.ncol = std::max(b.ncol, (g.nq + 1) / 2 * 8);
        for (int r = g.run0; r < g.run0 + g.nrun; ++r) {
          b.m0 = std::min(b.m0, runs[r].n0);
          M0 = std::max(M0, runs[r].n0);
          b.m1 = std::min(b.m1, runs[r].n1);
          M1 = std::max(M1, runs[r].n1);
        }
      }
      if (b.nstrip == 0) continue;
      b.c0 = M0 - b.m0 + 1;
      b.c1 = d == 3 ? M1 - b.m1 + 1 : 0;
      if (d != 3) b.m1 = 0;
      out->entries = std::max(out->entries, b.ncol + b.c0 + b.c1);
      out->tiles = std::max(out->tiles, b.ntile);
      for (int s = b.strip0; s < b.strip0 + b.nstrip; ++s)
        for (int r = 0; r < 8; ++r) {   // rows past the strip's runs repeat its last (weights 0)
          const GridRun& g = runs[out->strips[s].run0 + std::min(r, out->strips[s].nrun - 1)];
          out->rows.push_back(GridRow{b.ncol + g.n0 - b.m0,
                                      d == 3 ? b.ncol + b.c0 + g.n1 - b.m1 : 0, g.n0, g.n1});
        }
      out->blocks.push_back(b);
    }
  }
}

// Runs of a 1-D k-set on columns |c| <= C: n = q (2 C + 1) + c.
std::vector<GridRun> split_runs_1d(const std::vector<GridRun>& runs, int C) {
  const int S = 2 * C + 1;
  auto fdiv = [](int x, int y) { return x >= 0 ? x / y : -((-x + y - 1) / y); };
  std::vector<GridRun> out;
  for (const GridRun& g : runs)
    for (int q = fdiv(g.a + C, S); q <= fdiv(g.b + C, S); ++q) {
      const int a = std::max(g.a, q * S - C), b = std::min(g.b, q * S + C);
      out.push_back(GridRun{q, 0, a - q * S, b - q * S, g.kstart + a - g.a, 0});
    }
  return out;
}

void grid_sizes(ProbDev* P, const GridPlan& gp);

// A line grid: `rows` holds the k-set in run order (M x d). Rows are multiples
// i v of primitive vectors v; a line's multiples are cut into strips of 8 rows
// i = q step + c, |c| < 4 nq, step = 8 nq - 1, with the nq (at most 4) that
// costs least; as many strips share a block as its table holds. Only pass 1
// takes this form (the structure factor's k-set: every multiple up to a large
// cut-off along each of ~600 directions, runs of one row for the recurrences:
// 16 densities of N = 1000 on 96 660 rows 11.3 ms, on lines 0.63 ms; two thirds
// of that is forming tables, three sincospi and 24 products per strip and
// particle against 512 FMAs of a full strip).
void plan_lines(const std::vector<int>& rows, ProbDev* P, GridPlan* gp) {
  const int d = P->d, m = P->M;
  if (d < 2) return;
  std::map<std::array<int, 3>, std::vector<std::pair<int, int>>> lines;   // v -> (i, row)
  for (int k = 0; k < m; ++k) {
    std::array<int, 3> v{0, 0, 0};
    int g = 0, sign = 0;
    for (int a = 0; a < d; ++a) {
      v[a] = rows[(size_t)k * d + a];
      g = std::gcd(g, std::abs(v[a]));
      if (sign == 0) sign = (v[a] > 0) - (v[a] < 0);
    }
    for (int a = 0; a < d; ++a) v[a] /= g * sign;
    lines[v].push_back({g * sign, k});
  }
  if ((long long)lines.size() * 16 > m) return;   // short lines: mostly padding
  struct Strip {
    GridLine line;
    int nq;
    std::vector<int2> k;   // per slot
  };
  std::vector<Strip> strips;
  auto fdiv = [](int x, int y) { return x >= 0 ? x / y : -((-x + y - 1) / y); };
  for (auto& [v, ms] : lines) {
    int lo = ms[0].first, hi = lo;
    for (const auto& e : ms) {
      lo = std::min(lo, e.first);
      hi = std::max(hi, e.first);
    }
    int nq = 1, best = 0;
    for (int t = 1; t <= 4; ++t) {
      const int S = 8 * t - 1, C = 4 * t - 1;
      const int ns = (fdiv(hi + C, S) - fdiv(lo + C, S)) / 8 + 1;
      const int cost = ns * (128 * t + 250);   // DMMA work and tables per particle
      if (t == 1 || cost < best) {
        best = cost;
        nq = t;
      }
    }
    const int S = 8 * nq - 1, C = 4 * nq - 1, q_lo = fdiv(lo + C, S);
    const int ns = (fdiv(hi + C, S) - q_lo) / 8 + 1;
    const size_t first = strips.size();
    for (int s = 0; s < ns; ++s)
      strips.push_back(Strip{GridLine{{v[0], v[1], v[2]}, S, q_lo + 8 * s, (nq + 1) / 2 * 8}, nq,
                             std::vector<int2>(32 * nq, make_int2(-1, -1))});
    for (const auto& [i, k] : ms) {
      const int q = fdiv(i + C, S), c = i - q * S, ac = std::abs(c);
      Strip& T = strips[first + (q - q_lo) / 8];
      const int r = (q - q_lo) % 8, row = r < 4 ? 2 * r : 2 * (r - 4) + 1;   // grid_perm(row) = r
      int2& e = T.k[32 * (ac / 4) + 4 * row + ac % 4];
      (c >= 0 ? e.x : e.y) = k;
    }
  }
  std::stable_sort(strips.begin(), strips.end(),
                   [](const Strip& x, const Strip& y) { return x.nq > y.nq; });
  GridPlan out;
  for (const Strip& T : strips) {
    const int entries = T.line.ncol + 8;
    GridBlock* b = out.blocks.empty() ? nullptr : &out.blocks.back();
    const int used = b ? b->ncol : 0;   // table entries so far
    if (!b || used + entries > kGridMaxEntries || b->nstrip == kGridStrips || b->ntile + (T.nq + 1) / 2 > 4) {
      out.blocks.push_back(GridBlock{});
      b = &out.blocks.back();
      b->strip0 = (int)out.strips.size();
    }
    GridStrip g{};
    g.nrun = 8;
    g.nq = T.nq;
    g.slot0 = (int)out.slotk.size();
    g.col0 = b->ncol;
    for (int r = 0; r < 8; ++r) out.rows.push_back(GridRow{g.col0 + T.line.ncol + r, 0, 0, 0});
    out.strips.push_back(g);
    out.lines.push_back(T.line);
    out.slotk.insert(out.slotk.end(), T.k.begin(), T.k.end());
    b->nstrip += 1;
    b->ntile += (T.nq + 1) / 2;
    b->ncol += entries;
    out.entries = std::max(out.entries, b->ncol);
  }
  if ((long long)out.slotk.size() > 2ll * m) return;
  *gp = out;
  P->grid = 2;
  P->gcls = kGridLines;
  P->gstep = 1;
  P->gslots = (int)out.slotk.size();
  P->grhow = m + (reduce_chunks(P->gslots) + 1) / 2;
  P->gtile = P->N <= 64 ? 64 : P->N <= 128 ? 128 : 256;   // many blocks: few, large tiles
  grid_sizes(P, out);
}

// Tile counts and table stride, and the check that the form fits the fixed
// scratch of cco_energy_grad_noalloc wherever the recurrence form does.
void grid_sizes(ProbDev* P, const GridPlan& gp) {
  P->ngblk = (int)gp.blocks.size();
  P->gts = gp.entries | 1;
  P->gntile = (P->N + P->gtile - 1) / P->gtile;
  const size_t seg = 2 * (size_t)P->M + (size_t)P->ntile1 * P->M;
  const size_t own = (size_t)P->M + P->grhow + 2 * (size_t)P->gntile * P->gslots + eval_roots_words(*P);
  if (sizeof(double2) * own > CCO_NOALLOC_SCRATCH_BYTES - 65536 &&
      sizeof(double2) * seg <= CCO_NOALLOC_SCRATCH_BYTES)
    P->grid = P->groots = 0;
}

// Whether and how FP64 lanes of a problem run the grid form. The form costs 12
// FMAs per grid cell and particle (4 density, 8 gradient) plus the tables,
// where the recurrences need 14 or more instructions per k-set row: it is taken
// when the slots (cells with their padding) are at most twice the rows.
void plan_grid(const std::vector<GridRun>& runs, ProbDev* P, GridPlan* gp) {
  // every strip of 8 runs takes a quad (32 slots) or more: sets of short runs are
  // refused before a layout is made (90 000 runs of about one row: 11 layouts took 290 ms)
  if (runs.empty() || 32ll * (long long)((runs.size() + 7) / 8) > 2ll * P->M) return;
  // the layout that costs least per particle: products and table entries (both
  // passes), among block shapes whose tables fit
  int step = 1;
  double best = -1.0;
  auto consider = [&](const std::vector<GridRun>& r, int cols, int strips, bool by_length, int st) {
    GridPlan g;
    grid_layout(r, P->d, cols, strips, by_length, &g);
    double cost = (P->d == 1 ? 8.0 : 12.0) * 32.0 * (double)g.quads.size();
    for (const GridBlock& b : g.blocks) cost += 16.0 * (b.ncol + b.c0 + b.c1);
    if (g.entries > kGridMaxEntries || g.tiles > kGridMaxTiles || (best >= 0.0 && cost >= best)) return;
    best = cost;
    step = st;
    *gp = g;
  };
  if (P->d == 1) {
    for (const int nc : {4, 8, 12, 16, 24, 32})
      consider(split_runs_1d(runs, nc - 1), nc, std::min(kGridStrips, (kGridMaxEntries - nc) / 8),
               true, 2 * nc - 1);
  } else {
    static const int shapes[][2] = {{32, 2}, {24, 3}, {24, 4}, {16, 4}, {24, 2}, {16, 2}, {16, 1}, {8, 1}};
    for (int i = 0; i < 4; ++i) consider(runs, shapes[i][0], shapes[i][1], true, 1);
    for (int i = 1; i < 8; ++i) consider(runs, shapes[i][0], shapes[i][1], false, 1);
  }
  if (best < 0.0) return;
  const long long slots = 32ll * (long long)gp->quads.size();
  if (slots > 2ll * P->M) return;
  P->grid = 1;
  P->ngblk = (int)gp->blocks.size();
  P->gcls = gp->tiles > 8 ? 2 : P->ngblk >= kGridRootsMin ? 1 : 0;
  P->gstep = step;
  P->gslots = (int)slots;
  // larger pass-1 tiles for larger N keep the partials (32 bytes per slot and
  // tile) and the reduction small once there are enough tiles to fill the GPU
  P->gtile = P->N <= 512 ? 64 : P->N <= 8192 ? 128 : 256;
  P->grhow = (int)slots * (P->d == 1 ? 2 : 4) + (reduce_chunks((int)slots) + 1) / 2;
  // seeds per virtual axis: multiples of 16 up to the largest |exponent| used
  // (the columns of a block's last tile included)
  int top[3] = {0, 0, 0};
  for (const GridBlock& b : gp->blocks) {
    top[0] = std::max({top[0], -b.m0 + 15, b.m0 + b.c0 - 1});
    if (P->d == 3) top[1] = std::max({top[1], -b.m1 + 15, b.m1 + b.c1 - 1});
    top[2] = std::max(top[2], b.lo + b.ncol - 1);
  }
  P->groff[0] = 0;
  P->groff[1] = 1 + top[0] / 16;
  P->groff[2] = P->groff[1] + (P->d == 3 ? 1 + top[1] / 16 : 0);
  P->groots = P->gcls > 0 ? P->groff[2] + 1 + top[2] / 16 : 0;
  grid_sizes(P, *gp);
}

// Arrays gathered into one upload, each at a 256-byte offset.
struct Blob {
  std::vector<unsigned char> bytes;
  template <class T>
  size_t add(const std::vector<T>& v) {
    const size_t o = (bytes.size() + 255) & ~(size_t)255, n = v.size() * sizeof(T);
    bytes.resize(o + std::max<size_t>(n, 1));
    if (n) memcpy(bytes.data() + o, v.data(), n);
    return o;
  }
};

// Absolute table rows of the digits of v on axis a (+ sign bit 24).
int pack_rows(int v, const TabLayout& T, int a) {
  const int neg = v < 0;
  int x = v < 0 ? -v : v;
  int out = 0;
  for (int l = 0; l < T.nlev[a]; ++l) {
    int dl;
    if (l == T.nlev[a] - 1) dl = x;
    else {
      dl = x % T.base[a];
      x /= T.base[a];
    }
    out |= ((T.row[a][l] + dl) & 255) << (8 * l);
  }
  return out | (neg << 24);
}

}  // namespace

extern "C" {

int cco_abi_version(void) { return CCO_ABI_VERSION; }

const char* cco_error_string(int code) {
  switch (code) {
    case CCO_OK: return "ok";
    case CCO_ERR_ARG: return "invalid argument";
    case CCO_ERR_OOM: return "out of device memory";
    case CCO_ERR_ADMISSION: return "refused by the HBM admission budget";
    case CCO_ERR_DEVICE: return "CUDA error";
    case CCO_ERR_TIMEOUT: return "timed out";
    case CCO_ERR_ROUNDS: return "relax did not finish within the round bound";
    case CCO_ERR_NODEVICE: return "no CUDA device";
    default: return "unknown error";
  }
}

const char* cco_last_error(void) { return g_last_error.c_str(); }

int cco_device_count(int* n_devices) {
  if (!n_devices) return fail(CCO_ERR_ARG, "n_devices is null");
  int n = 0;
  cudaError_t e = cudaGetDeviceCount(&n);
  if (e != cudaSuccess || n == 0) {
    *n_devices = 0;
    cudaGetLastError();
    return fail(CCO_ERR_NODEVICE, "no CUDA device visible (%s)",
                e == cudaSuccess ? "count 0" : cudaGetErrorString(e));
  }
  *n_devices = n;
  return CCO_OK;
}

int cco_problem_create(int device, int d, int n_particles, int m, const int32_t* n_vectors,
                       const double* weights, double volume, cco_problem** out) {
  return cco_problem_create_rows(device, d, n_particles, m, n_vectors, weights, volume, m, nullptr,
                                 out);
}

int cco_problem_create_rows(int device, int d, int n_particles, int m, const int32_t* n_vectors,
                            const double* weights, double volume, int total, const int32_t* rows,
                            cco_problem** out) {
  if (!out) return fail(CCO_ERR_ARG, "out is null");
  *out = nullptr;
  if (d < 1 || d > 3) return fail(CCO_ERR_ARG, "d must be 1, 2 or 3, got %d", d);
  if (n_particles < 1) return fail(CCO_ERR_ARG, "n_particles must be >= 1");
  if (m < 1) return fail(CCO_ERR_ARG, "empty k-set: no k-vectors in the shell");
  if (!n_vectors || !weights) return fail(CCO_ERR_ARG, "null k-set arrays");
  if (!(volume > 0.0) || !std::isfinite(volume)) return fail(CCO_ERR_ARG, "volume must be finite and > 0");
  if (total < m) return fail(CCO_ERR_ARG, "total %d below the %d rows", total, m);
  std::vector<int> row_of(total, -1);   // padded column -> row, then run-order row
  for (int k = 0; k < m; ++k) {
    const int c = rows ? rows[k] : k;
    if (c < 0 || c >= total || row_of[c] >= 0)
      return fail(CCO_ERR_ARG, "row %d: column %d is out of range or taken", k, c);
    row_of[c] = k;
  }
  int ndev = 0;
  if (cco_device_count(&ndev) != CCO_OK) return CCO_ERR_NODEVICE;
  if (device < 0 || device >= ndev) return fail(CCO_ERR_ARG, "device %d out of range", device);

  // validate rows
  std::vector<int> R(3, 0);
  for (int k = 0; k < m; ++k) {
    bool nz = false;
    for (int a = 0; a < d; ++a) {
      const int v = n_vectors[(size_t)k * d + a];
      if (v < -65535 || v > 65535) return fail(CCO_ERR_ARG, "|n| too large at row %d", k);
      R[a] = std::max(R[a], std::abs(v));
      nz |= v != 0;
    }
    if (!nz) return fail(CCO_ERR_ARG, "row %d is the zero vector (padding rows are handled by the caller)", k);
    if (!std::isfinite(weights[k])) return fail(CCO_ERR_ARG, "non-finite weight at row %d", k);
  }
  // run order: prefix lexicographic, then the last axis ascending
  std::vector<int> order(m);
  for (int k = 0; k < m; ++k) order[k] = k;
  std::stable_sort(order.begin(), order.end(), [&](int x, int y) {
    for (int a = 0; a < d; ++a) {
      const int u = n_vectors[(size_t)x * d + a], v = n_vectors[(size_t)y * d + a];
      if (u != v) return u < v;
    }
    return false;
  });
  for (int k = 1; k < m; ++k) {
    bool same = true;
    for (int a = 0; a < d; ++a)
      same &= n_vectors[(size_t)order[k] * d + a] == n_vectors[(size_t)order[k - 1] * d + a];
    if (same) return fail(CCO_ERR_ARG, "duplicate k row (rows %d and %d)", order[k - 1], order[k]);
  }
  ProbDev P{};
  P.d = d;
  P.N = n_particles;
  P.M = m;
  for (int a = 0; a < 3; ++a) P.rmax[a] = R[a];
  P.compact = compact_smem(P) > kPersistMaxSmem                              ? 0
              : compact_smem(P) + compact_phase_smem(P) > kPersistMaxSmem ? 1
                                                                          : 2;
  {
    const int Rv[3] = {R[0], R[1], R[2]};
    P.t1 = make_layout(Rv, d, (int)(kPass1TableBudget / (kPass1Stride * sizeof(double2))));
    P.t2 = make_layout(Rv, d, (int)(kPass2TableBudget / (kPass2Tile * sizeof(double2))));
  }
  if (P.t1.nrows > 255 || P.t2.nrows > 255)
    return fail(CCO_ERR_ARG, "k-set phase tables too large (%d / %d rows)", P.t1.nrows, P.t2.nrows);
  P.ntile1 = (n_particles + kPass1Tile - 1) / kPass1Tile;
  P.ntile2 = (n_particles + kPass2Tile - 1) / kPass2Tile;
  P.vol = volume;
  P.gpref = (2.0 * (2.0 * M_PI)) / volume;

  // runs -> segments (headers carry each pass's absolute table rows)
  std::vector<SegHdr> s1, s2;
  std::vector<GridRun> runs;
  auto emit = [&](std::vector<SegHdr>& dst, const TabLayout& T, int kstart, int len, int maxlen) {
    for (int off = 0; off < len; off += maxlen) {
      SegHdr h{};
      h.kstart = kstart + off;
      h.len = std::min(maxlen, len - off);
      const int* nv = n_vectors + (size_t)order[h.kstart] * d;
      for (int a = 0; a < d; ++a) {
        h.n[a] = nv[a];
        h.dig[a] = pack_rows(nv[a], T, a);
      }
      dst.push_back(h);
    }
  };
  int start = 0;
  for (int k = 1; k <= m; ++k) {
    bool brk = (k == m);
    if (!brk) {
      const int* p = n_vectors + (size_t)order[k - 1] * d;
      const int* c = n_vectors + (size_t)order[k] * d;
      for (int a = 0; a < d - 1; ++a) brk |= p[a] != c[a];
      brk |= c[d - 1] != p[d - 1] + 1;
    }
    if (brk) {
      emit(s1, P.t1, start, k - start, kSeg1Len);
      emit(s2, P.t2, start, k - start, kSeg2Len);
      const int* nv = n_vectors + (size_t)order[start] * d;
      GridRun g{};
      g.n0 = d >= 2 ? nv[0] : 0;
      g.n1 = d >= 3 ? nv[1] : 0;
      g.a = nv[d - 1];
      g.b = nv[d - 1] + (k - start) - 1;
      g.kstart = start;
      runs.push_back(g);
      start = k;
    }
  }
  GridPlan gp;
  const char* env = getenv("CCO_PASS1_GEMM");   // 0: the per-segment form everywhere
  const bool allow = !(env && atoi(env) == 0);
  const int dense_blocks = allow ? folded_blocks(runs, d, m) : 0;
  if (allow) plan_grid(runs, &P, &gp);
  if (allow && !P.grid) {
    std::vector<int> rows((size_t)m * d);
    for (int k = 0; k < m; ++k)
      for (int a = 0; a < d; ++a) rows[(size_t)k * d + a] = n_vectors[(size_t)order[k] * d + a];
    plan_lines(rows, &P, &gp);
  }
  if (!P.grid) gp = GridPlan{};   // nothing to upload of a refused layout
  // longest segments first: pass-1 warps share trip counts, pass 2 pairs
  // segments of similar length
  auto by_len = [](const SegHdr& x, const SegHdr& y) { return x.len > y.len; };
  std::stable_sort(s1.begin(), s1.end(), by_len);
  std::stable_sort(s2.begin(), s2.end(), by_len);
  P.nseg1 = (int)s1.size();
  P.nseg2 = (int)s2.size();
  {
    // logical pass-2 slices: at least one segment pair each, at most 8 (a
    // launch of few lanes spreads a particle's slices over up to 8 threads)
    const int npairs = (P.nseg2 + 1) / 2;
    int sl = 1;
    while (sl < 8 && 2 * sl <= npairs) sl *= 2;
    P.sl2 = sl;
  }

  const size_t smem1 = eval_smem1(P);
  const size_t smem2 = std::max(std::max(eval_smem2(P, 1), eval_smem2(P, 8)),
                                std::max(eval_smem2(P, 1, true), eval_smem2(P, 8, true)));
  if (smem1 > 220 * 1024 || smem2 > 220 * 1024)
    return fail(CCO_ERR_ARG, "k-set phase tables too large for shared memory (%d / %d rows)",
                P.t1.nrows, P.t2.nrows);

  DeviceGuard guard(device);
  const cudaError_t cfg_err = eval_configure();
  if (cfg_err != cudaSuccess) return cuda_fail(cfg_err, "eval_configure");

  auto* pr = new cco_problem();
  pr->device = device;
  pr->d = d;
  pr->N = n_particles;
  pr->M = m;
  std::vector<double> w_run(m);
  std::vector<int> r2r(m);
  std::vector<double4> krow(m);
  for (int k = 0; k < m; ++k) {
    w_run[k] = weights[order[k]];
    r2r[k] = order[k];
    const int32_t* nv = n_vectors + (size_t)order[k] * d;
    krow[k] = make_double4(nv[0], d > 1 ? nv[1] : 0, d > 2 ? nv[2] : 0, w_run[k]);
  }
  std::vector<int> run_of(m);
  for (int k = 0; k < m; ++k) run_of[order[k]] = k;
  for (int& c : row_of)
    if (c >= 0) c = run_of[c];
  pr->run2ref = r2r;
  pr->total = total;
  // one device block for everything the problem uploads
  Blob blob;
  const size_t o_seg1 = blob.add(s1), o_seg2 = blob.add(s2), o_w = blob.add(w_run),
               o_r2r = blob.add(r2r), o_krow = blob.add(krow), o_row = blob.add(row_of),
               o_grun = blob.add(gp.runs), o_gblk = blob.add(gp.blocks),
               o_gstrip = blob.add(gp.strips), o_gquad = blob.add(gp.quads),
               o_grow = blob.add(gp.rows), o_gline = blob.add(gp.lines),
               o_gslotk = blob.add(gp.slotk);
  const size_t o_dev = blob.add(std::vector<ProbDev>(1));
  cudaError_t e = cudaMalloc(&pr->block, blob.bytes.size());
  auto at = [&](size_t o) { return static_cast<void*>(pr->block + o); };
  if (e == cudaSuccess) {
    P.seg1 = static_cast<SegHdr*>(at(o_seg1));
    P.seg2 = static_cast<SegHdr*>(at(o_seg2));
    P.w_run = static_cast<double*>(at(o_w));
    P.run2ref = static_cast<int*>(at(o_r2r));
    P.grun = static_cast<GridRun*>(at(o_grun));
    P.gblk = static_cast<GridBlock*>(at(o_gblk));
    P.gstrip = static_cast<GridStrip*>(at(o_gstrip));
    P.gquad = static_cast<GridQuad*>(at(o_gquad));
    P.grow = static_cast<GridRow*>(at(o_grow));
    P.gline = static_cast<GridLine*>(at(o_gline));
    P.gslotk = static_cast<int2*>(at(o_gslotk));
    pr->krow = static_cast<double4*>(at(o_krow));
    P.krow = pr->krow;
    pr->row_of = static_cast<int*>(at(o_row));
    pr->dev = static_cast<ProbDev*>(at(o_dev));
    memcpy(blob.bytes.data() + o_dev, &P, sizeof(ProbDev));
    e = cudaMemcpy(pr->block, blob.bytes.data(), blob.bytes.size(), cudaMemcpyHostToDevice);
  }
  pr->host = P;
  pr->smem1 = smem1;
  pr->smem2 = smem2;
  pr->smemG = eval_smemG(P);
  pr->smemH = eval_smemH(P);
  pr->dense_blocks = dense_blocks;
  if (e != cudaSuccess) {
    cco_problem_destroy(pr);
    return cuda_fail(e, "cco_problem_create upload");
  }
  *out = pr;
  return CCO_OK;
}

int cco_problem_destroy(cco_problem* p) {
  if (!p) return CCO_OK;
  DeviceGuard guard(p->device);
  cudaFree(p->block);
  delete p;
  return CCO_OK;
}

int cco_problem_info(const cco_problem* p, int* d, int* n_particles, int* m, int* n_seg1,
                     int* n_seg2, int* table_rows) {
  if (!p) return fail(CCO_ERR_ARG, "null problem");
  if (d) *d = p->d;
  if (n_particles) *n_particles = p->N;
  if (m) *m = p->M;
  if (n_seg1) *n_seg1 = p->host.nseg1;
  if (n_seg2) *n_seg2 = p->host.nseg2;
  if (table_rows) *table_rows = p->host.t1.nrows * 256 + p->host.t2.nrows;
  return CCO_OK;
}

int cco_problem_pass1_form(const cco_problem* p, int* gemm_blocks) {
  if (!p || !gemm_blocks) return fail(CCO_ERR_ARG, "null argument");
  *gemm_blocks = p->host.grid == 1 ? p->dense_blocks : 0;
  return CCO_OK;
}

}  // extern "C"

// ------------------------------------------------------------ eval workspace
namespace {

__global__ void k_make_lanes(EvalLane* lanes, EvalItem* it1, EvalItem* it2, int B, int nt1,
                             int nt2, int total, const double* s, size_t s_stride, double* f,
                             size_t f_stride, double* g, size_t g_stride, double2* rho,
                             double2* rhow, double2* part, double2* roots, int M,
                             size_t rhow_stride, size_t part_stride, size_t roots_stride,
                             int prec) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    if (i < B) {
      EvalLane L;
      L.s = s + (size_t)i * s_stride;
      L.f = f + (size_t)i * f_stride;
      L.g = g ? g + (size_t)i * g_stride : nullptr;
      L.rho = rho + (size_t)i * M;
      L.rhow = rhow + (size_t)i * rhow_stride;
      L.part = part + (size_t)i * part_stride;
      L.roots = roots + (size_t)i * roots_stride;
      L.status = nullptr;
      L.prec = nullptr;
      L.fixed_prec = prec;
      L.prob = 0;
      lanes[i] = L;
    }
    const int j = i - B;
    if (j >= 0) {
      if (j < B * nt1) it1[j] = EvalItem{j / nt1, j % nt1};
      if (j < B * nt2) it2[j] = EvalItem{j / nt2, j % nt2};
    }
  }
}

size_t round256(size_t b) { return (b + 255) & ~(size_t)255; }

// Device buffers of one batched evaluation: densities, partials and the plan.
// One problem and one arithmetic, so every lane takes the same form: it1 and
// it2 hold the items of that form's two passes.
struct EvalWS {
  EvalLane* lanes = nullptr;
  EvalItem* it1 = nullptr;
  EvalItem* it2 = nullptr;
  double2* rho = nullptr;
  double2* rhow = nullptr;
  double2* part = nullptr;
  double2* roots = nullptr;
  unsigned char* block = nullptr;   // the allocation that holds them (null: the caller's memory)
  EvalPlan plan{};
  int prec = PREC_FP64;   // arithmetic of every lane of this workspace
  int cap = 0, split = 1;   // lanes that fit, pass-2 threads per particle: of the carve

  // Element counts of one lane.
  struct Sizes {
    bool grid, grid2;   // the grid form in pass 1, in pass 2
    int nt1, nt2;
    size_t rhow, part, roots;   // double2 words
  };
  static Sizes sizes(const cco_problem* p, int prec, int split) {
    Sizes z;
    const ProbDev& h = p->host;
    z.grid = h.grid && prec == PREC_FP64;
    z.nt1 = z.grid ? h.gntile * h.ngblk : h.ntile1;
    z.grid2 = z.grid && h.grid == 1;
    z.nt2 = z.grid2 ? (h.N + kGridTile2 - 1) / kGridTile2 : pass2_tiles(h, split);
    z.rhow = z.grid ? (size_t)h.grhow : (size_t)h.M;
    z.part = z.grid ? 2 * (size_t)h.gntile * h.gslots : (size_t)h.ntile1 * h.M;
    z.roots = z.grid ? eval_roots_words(h) : 0;
    return z;
  }
  // Byte offsets of the buffers of up to B lanes in one block of memory. The
  // pass-2 split is part of it: fewer lanes would choose a larger one, and with
  // it more items than the block has room for.
  struct Carve {
    int lanes, split;
    size_t it1, it2, rho, rhow, part, roots, total;
  };
  static Carve carve(const cco_problem* p, int B, int prec) {
    Carve c;
    c.lanes = B;
    c.split = pass2_split((long long)B * p->host.ntile2);
    const Sizes z = sizes(p, prec, c.split);
    c.it1 = round256(sizeof(EvalLane) * B);
    c.it2 = c.it1 + round256(sizeof(EvalItem) * (size_t)B * z.nt1);
    c.rho = c.it2 + round256(sizeof(EvalItem) * (size_t)B * z.nt2);
    c.rhow = c.rho + round256(sizeof(double2) * (size_t)B * p->M);
    c.part = c.rhow + round256(sizeof(double2) * (size_t)B * z.rhow);
    c.roots = c.part + round256(sizeof(double2) * (size_t)B * z.part);
    c.total = c.roots + round256(sizeof(double2) * (size_t)B * z.roots);
    return c;
  }
  void place(unsigned char* base, const Carve& c) {
    cap = c.lanes;
    split = c.split;
    lanes = reinterpret_cast<EvalLane*>(base);
    it1 = reinterpret_cast<EvalItem*>(base + c.it1);
    it2 = reinterpret_cast<EvalItem*>(base + c.it2);
    rho = reinterpret_cast<double2*>(base + c.rho);
    rhow = reinterpret_cast<double2*>(base + c.rhow);
    part = reinterpret_cast<double2*>(base + c.part);
    roots = reinterpret_cast<double2*>(base + c.roots);
  }
  // one stream-ordered allocation per evaluation (six and their frees took a
  // third of a small call's host time), `extra` bytes of the caller's in front
  cudaError_t alloc(const cco_problem* p, int B, cudaStream_t st, size_t extra = 0) {
    const Carve c = carve(p, B, prec);
    const size_t front = round256(extra);
    const cudaError_t e = pool_alloc(&block, front + c.total, st);
    if (e == cudaSuccess) place(block + front, c);
    return e;
  }
  cudaError_t build(const cco_problem* p, int B, const double* s, size_t s_stride, double* f,
                    size_t f_stride, double* g, size_t g_stride, cudaStream_t st) {
    if (B > cap) return cudaErrorInvalidValue;
    const Sizes z = sizes(p, prec, split);
    const int total = B * std::max(z.nt1, z.nt2) + B;
    const int blocks = std::min(1024, (total + 255) / 256);
    k_make_lanes<<<blocks, 256, 0, st>>>(lanes, it1, it2, B, z.nt1, z.nt2, total, s, s_stride, f,
                                         f_stride, g, g_stride, rho, rhow, part, roots, p->M,
                                         z.rhow, z.part, z.roots, prec);
    plan.probs = p->dev;
    plan.lanes = lanes;
    plan.items1 = plan.itemsG = it1;
    plan.items2 = plan.itemsH = it2;
    plan.n_lanes = B;
    plan.chain = true;
    plan.n_items1 = z.grid ? 0 : B * z.nt1;
    plan.n_items2 = z.grid2 ? 0 : B * z.nt2;
    const int nG = z.grid ? B * z.nt1 : 0, nH = z.grid2 ? B * z.nt2 : 0;
    for (int D = 0; D <= 3; ++D) {
      plan.d_off1[D] = D >= p->d ? plan.n_items1 : 0;
      plan.d_off2[D] = D >= p->d ? plan.n_items2 : 0;
    }
    // one problem: its items are all of its column class
    for (int D = 1; D <= 3; ++D)
      for (int c = 0; c <= kGridClasses; ++c)
        plan.q_offG[D - 1][c] = (D == p->d && c > p->host.gcls) ? nG : 0;
    for (int D = 1; D <= 3; ++D)
      for (int c = 0; c <= 2; ++c)
        plan.h_off[D - 1][c] = (D == p->d && c > (p->host.gcls > 0)) ? nH : 0;
    plan.smemG = p->smemG;
    plan.smemH = p->smemH;
    plan.n_grid = z.roots > 0 ? B : 0;
    plan.root_chunks = (int)((z.roots + kRootChunk - 1) / kRootChunk);
    plan.dyn_prec = prec == PREC_FP32 ? 1 : 0;
    plan.max_d = p->d;
    plan.smem1 = p->smem1;
    plan.smem2 = eval_smem2(p->host, split);
    plan.smem2_f32 = eval_smem2(p->host, split, true);
    plan.split2 = split;
    plan.chunks1 = 1;
    plan.red_chunks = reduce_chunks(z.grid ? p->host.gslots : p->M);
    plan.want_grad = g != nullptr;
    return cudaGetLastError();
  }
  void release(cudaStream_t st) {
    if (block) cudaFreeAsync(block, st);
    block = nullptr;
  }
};

}  // namespace

namespace {

// One batched evaluation; `after` gets the run-order densities on the stream.
template <class After>
int evaluate_batch(cco_problem* p, void* stream, int batch, const double* s, double* phi,
                   double* grad, After after) {
  DeviceGuard guard(p->device);
  cudaStream_t st = (cudaStream_t)stream;
  EvalWS ws;
  CCO_CUDA(ws.alloc(p, batch, st, phi ? 0 : sizeof(double) * batch));
  const size_t nd = (size_t)p->N * p->d;
  cudaError_t e = ws.build(p, batch, s, nd, phi ? phi : reinterpret_cast<double*>(ws.block), 1, grad,
                           nd, st);
  if (e == cudaSuccess) e = eval_launch(ws.plan, st);
  if (e == cudaSuccess) e = after(ws.rho, st);
  ws.release(st);
  CCO_CUDA(e);
  CCO_CUDA(cudaGetLastError());
  return CCO_OK;
}

}  // namespace

extern "C" int cco_energy_grad(cco_problem* p, void* stream, int batch, const double* s,
                               double* phi, double* grad, double* rho_re, double* rho_im) {
  if (!p) return fail(CCO_ERR_ARG, "null problem");
  if (batch < 0) return fail(CCO_ERR_ARG, "batch must be >= 0");
  if (batch == 0) return CCO_OK;
  if (!s || !phi) return fail(CCO_ERR_ARG, "null s or phi");
  return evaluate_batch(p, stream, batch, s, phi, grad, [&](const double2* rho, cudaStream_t st) {
    if (!rho_re && !rho_im) return cudaSuccess;
    return rho_scatter(rho, p->host.run2ref, p->M, batch, p->M, rho_re, rho_im, st);
  });
}

extern "C" int cco_energy_grad_rows(cco_problem* p, void* stream, int batch, const double* s,
                                    double* phi, double* grad, double* rho_re, double* rho_im) {
  if (!p) return fail(CCO_ERR_ARG, "null problem");
  if (batch < 0) return fail(CCO_ERR_ARG, "batch must be >= 0");
  if (batch == 0) return CCO_OK;
  if (!s || !phi) return fail(CCO_ERR_ARG, "null s or phi");
  return evaluate_batch(p, stream, batch, s, phi, grad, [&](const double2* rho, cudaStream_t st) {
    if (!rho_re && !rho_im) return cudaSuccess;
    return rho_rows(rho, p->row_of, p->total, p->M, p->N, batch, rho_re, rho_im, st);
  });
}

extern "C" int cco_structure_sums(cco_problem* p, void* stream, int batch, const double* s,
                                  double* tot, double* tot2) {
  if (!p) return fail(CCO_ERR_ARG, "null problem");
  if (batch < 0) return fail(CCO_ERR_ARG, "batch must be >= 0");
  if (batch == 0) return CCO_OK;
  if (!s || !tot || !tot2) return fail(CCO_ERR_ARG, "null argument");
  return evaluate_batch(p, stream, batch, s, nullptr, nullptr, [&](const double2* rho, cudaStream_t st) {
    return structure_sums(rho, p->host.run2ref, p->M, p->N, batch, tot, tot2, st);
  });
}

extern "C" int cco_energy_grad_fp32(cco_problem* p, void* stream, int batch, const double* s,
                                    double* phi, double* grad) {
  if (!p) return fail(CCO_ERR_ARG, "null problem");
  if (batch < 0) return fail(CCO_ERR_ARG, "batch must be >= 0");
  if (batch == 0) return CCO_OK;
  if (!s || !phi) return fail(CCO_ERR_ARG, "null s or phi");
  DeviceGuard guard(p->device);
  cudaStream_t st = (cudaStream_t)stream;
  EvalWS ws;
  ws.prec = PREC_FP32;
  CCO_CUDA(ws.alloc(p, batch, st));
  const size_t nd = (size_t)p->N * p->d;
  CCO_CUDA(ws.build(p, batch, s, nd, phi, 1, grad, nd, st));
  CCO_CUDA(eval_launch(ws.plan, st));
  ws.release(st);
  CCO_CUDA(cudaGetLastError());
  return CCO_OK;
}

extern "C" int cco_hessian(cco_problem* p, void* stream, int batch, const double* s,
                           double* hess) {
  if (!p) return fail(CCO_ERR_ARG, "null problem");
  if (batch < 0) return fail(CCO_ERR_ARG, "batch must be >= 0");
  if (batch == 0) return CCO_OK;
  if (!s || !hess) return fail(CCO_ERR_ARG, "null s or hess");
  if (batch > 65535) return fail(CCO_ERR_ARG, "batch %d > 65535: split it", batch);
  DeviceGuard guard(p->device);
  cudaStream_t st = (cudaStream_t)stream;
  EvalWS ws;
  CCO_CUDA(ws.alloc(p, batch, st, sizeof(double) * batch));
  double* phi = reinterpret_cast<double*>(ws.block);
  const size_t nd = (size_t)p->N * p->d;
  CCO_CUDA(ws.build(p, batch, s, nd, phi, 1, nullptr, 0, st));
  CCO_CUDA(eval_launch(ws.plan, st));   // the density the diagonal blocks need
  CCO_CUDA(hessian_launch(p, st, batch, s, ws.rho, hess));
  ws.release(st);
  CCO_CUDA(cudaGetLastError());
  return CCO_OK;
}

// ------------------------------------------------- evaluation without allocation
namespace {

// Scratch of cco_energy_grad_noalloc: one fixed device array in the library,
// resident on every GPU that loads it until the process exits. Host code must
// never pass this name to a kernel: on the host it is only a stand-in for the
// symbol; the device address is resolved per device below.
static __device__ __align__(256) unsigned char g_noalloc_scratch[CCO_NOALLOC_SCRATCH_BYTES];

constexpr int kNoallocMaxDevices = 64;
std::mutex g_noalloc_mu;
void* g_noalloc_addr[kNoallocMaxDevices] = {};

// Device address of the scratch on `device`, resolved on the first call with
// that device current (the caller holds a DeviceGuard for it).
int noalloc_scratch(int device, unsigned char** out) {
  if (device < 0 || device >= kNoallocMaxDevices)
    return fail(CCO_ERR_ARG, "device %d out of range for the fixed scratch", device);
  std::lock_guard<std::mutex> lk(g_noalloc_mu);
  if (g_noalloc_addr[device] == nullptr) {
    void* addr = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&addr, g_noalloc_scratch);
    if (e != cudaSuccess) return cuda_fail(e, "cudaGetSymbolAddress(fixed scratch)");
    g_noalloc_addr[device] = addr;
  }
  *out = static_cast<unsigned char*>(g_noalloc_addr[device]);
  return CCO_OK;
}

}  // namespace

extern "C" int cco_energy_grad_noalloc(cco_problem* p, void* stream, int batch, const double* s,
                                       double* phi, double* grad) {
  if (!p) return fail(CCO_ERR_ARG, "null problem");
  if (batch < 0) return fail(CCO_ERR_ARG, "batch must be >= 0");
  if (batch == 0) return CCO_OK;
  if (!s || !phi) return fail(CCO_ERR_ARG, "null s or phi");
  // The scratch a call may ask for: rho, w rho and the per-segment partials of
  // the batch plus its items. The grid form's layout of the same data can be
  // larger (padded cells), so such a batch runs in parts that fit; its lanes
  // do not depend on one another.
  const size_t M = (size_t)p->M;
  {
    const size_t B = (size_t)batch, nt1 = (size_t)p->host.ntile1;
    const size_t nt2 = (size_t)pass2_tiles(p->host, pass2_split((long long)batch * p->host.ntile2));
    const size_t gemm = (size_t)p->dense_blocks * nt1;
    const size_t need = round256(sizeof(EvalLane) * B) + round256(sizeof(EvalItem) * B * nt1) +
                        round256(sizeof(EvalItem) * B * nt2) + 2 * round256(sizeof(double2) * B * M) +
                        round256(sizeof(double2) * B * nt1 * M) + round256(sizeof(EvalItem) * B * gemm);
    if (need > CCO_NOALLOC_SCRATCH_BYTES)
      return fail(CCO_ERR_ARG,
                  "batch %d needs %zu bytes of fixed scratch, the limit is %zu: split the batch",
                  batch, need, (size_t)CCO_NOALLOC_SCRATCH_BYTES);
  }
  DeviceGuard guard(p->device);
  unsigned char* base = nullptr;
  const int rc = noalloc_scratch(p->device, &base);
  if (rc != CCO_OK) return rc;
  cudaStream_t st = (cudaStream_t)stream;
  const size_t nd = (size_t)p->N * p->d;
  int part_b = batch;
  while (part_b > 1 && EvalWS::carve(p, part_b, PREC_FP64).total > CCO_NOALLOC_SCRATCH_BYTES)
    part_b = (part_b + 1) / 2;
  const EvalWS::Carve c = EvalWS::carve(p, part_b, PREC_FP64);
  if (c.total > CCO_NOALLOC_SCRATCH_BYTES)
    return fail(CCO_ERR_ARG, "one configuration needs %zu bytes of fixed scratch, the limit is %zu",
                c.total, (size_t)CCO_NOALLOC_SCRATCH_BYTES);
  for (int lo = 0; lo < batch; lo += part_b) {
    const int b = std::min(part_b, batch - lo);
    EvalWS ws;  // carved from the fixed scratch; never released
    ws.place(base, c);
    CCO_CUDA(ws.build(p, b, s + (size_t)lo * nd, nd, phi + lo, 1,
                      grad ? grad + (size_t)lo * nd : nullptr, nd, st));
    CCO_CUDA(eval_launch(ws.plan, st));
  }
  return CCO_OK;
}
