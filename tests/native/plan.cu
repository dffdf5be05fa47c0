// Planning of the tensor-core grid of a k-set, on the CPU: every row of the set in
// exactly one slot, in the place its phase is formed for, and the time planning
// takes next to sorting the set's rows once (which a problem's creation does anyway).
#include <chrono>
#include <cstdio>
#include <numeric>
#include <set>

#include "cco_api.cu"

namespace {

using Row = std::array<int, 3>;

double now() {
  return std::chrono::duration<double>(std::chrono::steady_clock::now().time_since_epoch()).count();
}

std::vector<GridRun> runs_of(const std::vector<Row>& rows, int d) {
  std::vector<GridRun> runs;
  for (size_t k = 0; k < rows.size(); ++k) {
    const Row& n = rows[k];
    bool next = k > 0;
    if (next) {
      Row want = rows[k - 1];
      want[d - 1] += 1;
      next = n == want;
    }
    if (next) {
      runs.back().b += 1;
    } else {
      runs.push_back(GridRun{d > 1 ? n[0] : 0, d > 2 ? n[1] : 0, n[d - 1], n[d - 1], (int)k, 0});
    }
  }
  return runs;
}

int failures = 0;

void check(const char* what, const std::set<Row>& set, int d, int N, int want_grid) {
  const std::vector<Row> rows(set.begin(), set.end());
  const int m = (int)rows.size();
  std::vector<Row> shuffled;   // a stride through the rows, as an unsorted set
  int stride = 7919;
  while (std::gcd(stride, m) != 1) ++stride;
  for (int k = 0; k < m; ++k) shuffled.push_back(rows[(long long)k * stride % m]);
  double sort = 1e30, plan = 1e30;
  const std::vector<GridRun> runs = runs_of(rows, d);
  ProbDev P{};
  GridPlan gp;
  for (int r = 0; r < 3; ++r) {
    std::vector<Row> x = shuffled;
    double t = now();
    std::stable_sort(x.begin(), x.end());
    sort = std::min(sort, now() - t);
    P = ProbDev{};
    P.d = d;
    P.N = N;
    P.M = m;
    P.ntile1 = (N + kPass1Tile - 1) / kPass1Tile;
    gp = GridPlan{};
    t = now();
    plan_grid(runs, &P, &gp);
    plan = std::min(plan, now() - t);
  }
  int bad = P.grid != want_grid;
  if (P.grid) {
    std::vector<int> seen(m, 0);
    for (int slot = 0; slot < P.gslots; ++slot) {
      const GridQuad& Q = gp.quads[slot >> 5];
      const int lane = slot & 31, row = lane >> 2, r = (row >> 1) + 4 * (row & 1), c = Q.c0 + (lane & 3);
      if (r >= Q.nrun) continue;
      const GridRun& g = gp.runs[Q.run0 + r];
      for (int sign : {1, -1}) {
        const int n = sign * c;
        if ((sign < 0 && c == 0) || n < g.a || n > g.b) continue;
        const int k = g.kstart + n - g.a;
        Row at{0, 0, 0};
        if (d > 1) at[0] = g.n0;
        if (d > 2) at[1] = g.n1;
        at[d - 1] = d == 1 ? g.n0 * P.gstep + n : n;
        bad += k < 0 || k >= m || rows[k] != at;
        if (k >= 0 && k < m) seen[k] += 1;
      }
    }
    for (int k = 0; k < m; ++k) bad += seen[k] != 1;
  }
  // both compiled alike; small sets are bound by the count of layouts, not by their rows
  const bool slow = plan > 2.0 * sort + 2e-3;
  std::printf("%s: %d rows, %zu runs, grid %d, plan %.2f ms, sort %.2f ms%s%s\n", what, m, runs.size(), P.grid,
              1e3 * plan, 1e3 * sort, bad ? " WRONG" : "", slow ? " SLOW" : "");
  failures += bad != 0 || slow;
}

std::set<Row> ball(int d, double r) {
  std::set<Row> s;
  const int R = (int)r + 1;
  for (int a = -R; a <= R; ++a)
    for (int b = d > 1 ? -R : 0; b <= (d > 1 ? R : 0); ++b)
      for (int c = d > 2 ? -R : 0; c <= (d > 2 ? R : 0); ++c) {
        const Row n{a, b, c};
        if (n > Row{0, 0, 0} && a * a + b * b + c * c < r * r) s.insert(n);
      }
  return s;
}

// Every multiple up to length `top` of the primitive vectors up to `dirs`.
std::set<Row> lines(int d, double dirs, double top) {
  std::set<Row> s;
  for (const Row& v : ball(d, dirs)) {
    if (std::gcd(std::gcd(std::abs(v[0]), std::abs(v[1])), std::abs(v[2])) != 1) continue;
    const double l = std::sqrt((double)(v[0] * v[0] + v[1] * v[1] + v[2] * v[2]));
    for (int i = 1; i * l <= top; ++i) s.insert(Row{i * v[0], i * v[1], i * v[2]});
  }
  return s;
}

std::set<Row> far_runs(int R, int len, int count) {
  std::set<Row> s;
  unsigned x = 1;
  auto draw = [&] { return (int)((x = x * 1664525u + 1013904223u) >> 8); };
  for (int i = 0; i < count; ++i) {
    const int a = draw() % R + 1, b = draw() % (2 * R) - R;
    for (int j = 0; j < len; ++j) s.insert(Row{a, b + j, 0});
  }
  return s;
}

}  // namespace

int main() {
  check("disc", ball(2, 107.0), 2, 20000, 1);
  check("small disc", ball(2, 22.5), 2, 1000, 1);
  check("ball", ball(3, 13.7), 3, 4000, 1);
  check("line", ball(1, 3732.5), 1, 7777, 1);
  check("multiples of directions", lines(2, 24.9, 500.0), 2, 1000, 0);
  check("long multiples of directions", lines(2, 24.9, 2000.0), 2, 1000, 0);
  check("far rows", far_runs(65000, 1, 20000), 2, 1000, 0);
  check("far rows in space", lines(3, 4.2, 900.0), 3, 500, 0);
  return failures != 0;
}
