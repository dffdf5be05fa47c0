// Host loops of the isotropic structure factor: its k-set and its bins
// (src/xla_cco/analysis/structure.py:113-201 of the reference). As array
// operations both went through a dozen fresh 800 KB temporaries (97 000 rows:
// 6.1 and 2.6 ms); one pass each keeps the same operations in the same order.
#include <cmath>
#include <cstdint>

#include "cco.h"
#include "cco_host.cuh"

using namespace cco;

extern "C" {

int cco_isotropic_rows(int d, int n_dir, const int64_t* dir, const double* k_dir,
                       const double* q_dir, double limit, int64_t cap, double* n_vec, double* sq,
                       int64_t* count) {
  if (d < 1 || d > 3 || n_dir < 0 || cap < 0) return fail(CCO_ERR_ARG, "bad sizes");
  if (!dir || !k_dir || !q_dir || !n_vec || !sq || !count) return fail(CCO_ERR_ARG, "null argument");
  int64_t out = 0;
  for (int v = 0; v < n_dir; ++v) {
    const int64_t last = (int64_t)std::sqrt(limit / q_dir[v]) + 2;
    for (int64_t i = 1; i <= last; ++i) {
      const double x = (double)i;
      double m2 = 0.0;
      for (int c = 0; c < d; ++c) {
        const double comp = x * k_dir[(size_t)v * d + c];
        m2 = m2 + comp * comp;
      }
      if (!(m2 <= limit)) continue;
      if (out >= cap) return fail(CCO_ERR_ARG, "more than %lld rows", (long long)cap);
      for (int c = 0; c < d; ++c) n_vec[(size_t)out * d + c] = x * (double)dir[(size_t)v * d + c];
      sq[out++] = m2;
    }
  }
  *count = out;
  return CCO_OK;
}

int cco_bin_sums(int64_t m, const double* k, const double* s, const double* s2, double width,
                 int64_t nb, double* sums) {
  if (m < 0 || nb < 1) return fail(CCO_ERR_ARG, "bad sizes");
  if (!k || !s || !s2 || !sums) return fail(CCO_ERR_ARG, "null argument");
  for (int64_t i = 0; i < m; ++i) {
    const double b = std::floor(k[i] / width);
    if (!(b >= 0.0 && b < (double)nb)) return fail(CCO_ERR_ARG, "row %lld outside the bins", (long long)i);
    double* o = sums + 5 * (int64_t)b;
    o[0] += 1.0;
    o[1] += k[i];
    o[2] += s[i];
    o[3] += k[i] * k[i];
    o[4] += s2[i];
  }
  return CCO_OK;
}

}  // extern "C"
