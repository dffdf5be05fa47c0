// Launches on a first and a second device (two_devices_runtime.cpp).
#include <cstdio>

#include "cco_host.cuh"

namespace cco {
cudaError_t device_pool(cudaMemPool_t* p) { *p = nullptr; return cudaSuccess; }
size_t eval_smem2(const ProbDev&, int, bool) { return 0; }
}  // namespace cco

static int device = 0, bad = 0;

static void check(const char* what, int d, cudaError_t e) {
  if (e == cudaSuccess) return;
  ++bad;
  std::printf("device %d: %s d=%d failed (%d)\n", device, what, d, (int)e);
}

int main() {
  for (int dev : {0, 1, 0}) {
    device = dev;
    cudaSetDevice(dev);
    for (int d = 1; d <= 3; ++d) {
      cco_problem p;
      p.d = p.host.d = d;
      p.N = p.host.N = 40;
      p.M = p.host.M = 30;
      p.host.vol = 1.0;
      check("hessian", d, cco::hessian_launch(&p, nullptr, 1, nullptr, nullptr, nullptr));
    }
    cco::DescentArgs a{};
    for (int lanes : {1, 1000}) {
      a.B = lanes;
      for (int d = 1; d <= 3; ++d)
        for (int bit : {d - 1, d + 2})
          check("descent", d,
                cco::persist_descent(a, cco::EvalPlan{}, cco::kPersistMaxSmem, 1 << bit, 1, nullptr, nullptr));
    }
  }
  std::printf("%d bad\n", bad);
  return bad != 0;
}
