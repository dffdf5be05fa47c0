// A process with two devices, on the CPU: the CUDA runtime calls that the linked
// sources make are defined here. Function attributes are kept per device, as the
// runtime keeps them, and a launch with more dynamic shared memory than its kernel
// was allowed on the current device fails. No kernel runs.
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <map>
#include <utility>

namespace {
int device = 0;
cudaError_t last = cudaSuccess;
std::map<std::pair<int, const void*>, size_t> allowed;
struct Config {
  dim3 grid, block;
  size_t smem;
  void* stream;
} config;
}  // namespace

extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { device = d; return cudaSuccess; }
cudaError_t cudaGetLastError() { const cudaError_t e = last; last = cudaSuccess; return e; }
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int value) {
  if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) allowed[{device, f}] = (size_t)value;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3, dim3, void**, size_t smem, cudaStream_t) {
  const auto it = allowed.find({device, f});
  if (smem > (it == allowed.end() ? 48 * 1024 : it->second)) last = cudaErrorInvalidValue;
  return last;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void** args) {
  return cudaLaunchKernel(f, c->gridDim, c->blockDim, args, c->dynamicSmemBytes, c->stream);
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) {
  *n = 1;
  return cudaSuccess;
}
cudaError_t cudaMallocFromPoolAsync(void** p, size_t, cudaMemPool_t, cudaStream_t) {
  *p = std::malloc(1);
  return cudaSuccess;
}
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { std::free(p); return cudaSuccess; }
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, CUstream_st* s) {
  config = Config{g, b, smem, s};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* smem, void* s) {
  *g = config.grid;
  *b = config.block;
  *smem = config.smem;
  *static_cast<void**>(s) = config.stream;
  return cudaSuccess;
}
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
char __cudaInitModule(void**) { return 1; }
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*, dim3*, int*) {}
}
