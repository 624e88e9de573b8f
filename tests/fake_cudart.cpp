// A CUDA runtime without a GPU, for the host side of the launchers: launches are refused as the real one would refuse them
// (dynamic shared memory above the 48 KB that every kernel may use and above the kernel's limit on the current device),
// counted, and otherwise ignored.
#include <cuda.h>
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <utility>

#include "api.h"
#include "launch_hints.h"

namespace {
int device = 0, launches = 0;
int late_waits = 0;         // one bit for each launch, the last one lowest
cudaError_t last_error = cudaSuccess;
std::map<std::pair<const void*, int>, int> limits;

cudaError_t launch(const void* func, size_t smem) {
  const auto it = limits.find({func, device});
  const size_t limit = it == limits.end() ? 48 * 1024 : it->second;
  if (smem > limit) return last_error = cudaErrorInvalidValue;
  ++launches;
  late_waits = late_waits << 1 | (gfs_host::launch_hints().late_wait ? 1 : 0);
  return cudaSuccess;
}
CUresult encode(CUtensorMap* out) {
  std::memset(out, 0, sizeof(*out));
  return CUDA_SUCCESS;
}
}  // namespace

extern "C" {
void fake_set_device(int dev) { device = dev; }
int fake_launches() { return launches; }

// three products of M x N x K in a scope in which the first one waits late
int fake_late_waits(int M, int N, int K) {
  late_waits = 0;
  const gfs_host::WithHints hints(true, true);
  void* p = reinterpret_cast<void*>(1 << 20);
  for (int i = 0; i < 3; ++i)
    if (gfs_linear(p, p, p, nullptr, M, N, K, K, K, N, 0, 0, 0, nullptr, nullptr, 0, 0, 1, 60, nullptr) != 0) return -1;
  return late_waits << 1 | (gfs_host::launch_hints().early_b ? 1 : 0);
}

cudaError_t cudaGetDevice(int* dev) { *dev = device; return cudaSuccess; }
cudaError_t cudaGetLastError() { return std::exchange(last_error, cudaSuccess); }
const char* cudaGetErrorString(cudaError_t) { return "error of the fake runtime"; }
cudaError_t cudaDeviceGetAttribute(int* value, cudaDeviceAttr, int) { *value = 148; return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void* func, cudaFuncAttribute attr, int value) {
  if (attr == cudaFuncAttributeMaxDynamicSharedMemorySize) limits[{func, device}] = value;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* func, dim3, dim3, void**, size_t smem, cudaStream_t) { return launch(func, smem); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* cfg, const void* func, void**) {
  return launch(func, cfg->dynamicSmemBytes);
}
static size_t pushed_smem;
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t smem, CUstream_st*) { pushed_smem = smem; return 0; }
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* smem, void* stream) {
  *grid = *block = dim3{1, 1, 1};
  *smem = pushed_smem;
  *static_cast<void**>(stream) = nullptr;
  return cudaSuccess;
}
cudaError_t cudaMalloc(void** p, size_t n) { *p = std::calloc(1, n); return cudaSuccess; }
cudaError_t cudaFree(void* p) { std::free(p); return cudaSuccess; }
cudaError_t cudaMemset(void*, int, size_t) { return cudaSuccess; }
cudaError_t cudaMemsetAsync(void*, int, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode*) { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = nullptr; return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGetDriverEntryPoint(const char*, void** fn, unsigned long long, cudaDriverEntryPointQueryResult* q) {
  *fn = reinterpret_cast<void*>(encode);
  if (q != nullptr) *q = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}
void** __cudaRegisterFatBinary(void*) { return nullptr; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, void*, void*, void*, void*, int*) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
}
