// Library-wide C ABI: error reporting and version.
#include <string.h>

#include <map>
#include <mutex>
#include <utility>

#include "common.cuh"

namespace ab {

static thread_local char g_last_error[512] = "";

int fail(int code, const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_last_error, sizeof(g_last_error), fmt, ap);
  va_end(ap);
  return code;
}

int cuda_status(cudaError_t e, const char* what) {
  return fail(AB_ERR_CUDA, "%s: %s (%s)", what, cudaGetErrorString(e), cudaGetErrorName(e));
}

cudaError_t allow_smem(const void* kernel, size_t bytes) {
  static std::mutex lock;
  static std::map<std::pair<int, const void*>, size_t> limits;   // one entry a kernel and device
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const std::lock_guard<std::mutex> hold(lock);
  size_t& limit = limits[{dev, kernel}];
  if (bytes <= limit) return cudaSuccess;
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e == cudaSuccess) limit = bytes;
  return e;
}

}  // namespace ab

extern "C" const char* ab_last_error(void) { return ab::g_last_error; }

extern "C" const char* ab_version(void) { return "augurv2_b200 0.1 (sm_100a)"; }
