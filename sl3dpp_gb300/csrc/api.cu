// Error text, version and the device-memory helpers of the sl3dgpu C ABI.
#include <cstdint>
#include <mutex>
#include <set>
#include <string>
#include <utility>

#include "call_gate.cuh"
#include "common.cuh"

namespace sl3dgpu {

namespace {
thread_local std::string lastError;
}

void SetError(const std::string& text) { lastError = text; }

unsigned long long ContextId() {
  using GetId = int (*)(void* context, unsigned long long* id);
  static const GetId get = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult found{};
    if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &f, 12000, cudaEnableDefault, &found) != cudaSuccess ||
        found != cudaDriverEntryPointSuccess)
      f = nullptr;
    return reinterpret_cast<GetId>(f);
  }();
  unsigned long long id = 0;
  return get != nullptr && get(nullptr, &id) == 0 ? id : 0;
}

cudaError_t AllowDynamicSmemOnce(const void* kernel) {
  static std::mutex lock;
  static std::set<std::pair<unsigned long long, const void*>> done;  // (context, kernel)
  // what this thread last found done, by the kernel's address: no lock on most launches
  struct Seen {
    unsigned long long context = 0;
    const void* kernel = nullptr;
  };
  thread_local Seen seen[64];
  const unsigned long long context = ContextId();
  Seen& mine = seen[(reinterpret_cast<uintptr_t>(kernel) >> 4) % 64];
  if (context != 0 && mine.context == context && mine.kernel == kernel) return cudaSuccess;
  std::lock_guard<std::mutex> guard(lock);
  if (context != 0 && done.count({context, kernel}) != 0) {
    mine = Seen{context, kernel};
    return cudaSuccess;
  }
  int device = 0, optin = 0;
  if (const cudaError_t e = cudaGetDevice(&device); e != cudaSuccess) return e;
  if (const cudaError_t e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
      e != cudaSuccess)
    return e;
  cudaFuncAttributes a{};
  if (const cudaError_t e = cudaFuncGetAttributes(&a, kernel); e != cudaSuccess) return e;
  if (const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 optin - static_cast<int>(a.sharedSizeBytes));
      e != cudaSuccess)
    return e;
  if (context != 0) done.insert({context, kernel});
  return cudaSuccess;
}

}  // namespace sl3dgpu

extern "C" const char* sl3dgpu_last_error(void) { return sl3dgpu::lastError.c_str(); }

extern "C" const char* sl3dgpu_version(void) { return "sl3dgpu 0.1 (sm_103a)"; }

extern "C" int sl3dgpu_device_alloc(long long bytes, void** out) {
  const sl3dgpu::LibraryCall inside;
  if (out == nullptr || bytes < 0) {
    sl3dgpu::SetError("device_alloc: an output pointer and bytes >= 0");
    return SL3DGPU_ERR_ARGUMENT;
  }
  *out = nullptr;
  if (bytes == 0) return SL3DGPU_OK;
  SL3D_CUDA(cudaMalloc(out, static_cast<size_t>(bytes)));
  return SL3DGPU_OK;
}

extern "C" int sl3dgpu_device_free(void* p) {
  const sl3dgpu::LibraryCall inside;
  if (p != nullptr) SL3D_CUDA(cudaFree(p));
  return SL3DGPU_OK;
}

extern "C" int sl3dgpu_device_copy(void* dst, const void* src, long long bytes) {
  const sl3dgpu::LibraryCall inside;
  if (bytes < 0 || (bytes > 0 && (dst == nullptr || src == nullptr))) {
    sl3dgpu::SetError("device_copy: two pointers and bytes >= 0");
    return SL3DGPU_ERR_ARGUMENT;
  }
  if (bytes > 0) SL3D_CUDA(cudaMemcpy(dst, src, static_cast<size_t>(bytes), cudaMemcpyDefault));
  return SL3DGPU_OK;
}
