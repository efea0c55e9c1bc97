// Process-wide pieces every library built from this directory carries: the launch counter behind
// kllm_launch_count(), the version string and the error names of include/kllm_b200.h.
#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>
#include <mutex>

#include "kllm_host.h"

namespace kllm {
std::atomic<uint64_t>& launch_counter() {
  static std::atomic<uint64_t> c{0};
  return c;
}

int* wait_flag() {
  static std::atomic<int*> flag{nullptr};
  if (int* p = flag.load(std::memory_order_acquire)) return p;
  static std::mutex m;
  std::lock_guard<std::mutex> lock(m);
  int* p = flag.load(std::memory_order_relaxed);
  if (p == nullptr) {
    void* v = nullptr;
    if (cudaHostAlloc(&v, sizeof(int), cudaHostAllocMapped | cudaHostAllocPortable) != cudaSuccess) {
      cudaGetLastError();
      return nullptr;  // tried again at the next call
    }
    p = static_cast<int*>(v);
    *p = 0;
    flag.store(p, std::memory_order_release);
  }
  return p;
}
int take_wait_error() {
  int* p = wait_flag();
  if (p == nullptr || __atomic_load_n(p, __ATOMIC_RELAXED) == 0) return 0;
  __atomic_store_n(p, 0, __ATOMIC_RELAXED);
  return 1;
}
}  // namespace kllm

extern "C" {
const char* kllm_version(void) { return "kllm_b200 0.1 (sm_100a)"; }

const char* kllm_error_string(int code) {
  switch (code) {
    case KLLM_OK: return "ok";
    case KLLM_E_INVALID: return "invalid argument";
    case KLLM_E_UNSUPPORTED: return "unsupported shape";
    case KLLM_E_STATE: return "invalid decoder state";
    case KLLM_E_NODEVICE: return "no CUDA device";
    case KLLM_E_COMM: return "tensor-parallel transport unavailable or failed";
    default: return code > 0 ? cudaGetErrorString(static_cast<cudaError_t>(code)) : "unknown";
  }
}

uint64_t kllm_launch_count(void) { return kllm::launch_counter().load(); }
}
