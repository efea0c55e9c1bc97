// Process-wide pieces every library built from this directory carries: the launch counter behind
// kllm_launch_count(), the flags of products enqueued by themselves, the version string and the error names of include/kllm_b200.h.
#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>

#include "../../include/kllm_seq.h"
#include "kllm_host.h"
#include "wait_flag.h"

namespace kllm {
std::atomic<uint64_t>& launch_counter() {
  static std::atomic<uint64_t> c{0};
  return c;
}

namespace {
StreamWaitFlags& stream_flags() {
  static StreamWaitFlags f;
  return f;
}
}  // namespace
int* stream_wait_flag(cudaStream_t stream) {
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  unsigned long long id = 0;
  if (cudaStreamIsCapturing(stream, &capture) == cudaSuccess && capture == cudaStreamCaptureStatusNone &&
      cudaStreamGetId(stream, &id) == cudaSuccess)
    return stream_flags().get(id);
  cudaGetLastError();
  return stream_flags().shared();
}
int take_own_wait_flag(int* flag) { return flag != stream_flags().shared() && take_wait_flag(flag); }
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

int kllm_product_status(void* stream) {
  const cudaError_t e = cudaStreamSynchronize(static_cast<cudaStream_t>(stream));
  if (e != cudaSuccess) return static_cast<int>(e);
  const int own = kllm::take_wait_flag(kllm::stream_wait_flag(static_cast<cudaStream_t>(stream)));
  return own | kllm::take_wait_flag(kllm::stream_flags().shared()) ? KLLM_E_STATE : 0;
}

uint64_t kllm_launch_count(void) { return kllm::launch_counter().load(); }
}
