// Where waits that run out inside a kernel are noted, so that each reaches the one who launched that kernel: an engine and a decoder
// have a flag of their own, the products that a program enqueues by themselves have one per stream.  A flag is an int of mapped host
// memory: a kernel writes it, the host reads it without a copy once it has waited for the owner's stream.
#pragma once
#include <cuda_runtime.h>

#include <mutex>
#include <unordered_map>

namespace kllm {

// memory for n flags, all 0 (nullptr: there is none).  The calling thread may be inside a stream capture, which forbids this kind
// of allocation unless it says that it means it.
inline int* new_wait_flags(int n) {
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  cudaThreadExchangeStreamCaptureMode(&mode);
  void* p = nullptr;
  const cudaError_t e = cudaHostAlloc(&p, sizeof(int) * n, cudaHostAllocMapped | cudaHostAllocPortable);
  cudaThreadExchangeStreamCaptureMode(&mode);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return nullptr;
  }
  for (int i = 0; i < n; ++i) static_cast<int*>(p)[i] = 0;
  return static_cast<int*>(p);
}
// 1 when the flag was raised since the last call
inline int take_wait_flag(int* p) { return p != nullptr && __atomic_exchange_n(p, 0, __ATOMIC_RELAXED) != 0; }

// The flag of one engine or decoder; it outlives that owner's kernels.
class WaitFlag {
 public:
  WaitFlag() = default;
  WaitFlag(const WaitFlag&) = delete;
  WaitFlag& operator=(const WaitFlag&) = delete;
  ~WaitFlag() {
    if (p_ != nullptr) cudaFreeHost(p_);
  }
  int* get() { return p_ != nullptr ? p_ : (p_ = new_wait_flags(1)); }
  int take() { return take_wait_flag(p_); }

 private:
  int* p_ = nullptr;
};

// One flag per stream, by the stream's id (unlike handles, ids are never used again).  A product that is captured cannot ask for the id
// and runs on other streams anyway: captured products, and streams after the first kStreams, share one more flag, which is taken by
// whoever asks for a status next.  What they noted is then never lost, and never taken for a wait of another stream's product.
class StreamWaitFlags {
 public:
  static constexpr int kStreams = 1023;
  int* get(unsigned long long id) {
    std::lock_guard<std::mutex> lock(m_);
    if (!allocate()) return nullptr;
    const auto it = place_.find(id);
    if (it != place_.end()) return flags_ + it->second;
    const int n = static_cast<int>(place_.size());
    if (n >= kStreams) return flags_ + kStreams;
    place_.emplace(id, n);
    return flags_ + n;
  }

  int* shared() {
    std::lock_guard<std::mutex> lock(m_);
    return allocate() ? flags_ + kStreams : nullptr;
  }

 private:
  bool allocate() { return flags_ != nullptr || (flags_ = new_wait_flags(kStreams + 1)) != nullptr; }  // (tried again at the next call)
  std::mutex m_;
  int* flags_ = nullptr;  // kept as long as the process runs: a kernel may still write there
  std::unordered_map<unsigned long long, int> place_;
};

// runtime.cu: where a product on `stream` notes a wait that ran out (nullptr: no device or no memory), and whether one is noted that
// is certain to be this stream's (the shared flag is left to kllm_product_status)
int* stream_wait_flag(cudaStream_t stream);
int take_own_wait_flag(int* flag);

}  // namespace kllm
