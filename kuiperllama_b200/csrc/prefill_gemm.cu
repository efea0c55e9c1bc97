// Batched products for prompt prefill on the 5th-generation tensor cores (sm_100a):
//     out[T, N] = x[T, K] . w[N, K]^T        fp32 storage, TF32 multiply, fp32 accumulate
// plain (with an optional bias), gated (two weight matrices joined by SiLU * gate) and added to a residual.
//
// The reference feeds a prompt through one full single-token forward per position (demo/main.cpp:
// 18-23, llama3.cpp:147-167) -- T GEMVs that stream every weight T times.  With the T prompt rows
// as the N dimension of a tcgen05.mma the weights are streamed once per block of tokens.
//
// These are explicitly TOLERANCED: TF32 keeps 10 mantissa bits of each operand, so results agree with the fp32 GEMV
// path to ~1e-3 relative, not bit for bit (tests/test_prefill_gpu.py states the bound).  The bit-exact decode path
// never calls them.  The kernel is the sequence engine's split product with operands read as TF32
// (seq_gemm_split.cuh): a projection of a 2048-wide model has 16 feature tiles, so K is split until the grid fills the chip.
// Measured with the attention of prefill.cu in tiles, 900 tokens through 4 layers of TinyLlama-1.1B: 12.9 -> 3.0 ms; of the 12.9,
// 4.2 ms were products of 256-token blocks whose grids had 2, 16 or 44 CTAs.
#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "../../include/kllm_b200.h"
#include "kllm_host.h"
#include "seq_engine.h"
#include "seq_gemm_split.cuh"
#include "wait_flag.h"

namespace kllm {
namespace {

// The narrowest token block that holds the rows; where 128-token tiles fill the chip, persistent CTAs.
template <int OUT>
int product(const seq::umma::SplitArgs& p, cudaStream_t s, bool ahead = true) {
  using namespace seq::umma;
  if constexpr (OUT != kThree)
    if (fills_chip(p.T, p.N)) return launch_tiles<kTf32, OUT>(p, s);
  if (p.T <= 16) return launch_split<kTf32, 16, OUT, 5>(p, s, ahead);
  if (p.T <= 32) return launch_split<kTf32, 32, OUT, 5>(p, s, ahead);
  if (p.T <= 64) return launch_split<kTf32, 64, OUT, 4>(p, s, ahead);
  return launch_split<kTf32, 128, OUT, 3>(p, s, ahead);
}
// TMA needs 16-byte aligned bases and row pitches
bool aligned(const void* x, const void* w, int K) {
  return (K & 3) == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0 && (reinterpret_cast<uintptr_t>(w) & 15) == 0;
}
constexpr seq::GatedAct kSwiglu{KLLM_SEQ_ACT_SWIGLU, 0.f, 0.f};

}  // namespace

int prefill_product(const float* x, const float* w, const float* bias, float* out, int T, int K, int N, cudaStream_t s,
                    int* wait, bool ahead) {
  if (!aligned(x, w, K)) return KLLM_E_UNSUPPORTED;
  return product<seq::umma::kPlain>({x, w, nullptr, bias, nullptr, out, T, N, K, 1, kSwiglu, wait}, s, ahead);
}
// Queries, keys and values: one launch while the queries alone do not fill the chip (900 x 2048 against 2048 + 256 + 256 rows: one after the
// other 25 + 15 + 15 us, the last two bound by the way to and through a cluster of eight; together 32).
int prefill_product_three(const float* x, const float* const (&w)[3], const float* const (&bias)[3], float* const (&out)[3], int T, int K,
                          const int (&N)[3], cudaStream_t s, int* wait) {
  using namespace seq::umma;
  if (fills_chip(T, N[0])) {
    for (int i = 0; i < 3; ++i)
      if (const int rc = prefill_product(x, w[i], bias[i], out[i], T, K, N[i], s, wait)) return rc;
    return 0;
  }
  for (int i = 0; i < 3; ++i)
    if (!aligned(x, w[i], K)) return KLLM_E_UNSUPPORTED;
  return product<kThree>({x, w[0], w[1], bias[0], nullptr, out[0], T, N[0], K, 1, kSwiglu, wait, w[2], bias[1], bias[2], out[1], out[2],
                          N[1], N[2]}, s);
}
int prefill_product_add(const float* x, const float* w, float* residual, int T, int K, int N, cudaStream_t s, int* wait) {
  if (!aligned(x, w, K)) return KLLM_E_UNSUPPORTED;
  return product<seq::umma::kAdd>({x, w, nullptr, nullptr, residual, residual, T, N, K, 1, kSwiglu, wait}, s);
}
int prefill_product_gated(const float* x, const float* w1, const float* w3, float* out, int T, int K, int N, cudaStream_t s,
                          int* wait) {
  if (!aligned(x, w1, K) || !aligned(x, w3, K)) return KLLM_E_UNSUPPORTED;
  return product<seq::umma::kGated>({x, w1, w3, nullptr, nullptr, out, T, N, K, 1, kSwiglu, wait}, s);
}

}  // namespace kllm

extern "C" int kllm_gemm_tf32(const float* x, const float* w, float* out, int n_tokens, int in_dim, int out_dim,
                              void* stream) {
  if (!x || !w || !out || n_tokens <= 0 || in_dim <= 0 || out_dim <= 0) return KLLM_E_INVALID;
  const cudaStream_t s = static_cast<cudaStream_t>(stream);
  int* const wait = kllm::stream_wait_flag(s);
  if (wait == nullptr) return KLLM_E_STATE;
  if (const int rc = kllm::prefill_product(x, w, nullptr, out, n_tokens, in_dim, out_dim, s, wait, false)) return rc;
  return kllm::take_own_wait_flag(wait) ? KLLM_E_STATE : 0;
}
