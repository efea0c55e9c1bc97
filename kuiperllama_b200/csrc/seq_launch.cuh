// Launches that may begin while the kernel before them on the stream still runs (programmatic dependent launch).  A decode step is
// a chain of some thirty to sixty kernels of a few microseconds; without this each begins only when the one before has drained.
//
// A kernel launched by launch_ahead() calls after_previous() before it reads anything that an earlier kernel wrote and before it
// writes anything; ahead of that call it may set itself up and read weights, which no kernel writes, and, in a step of the engine, what was
// complete before the step's first kernel began, which is an ordinary launch: the step's index arrays, and keys and page entries of
// earlier steps.  (That an earlier kernel of the step must have ended is not enough: only the wait makes its stores visible.)  Every such kernel does call
// it, so a kernel that has finished vouches for all kernels before it, not for its predecessor alone.  next_may_start() lets the
// following kernel's CTAs take up what room is left; a kernel that allocates TMEM calls it after the allocation, so that a CTA which
// waits for this kernel never holds columns that this kernel still needs.
//
// Such a kernel is alive while earlier ones still write.  Loads through the read-only path (__ldg, ld.global.nc, a
// `const __restrict__` parameter) are allowed only for data that nothing writes during the kernel's whole life, and the compiler may
// move them, and accesses through any `__restrict__` parameter, across after_previous().  So in these kernels weights alone are
// `__restrict__` or read that way; whatever a kernel of the step reads or writes besides goes through plain pointers
// (tests/test_launch_rules.py).
//
// Only inside a step: its weights are not written by any kernel on the stream.  A product that a caller enqueues by itself begins
// after everything the caller enqueued before, which may have written its weights.
#pragma once
#include <cuda_runtime.h>

#include <utility>

namespace kllm {
namespace seq {

__device__ __forceinline__ void after_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void next_may_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// (ahead == false: an ordinary launch, behind everything that is on the stream)
template <typename... P, typename... A>
inline cudaError_t launch_maybe_ahead(bool ahead, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                                      A&&... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = ahead ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, P(std::forward<A>(args))...);
}
template <typename... P, typename... A>
inline cudaError_t launch_ahead(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A&&... args) {
  return launch_maybe_ahead(true, kernel, grid, block, smem, stream, std::forward<A>(args)...);
}

}  // namespace seq
}  // namespace kllm
