// Launches whose prologue overlaps the kernel before them in the stream (programmatic dependent launch).
//
// A kernel launched this way may start when every CTA of its predecessor has called chain_trigger() or has ended.  It
// calls chain_wait() before it touches anything that earlier kernels write or read; that call returns when the
// predecessor has completed and its writes are visible.  Every kernel here waits in all of its CTAs before it triggers,
// so by the time a kernel starts, everything before its immediate predecessor has completed.  What overlaps is the
// launch itself and the set-up of barriers, tensor memory and descriptors: 1 to 2 us for each kernel of a chain of
// short ones.
//
// What a predecessor may still be writing must not be read ahead of chain_wait(), neither by the source nor by the
// compiler.  So kernels that start this way take plain pointers.  `const T* __restrict__` would promise memory that
// nobody writes while the kernel runs: the compiler could fetch it along the non-coherent path, and in front of the wait,
// whose memory clobber does not cover such an argument.  Loads through plain pointers stay behind the wait, and so do the
// caching-hint loads (volatile assembly, like the wait itself).
#pragma once
#include <cuda_runtime.h>

#include <atomic>
#include <utility>

namespace cmoe {

// Kernels that this process has launched through the package, for whoever reports them.
inline std::atomic<long long> g_kernel_launches{0};
inline void count_launch() { g_kernel_launches.fetch_add(1, std::memory_order_relaxed); }

template <typename... P, typename... A>
cudaError_t launch_chained(void (*kernel)(P...), dim3 grid, unsigned threads, size_t smem, cudaStream_t stream,
                           A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  count_launch();
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}

#ifdef __CUDACC__
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// A table that the kernel before the predecessor (or an older one) wrote, read without waiting for the predecessor: past
// L1, which the wait would have made coherent.
__device__ __forceinline__ int load_ahead_of_wait(const int* p) { return __ldcg(p); }
__device__ __forceinline__ void chain_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
#endif

}  // namespace cmoe
