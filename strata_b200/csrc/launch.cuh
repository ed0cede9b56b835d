// Kernel launches of this library: every kernel is launched with programmatic stream
// serialisation, so that the next kernel of the stream may start while the blocks of this one
// finish - its set-up (barriers, tensor memory, descriptors) and the launch latency overlap the
// tail - and every kernel begins with chain_begin(), which waits until everything before it in the
// stream has completed and is visible. Between two kernels of a block on a small tile the gap was
// 1.8 us (7 kernels of 3-13 us); it shows in calls whose kernels are short.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>

namespace strata {

// Executed by every thread of a kernel before its first access to global memory (reads and
// writes: the kernel before may still be reading what this one overwrites). A kernel that
// allocates tensor memory calls it after the allocation: only then may blocks of the next kernel
// share its SM, so they cannot take columns that this kernel's own blocks still wait for.
__device__ __forceinline__ void chain_begin() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// The kernel's dynamic shared-memory limit, raised once per device (`done`: one bit per device,
// one variable per kernel; concurrent first calls set the same value).
inline cudaError_t allow_smem(const void* kern, int bytes, std::atomic<uint64_t>& done) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const uint64_t bit = 1ull << (dev & 63);
  if (dev < 64 && (done.load(std::memory_order_relaxed) & bit)) return cudaSuccess;
  e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e == cudaSuccess && dev < 64) done.fetch_or(bit, std::memory_order_relaxed);
  return e;
}

// Returns 0 or -(cudaError) - 1000. cluster: blocks per cluster along x (1: none).
template <typename... P, typename... A>
inline int launch_kernel(void (*kern)(P...), dim3 grid, int threads, size_t smem, cudaStream_t stream,
                          int cluster, bool chained, const A&... args) {
  static_assert(sizeof...(P) == sizeof...(A), "one argument per kernel parameter");
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(static_cast<unsigned>(threads));
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  unsigned n = 0;
  if (chained) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (cluster > 1) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = static_cast<unsigned>(cluster);
    attr[n].val.clusterDim.y = 1;
    attr[n++].val.clusterDim.z = 1;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...);
  return e == cudaSuccess ? 0 : -static_cast<int>(e) - 1000;
}
template <typename... P, typename... A>
inline int launch_chained(void (*kern)(P...), dim3 grid, int threads, size_t smem, cudaStream_t stream,
                          int cluster, const A&... args) {
  return launch_kernel(kern, grid, threads, smem, stream, cluster, true, args...);
}
// The same without the overlap, for long persistent kernels: it gains them nothing, and blocks that come in
// one by one as others leave land on other SMs than in a plain launch, neighbouring items away
// from each other (attention over 2 x 32 x 96 x 96 tokens: 5.64 ms chained, 5.59 plain).
template <typename... P, typename... A>
inline int launch_plain(void (*kern)(P...), dim3 grid, int threads, size_t smem, cudaStream_t stream,
                        int cluster, const A&... args) {
  return launch_kernel(kern, grid, threads, smem, stream, cluster, false, args...);
}

}  // namespace strata
