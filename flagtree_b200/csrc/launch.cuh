// Launch of a kernel whose prologue may overlap the end of the kernel before it in the stream (programmatic dependent launch).
//
// Every kernel launched this way executes griddep_launch(), which lets the next one begin as soon as all CTAs of this one have executed it (or have left), and
// griddep_wait() in all of its threads before its first access to global memory, which returns when the kernels
// before it have completed and their writes are visible.  Back to back (us, before / now): 50 x 7168 x 2304 bf16
// 12.3 / 10.1, 64 x 8192 x 3584 e4m3 14.6 / 13.1, one token of 128 heads in parts (two launches) 18.5 / 16.9, a decode step of three
// sequences (four launches) 45.1 / 40.2, 262 144 cache rows (five launches) 116.7 / 113.3.
// Where griddep_launch() stands: first, unless the CTAs of a kernel have several items of work and end at different times; those execute
// it last.  The next kernel's CTAs would otherwise crowd on the SMs that are through first and stay there: with a persistent kernel that let
// the next step's top-k kernel in early, a decode step of 128 tokens took 186 us, without any overlap 179, now 178.  For the same reason the cache
// writer's run kernel lets its successor in late where that one has much to do (kv_cache.cu), the bf16 GEMM leaves few rows on few SMs out (gemm.cu), and a
// kernel of few large CTAs asks for more than half of an SM's shared memory.
#pragma once
#include <cuda_runtime.h>

namespace ftb {

__device__ __forceinline__ void griddep_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// (No pointer that a kernel before may have written through is __restrict__ or read with __ldg: such a load may move above the wait.)
__device__ __forceinline__ void griddep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <class... P, class... A>
inline cudaError_t launch_overlapped(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, unsigned cluster, A... args) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = cluster; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = cluster > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

}  // namespace ftb
