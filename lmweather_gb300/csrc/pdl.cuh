// Programmatic dependent launch: a kernel launched with stage_launch may start while its predecessor drains. It waits in
// pdl_wait (everything the predecessor wrote is then visible, and the predecessor had waited for its own) before it
// touches anything an earlier kernel writes, and lets its successor start with pdl_trigger (the first thread of a CTA counts
// for it) when only its outputs are left. The persistent split kernels, whose CTAs are as many on every SM, trigger
// right after their wait: a successor then takes no SM from CTAs still to come, and it waits for all of them all the
// same. In a kernel launched without the attribute both do nothing.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>

#include "lmw_internal.h"

namespace lmw {
namespace {

// The wait takes the kernel's __restrict__ pointers to what earlier kernels of the chain write, and hands them back as values
// unknown before it: through a const __restrict__ parameter the compiler may read ahead of any instruction (the loads are
// of memory that the kernel has promised not to change), the wait included, and past the caches' coherence.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
template <class T> __device__ __forceinline__ void pdl_fresh(T &p) {
  unsigned long long v = reinterpret_cast<unsigned long long>(p);
  asm volatile("" : "+l"(v)::"memory");
  p = reinterpret_cast<T>(v);
}
template <class... T> __device__ __forceinline__ void pdl_wait(T &...p) {
  pdl_wait();
  (pdl_fresh(p), ...);
}
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Dynamic shared memory for a launch of `ctas` CTAs that need `need` bytes: where they are few, so much that no more than
// their even share fits on one SM. CTAs that start while the predecessor drains go where there is room, that is to the SMs
// that are done first, and would pile up there (a stage
// of one member, FP64: T85 44.4 -> 35.3 us, T170 105 -> 99; split form, T170: 49 -> 40). Past five
// CTAs per SM the share no longer pays (T31 x 3 with tracer, 768 CTAs in clusters of eight: 3.64 ms a run held to six, 3.54 free).
inline size_t even_share(size_t need, long ctas) {
  const long share = (ctas + kSMs - 1) / kSMs;
  return share > 5 ? need : std::max(need, kSmemPerSM / (share + 1) - 768);
}

// launch of a kernel that calls pdl_wait, in clusters of `cluster` CTAs along x
template <class... P, class... A>
void stage_launch(void (*k)(P...), dim3 grid, int threads, size_t smem, cudaStream_t stream, int cluster, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = cluster;
  at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = cluster > 1 ? 2 : 1;
  LMW_CUDA(cudaLaunchKernelEx(&cfg, k, static_cast<P>(args)...));
}

}  // namespace
}  // namespace lmw
