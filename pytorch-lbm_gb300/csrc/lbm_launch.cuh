// Programmatic dependent launch of the step kernels.
#pragma once
#include <cuda_runtime.h>

#include "lbm_common.cuh"

namespace lbm {

// Programmatic dependent launch between the step kernels: a kernel launched
// with the programmatic-serialization attribute may start while the kernel
// before it drains; it reads its descriptor, lets the next kernel be
// scheduled (each block triggers on entry, so the next grid starts during
// this grid's last wave), and waits for the previous grid to complete and
// flush its memory before it reads anything that grid wrote.
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Launch with programmatic stream serialization (see pdl_wait).
constexpr int kPdlOn = 1;  // 0: plain stream serialization
template <typename... KArgs, typename... Args>
static cudaError_t launch_pdl_sm(void (*fn)(KArgs...), int blocks, int threads, size_t smem, cudaStream_t st,
                                 const Args&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)blocks);
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = kPdlOn;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, fn, args...);
}
template <typename... KArgs, typename... Args>
static cudaError_t launch_pdl_bs(void (*fn)(KArgs...), int blocks, int threads, cudaStream_t st,
                                 const Args&... args) {
  return launch_pdl_sm(fn, blocks, threads, 0, st, args...);
}
template <typename... KArgs, typename... Args>
static cudaError_t launch_pdl(void (*fn)(KArgs...), int blocks, cudaStream_t st, const Args&... args) {
  return launch_pdl_bs(fn, blocks, kBlock, st, args...);
}

}  // namespace lbm
