// Ordering between the launches (and, in flow sweeps, the CTAs) of a solve sweep or of a
// pass through the network.
#pragma once
#include <cuda_runtime.h>

#include "common.hpp"

namespace pecs {
namespace {

// Programmatic dependent launch (launch_pdl): a level is launched while the previous
// one still runs; it stages what does not depend on that level (item
// records, index metadata, its block tile) and then waits for the previous
// grid's completion and memory (griddepcontrol.wait) before reading vectors.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }

// launches with programmatic stream serialisation
template <typename... P, typename... A>
void launch_pdl(void (*fn)(P...), dim3 grid, int threads, size_t smem, cudaStream_t st, A... args) {
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  PECS_CUDA(cudaLaunchKernelEx(&cfg, fn, args...));
}

// Polls of one wait before it gives up (with 64 ns sleeps and a global load
// each: tens to hundreds of milliseconds, against a whole sweep of well under
// a millisecond).
constexpr unsigned kFlowPollLimit = 1u << 18;

__device__ __forceinline__ int ld_acquire_gpu(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.b32 %0, [%1];\n" : "=r"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ void red_release_gpu(int* p, int v) {
  asm volatile("red.release.gpu.global.add.s32 [%0], %1;\n" ::"l"(p), "r"(v) : "memory");
}

// Bounded wait for *ctr >= target; false (and the error flag set) when the
// poll limit runs out.
__device__ __noinline__ bool flow_wait(const int* ctr, int target, int* err) {
  if (ld_acquire_gpu(ctr) >= target) return true;
  for (unsigned n = 0; n < kFlowPollLimit; ++n) {
    __nanosleep(64);
    if (ld_acquire_gpu(ctr) >= target) return true;
  }
  atomicExch(err, 1);
  return false;
}

}  // namespace
}  // namespace pecs
