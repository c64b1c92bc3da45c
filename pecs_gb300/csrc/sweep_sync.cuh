// Ordering between the launches (and, in flow sweeps, the CTAs) of a solve sweep.
#pragma once
#include <cuda_runtime.h>

namespace pecs {
namespace {

// Programmatic dependent launch: a sweep level is launched while the previous
// level still runs; it stages what does not depend on that level (item
// records, index metadata, its block tile) and then waits for the previous
// grid's completion and memory (griddepcontrol.wait) before reading vectors.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }

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
