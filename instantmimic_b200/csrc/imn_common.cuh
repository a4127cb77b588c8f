// imn_common.cuh -- helpers shared by the sm_100a kernels.
//
// Rounding contract: the translation units are compiled with -fmad=false, so a
// multiply followed by an add stays two roundings unless the source says
// fmaf(); sqrtf and '/' are the IEEE-rounded forms (nvcc defaults
// -prec-sqrt=true -prec-div=true, no fast-math).  Lane reductions follow a
// 32-lane shuffle-down tree whose lane-0 value is broadcast.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/imnewton.h"

#define IMN_FULL_MASK 0xFFFFFFFFu
#define IMN_MJ_MINVAL 1.0e-15f
#define IMN_MJ_MAXVAL 1.0e10f

namespace imn {

void set_error(const char* fmt, ...);
int sm_count();  // of the current device; 148 where there is none

// ---- launches that follow each other on a stream --------------------------------
//
// The stages of a step are kernels of 4 to 15 us, each the successor of the one before.  They are launched
// with programmatic stream serialisation: a kernel is launched once every block of its predecessor has
// released it or left, and waits in chain_wait until the predecessor's results are visible.
// Every kernel launched by launch_chained waits before it touches global memory; as it releases its
// successor only after its own wait, a waiting kernel has one unfinished kernel before it, and everything
// earlier is complete.  (Ordinary launches: a substep of 12 launches with 16 humanoid worlds 161 us
// against 146, the smooth stages of 8192 worlds 65 against 55, the implicit-fast tail 34 against 29.)
// A stage releases its successor by leaving (no call).  Released at once, the successor's blocks become
// resident while the grid drains and pile up on the SMs that drain first, where a later launch spreads them
// evenly, and a grid of few blocks gains nothing either.  us when every stage releases at once / grids of
// up to 64 blocks / none: factor with three right-hand sides and second solve, 4096 worlds 86 / 67 / 67, 256
// worlds 41.4 / 41.4 / 38.3; smooth stages, 8192 worlds 59 / 52 / 52, 2048 worlds 46 / 39 / 39; tail, 512 worlds
// 15.8 / 15.8 / 14.8.  The counter kernels of a solve, a block each, do release at once: the solve
// stages its tables meanwhile (substep of 512 worlds 145.1 -> 144.3 us, 4096 56-dof worlds 1096.6 -> 1094.1).
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void chain_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Largest dynamic shared memory one CTA may opt into on sm_100 (227 KB).
static const int kMaxSmem = 227 * 1024;

// Before a launch with `bytes` of dynamic shared memory.  More than 48 KB a block have to be allowed first, a
// limit of the function that all threads of the process share: it is always raised to the maximum,
// so that no call lowers it between another one's and that one's launch.
// whole_sm: several blocks are to fill an SM; the driver otherwise sizes the carve-out for one.
template <typename... P>
static inline cudaError_t allow_shared(void (*kernel)(P...), size_t bytes, bool whole_sm = false) {
  cudaError_t e = cudaSuccess;
  if (whole_sm) e = cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
  if (e == cudaSuccess && bytes > 48 * 1024) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem);
  return e;
}

template <typename... P, typename... A>
static inline cudaError_t launch_chained(void (*kernel)(P...), unsigned grid, unsigned threads, size_t bytes, cudaStream_t stream,
                                         A&&... args) {
  cudaLaunchAttribute follow;
  follow.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  follow.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid), cfg.blockDim = dim3(threads), cfg.dynamicSmemBytes = bytes, cfg.stream = stream;
  cfg.attrs = &follow, cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

__device__ __forceinline__ float safe_div(float x, float y) {
  return x / (y != 0.0f ? y : IMN_MJ_MINVAL);
}

// Jaref + alpha * jv with both roundings kept (newton_stages.py:18-19).
__device__ __forceinline__ float rounded_step(float a, float b, float c) {
  return __fadd_rn(a, __fmul_rn(b, c));
}

// Lane 0 of the shuffle-down tree, broadcast to the warp
// (newton_stages.py:39-45).
__device__ __forceinline__ float warp_tree_sum(float v) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v = v + __shfl_down_sync(IMN_FULL_MASK, v, off);
  return __shfl_sync(IMN_FULL_MASK, v, 0);
}

struct Vec3 {
  float c0, c1, c2;
};
__device__ __forceinline__ Vec3 v3(float a, float b, float c) { return Vec3{a, b, c}; }
__device__ __forceinline__ Vec3 operator+(Vec3 a, Vec3 b) {
  return Vec3{a.c0 + b.c0, a.c1 + b.c1, a.c2 + b.c2};
}
__device__ __forceinline__ Vec3 warp_tree_sum(Vec3 v) {
  return Vec3{warp_tree_sum(v.c0), warp_tree_sum(v.c1), warp_tree_sum(v.c2)};
}

}  // namespace imn
