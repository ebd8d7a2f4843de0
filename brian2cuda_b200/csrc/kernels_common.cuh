// Device helpers shared by the libb2b kernels.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "b2b_internal.h"

namespace b2b {

constexpr unsigned kFull = 0xffffffffu;

__device__ __forceinline__ float dexp(float x) { return expf(x); }
__device__ __forceinline__ double dexp(double x) { return exp(x); }
__device__ __forceinline__ float dfma(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ float dexpm1(float x) { return expm1f(x); }
__device__ __forceinline__ double dexpm1(double x) { return expm1(x); }

// z / (exp(z) - 1), i.e. 1/exprel(z) with Brian2's exprel (brian2cuda/cuda_generator.py:858-867):
// the removable singularity at z = 0 evaluates to its limit 1 instead of 0/0.  Rate
// functions of the form c*x/(exp(x/a) - 1) are evaluated as c*a*z_over_expm1(x/a).
template <typename R>
__device__ __forceinline__ R z_over_expm1(R z) {
  return fabs(z) < (R)1e-16 ? (R)1 : z / dexpm1(z);
}
__device__ __forceinline__ double dfma(double a, double b, double c) { return fma(a, b, c); }

// Brian2's clip(value, a_min, a_max) (brian2cuda/cuda_generator.py:902-914).
template <typename R>
__device__ __forceinline__ R dclip(R v, R lo, R hi) {
  if (v < lo) return lo;
  if (v > hi) return hi;
  return v;
}

__device__ __forceinline__ void set_status(int32_t* status, int32_t code) {
  if (status) atomicCAS(status, 0, code);
}

// Block-wide exclusive scan of one int per thread.  Returns the thread's exclusive prefix;
// *total receives the block total.  `s_warp` needs blockDim.x/32 + 1 ints.
__device__ __forceinline__ int block_exclusive_scan(int c, int* s_warp, int* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nwarps = (blockDim.x + 31) >> 5;
  int x = c;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    int y = __shfl_up_sync(kFull, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) s_warp[warp] = x;
  __syncthreads();
  if (warp == 0) {
    int w = lane < nwarps ? s_warp[lane] : 0;
    int wx = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      int y = __shfl_up_sync(kFull, wx, o);
      if (lane >= o) wx += y;
    }
    if (lane < nwarps) s_warp[lane] = wx - w;   // exclusive warp offsets
    if (lane == nwarps - 1) s_warp[32] = wx;     // block total
  }
  __syncthreads();
  *total = s_warp[32];
  return s_warp[warp] + x - c;
}

// Programmatic dependent launch: a kernel launched chained (launch_kernel) may start while the
// previous one of its stream still runs.  It waits for that one's completion, and the visibility
// of its memory, in previous_launch_done(), which every thread of every CTA calls before it touches
// anything a kernel of the step writes; launched ordinarily there is nothing to wait for.  Ahead
// of it a kernel may read what stays as it is for a chunk of steps: its parameters, the clock,
// constants, random numbers.  A kernel that calls let_next_launch_start() lets the next one's CTAs
// in as room comes free.
__device__ __forceinline__ void previous_launch_done() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}
__device__ __forceinline__ void let_next_launch_start() {
  asm volatile("griddepcontrol.launch_dependents;");
}
template <class... KernelArgs, class... Args>
inline cudaError_t launch_kernel(void (*kernel)(KernelArgs...), dim3 grid, int block, size_t smem,
                                 cudaStream_t s, bool chained, const Args&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3((unsigned)block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = chained ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, KernelArgs(args)...);
}

// Floor modulo of a (possibly negative) step by the ring length.  Every kernel of a step
// starts with it, so steps below 2^31 (all but days of simulated time) take the 32-bit
// remainder: a 64-bit one is a long serial sequence in software.
__device__ __forceinline__ int ring_slot(int64_t step, int ring_len) {
  if ((uint64_t)step <= (uint64_t)INT32_MAX) return (int)((uint32_t)step % (uint32_t)ring_len);
  int64_t r = step % ring_len;
  return (int)(r < 0 ? r + ring_len : r);
}

}  // namespace b2b
