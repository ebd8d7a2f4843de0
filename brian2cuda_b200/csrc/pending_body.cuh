// The delivery half of the step forms whose every synaptic delay is at least one step
// (pending.cu: its own launch beside the update; neuron.cu: the CTAs after the update's in
// the one-launch step): the bundles due at step clock+k are added into the pending input
// acc[k & 1] instead of the target variables.
#pragma once
#include "delivery.cuh"

namespace b2b {
namespace {

constexpr int kPendingBlock = 256;
constexpr int kPendingUnroll = 4;   // rounds of a bundle whose loads a lane issues together

// The work of CTA `blk` of `nblk` delivering CTAs (blockDim.x threads each).
// CHAINED: in a launch that may start before the previous step's has ended.
template <typename R, bool WARP_PREFIX, int GROUP, int NP, bool CHAINED = false>
__device__ __forceinline__ void deliver_pending_body(const PendingArgs<NP>& F,
                                                     const int64_t* __restrict__ clock, int k,
                                                     int64_t blk, int64_t nblk, int* s_pref) {
  const int64_t ts = clock[0] + k;
  const int64_t warp0 = (blk * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = (nblk * blockDim.x) >> 5;
  const int64_t row = (int64_t)(k & 1) * F.n;
  // a quiet step has lanes to spare (us per step at as many as in a busy one / more: four there, LIF
  // f32 150,000 neurons with bundles of 4 3.73 / 3.64, 100,000 3.20 / 3.16; eight, HH f64 8001 3.27 /
  // 3.23, LIF f32 20,000 3.02 / 2.97)
  constexpr int kQuiet = GROUP < 8 ? 8 : 16;
  if constexpr (CHAINED) {
    // the projection's fields and the clock are in registers before the wait
    const AddDev& J = F.proj[0];
    asm volatile("" ::"l"(J.src_ring_cnt), "l"(J.src_ring_idx), "l"(J.src_n), "r"(J.src_ring_len),
                 "r"(J.dmin), "r"(J.nd), "r"(J.chunks), "l"(J.src_lo), "l"(J.src_hi), "l"(J.off),
                 "l"(J.post), "l"(ts));
    previous_launch_done();
  }
  for (int p = 0; p < (NP == 1 ? 1 : F.n_proj); ++p) {
    const AddDev& J = F.proj[p];
    const R* W = static_cast<const R*>(J.w);
    MemberCache<R> mc;
    for_each_due_item<WARP_PREFIX, GROUP, kQuiet>(J, ts, warp0, nwarps, s_pref,
                                                  [&](int64_t b0, int64_t b1, int64_t len,
                                                      int32_t pre, int64_t, auto width) {
      constexpr int kWidth = decltype(width)::value;
      const int glane = (threadIdx.x & 31) % kWidth;
      member_lookup<R>(J, pre, mc);
      // the loads of kPendingUnroll rounds first, then their atomics
      for (int64_t off = 0; off < len; off += kPendingUnroll * kWidth) {
        int32_t post[kPendingUnroll];
        R w[kPendingUnroll];
        bool v[kPendingUnroll];
#pragma unroll
        for (int u = 0; u < kPendingUnroll; ++u) {
          const int64_t s = b0 + off + u * kWidth + glane;
          v[u] = s < b1;
          post[u] = v[u] ? __ldg(J.post + s) : 0;
          w[u] = v[u] && W ? __ldg(W + s) : mc.w;
        }
#pragma unroll
        for (int u = 0; u < kPendingUnroll; ++u)
          if (v[u]) atomicAdd(mc.target + row + post[u], w[u]);
      }
    });
  }
}

}  // namespace
}  // namespace b2b
