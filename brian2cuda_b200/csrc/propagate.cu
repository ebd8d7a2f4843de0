// Spike propagation: delivery of due synapse bundles from the spike-history ring, with the
// on_pre / on_post effects (additive, and event-driven STDP with its traces) applied in the
// same pass.
//
// Reference: the per-step push of (pre, post-block, delay) bundle ids into CudaSpikeQueue
// slots `(current_offset + delay) % num_queues` under per-post-block spin locks with
// device-malloc growth (brian2cuda/brianlib/spikequeue.h:432-511, templates/
// synapses_push_spikes.cu:1056-1131), then the effect kernel over the current slot
// (templates/synapses.cu:12-164) with `_brian_atomicAdd` (cuda_generator.py:33-157).
//
// Here nothing is pushed.  Each population keeps the compacted spikes of its last
// `ring_len` steps (written by the neuron kernel).  A bundle (pre, d) is due at step ts
// exactly when pre spiked at step ts - d, so the delivery kernels enumerate, for every delay
// d of the projection, the spikes of ring slot ts - d and walk the synapse range of bundle
// (pre, d) in the (pre, delay)-sorted synapse arrays (delivery.cuh).  This is the same set of
// bundles the reference's queue holds in slot `current_offset` after its push, without the
// push kernel, the host sync on the spike count, the locks or the device heap.
#include <cooperative_groups.h>

#include <algorithm>
#include <mutex>
#include <vector>

#include "delivery.cuh"

namespace cg = cooperative_groups;

namespace b2b {

namespace {

constexpr int kDeliverBlock = 256;
constexpr int kAddUnroll = 4;

// Sum of `v` over the lanes whose key equals this lane's key; valid in every lane.
template <typename R>
__device__ __forceinline__ R peer_sum(unsigned peers, R v) {
  R acc = 0;
#pragma unroll 1
  for (int src = 0; src < 32; ++src) {
    const R x = __shfl_sync(kFull, v, src);
    if ((peers >> src) & 1u) acc += x;
  }
  return acc;
}

// T[post] += w for one synapse per lane; AGG sums lanes hitting the same element first.  The
// lanes of a warp may write different target arrays (the members of a projection that merges
// several Synapses objects), so lanes are matched on the element's address.
template <typename R, bool AGG>
__device__ __forceinline__ void add_to_target(R* T, int32_t post, R w, bool valid) {
  if constexpr (AGG) {
    const unsigned peers =
        __match_any_sync(kFull, valid ? (unsigned long long)(T + post) : 0ull);
    const R sum = peer_sum<R>(peers, valid ? w : (R)0);
    if (valid && (int)(threadIdx.x & 31) == __ffs(peers) - 1) atomicAdd(T + post, sum);
  } else {
    if (valid) atomicAdd(T + post, w);
  }
}

// Several additive projections in one launch: blockIdx.y picks the projection.  (One projection,
// the ordinary case, travels in a parameter block of its own size.)
template <int NP>
struct AddBatch {
  AddDev p[NP];
};
using ProjBatch = AddBatch<kMaxProjBatch>;

// ---- on_pre: target[post] += w -------------------------------------------------------------
template <typename R, bool HAS_W, bool AGG, bool WARP_PREFIX, int GROUP, int NP>
__global__ void __launch_bounds__(kDeliverBlock)
deliver_add_batch_kernel(const __grid_constant__ AddBatch<NP> B,
                         const int64_t* __restrict__ clock, int k) {
  extern __shared__ int s_pref[];
  const AddDev& P = B.p[NP == 1 ? 0 : blockIdx.y];
  const int64_t ts = clock[0] + k;
  const R* __restrict__ W = static_cast<const R*>(P.w);
  const int64_t warp0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const int glane = (threadIdx.x & 31) % GROUP;
  MemberCache<R> mc;
  let_next_launch_start();
  asm volatile("" ::"l"(P.src_ring_cnt), "l"(P.src_ring_idx), "r"(P.nd), "l"(P.off), "l"(P.post),
               "l"(ts));   // in registers before the wait
  previous_launch_done();
  for_each_due_item<WARP_PREFIX, GROUP>(P, ts, warp0, nwarps, s_pref,
                                        [&](int64_t b0, int64_t b1, int64_t len, int32_t pre,
                                            int64_t) {
    member_lookup<R>(P, pre, mc);
    // kAddUnroll rounds of the bundle per pass: their loads are all issued before the first
    // atomic, so each lane keeps several independent loads in flight
    for (int64_t off = 0; off < len; off += kAddUnroll * GROUP) {
      int32_t post[kAddUnroll];
      R w[kAddUnroll];
      bool v[kAddUnroll];
#pragma unroll
      for (int u = 0; u < kAddUnroll; ++u) {
        const int64_t s = b0 + off + u * GROUP + glane;
        v[u] = s < b1;
        post[u] = v[u] ? __ldg(P.post + s) : 0;
        w[u] = mc.w;
        if constexpr (HAS_W) w[u] = v[u] ? __ldg(W + s) : (R)0;
      }
#pragma unroll
      for (int u = 0; u < kAddUnroll; ++u)
        if (off + u * GROUP < len)  // warp-uniform
          add_to_target<R, AGG>(mc.target, post[u], w[u], v[u]);
    }
  });
}

// ---- event-driven additive STDP (examples/stdp.py:125-186) --------------------------------
// Brian2 keeps w, Apre, Apost and lastupdate per synapse and decays both traces lazily from
// lastupdate to t at every event of the synapse.  A synapse's Apre changes only at its
// bundle's events and its Apost only at its target's spikes, so all synapses of one bundle
// (pre, delay) hold one Apre and all synapses of one target one Apost: the traces are kept
// once per bundle and once per target, {value at the last event, time of that event}, decayed
// over one interval from there to t, and a synapse keeps its weight alone.  (The per-synapse
// form splits the same decay at the other pathway's events, one rounding per piece.)  In
// float32 the event time is rounded to float first, as brian2cuda does
// (brian2cuda/device.py:1034-1039).
// Per event this leaves the weight's read and write, the bundle key and the trace (L1 or L2
// hits) instead of a 16-byte record's read and write: 1e4 -> 1e3 all-to-all in float32, 1e7
// weights stay in the L2 cache (40 MB against 160 MB of records).  Measured there (4.7e6
// on_post events per step): on_post 67 -> 16 us (30 us with post-grouped records), the whole
// step 73.6 -> 19.6 us (44 us with post-grouped records).
template <typename R>
struct __align__(2 * sizeof(R)) Trace {
  R a, t;
};

// -(t - since)/tau as the decay's exponent (float32: one rounding, from the double quotient).
__device__ __forceinline__ float decay_arg(double t, float since, double, double inv_tau) {
  return (float)(((double)since - t) * inv_tau);
}
__device__ __forceinline__ double decay_arg(double t, double since, double tau, double) {
  return (since - t) / tau;
}
template <typename R>
__device__ __forceinline__ R decayed(const Trace<R>& x, double t, double tau, double inv_tau) {
  return x.a * dexp(decay_arg(t, x.t, tau, inv_tau));
}

// DELAYS: a neuron has several bundles, of which some may be empty: an item without synapses is
// left before its trace is evaluated.  us per step before / after, Poisson inputs at 15 Hz, float32:
// 50,000 -> 2000 at 0.01 over 301 delays 16.8 / 15.1, 100,000 -> 1000 at 0.005 over 41 10.9 / 10.4;
// without delays the branch only holds the loads back (20,000 -> 2000 at 0.02 8.1 / 8.4).
template <typename R, bool AGG, bool WARP_PREFIX, bool DELAYS>
__global__ void __launch_bounds__(kDeliverBlock)
deliver_stdp_pre_kernel(ProjDev P, const int64_t* __restrict__ clock, int k, double dt) {
  extern __shared__ int s_pref[];
  const int64_t ts = clock[0] + k;
  const double t = (double)ts * dt;
  R* __restrict__ W = static_cast<R*>(P.stdp_w);
  R* __restrict__ T = static_cast<R*>(P.target);
  Trace<R>* __restrict__ tr_pre = static_cast<Trace<R>*>(P.tr_pre);
  const Trace<R>* __restrict__ tr_post = static_cast<const Trace<R>*>(P.tr_post);
  const double inv_pre = 1.0 / P.taupre, inv_post = 1.0 / P.taupost;
  const R dApre = (R)P.dApre, wmin = (R)P.wmin, wmax = (R)P.wmax;
  const int64_t warp0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const int lane = threadIdx.x & 31;
  let_next_launch_start();
  asm volatile("" ::"l"(P.src_ring_cnt), "l"(P.src_ring_idx), "r"(P.nd), "l"(P.off), "l"(P.post),
               "d"(t), "d"(inv_pre), "d"(inv_post));   // in registers before the wait
  previous_launch_done();
  for_each_due_item<WARP_PREFIX, 32>(P, ts, warp0, nwarps, s_pref,
                                     [&](int64_t b0, int64_t b1, int64_t len, int32_t,
                                         int64_t head_key) {
    Trace<R> p{};
    if (DELAYS) {   // (nothing reads an empty bundle's trace; its load does not wait for the bounds)
      if (head_key >= 0 && lane == 0) p = tr_pre[head_key];
      if (len == 0) return;   // the same for the whole warp
    }
    // the item's (at most kChunk) synapses, kChunk/32 per lane: every load of the lane is
    // issued before the first weight is updated (distinct weights: no ordering between them)
    static_assert(kChunk % 32 == 0, "an item is whole rounds of the warp");
    constexpr int kPer = kChunk / 32;
    R wt[kPer];
    Trace<R> q[kPer];
    int64_t at[kPer];
    int32_t post[kPer];
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
      const int64_t s = b0 + lane + 32 * u;
      const bool ok = s < b1;
      post[u] = ok ? __ldg(P.post + s) : 0;
      at[u] = ok ? (P.rec_of ? (int64_t)__ldg(P.rec_of + s) : s) : -1;
      if (ok) {
        wt[u] = W[at[u]];
        q[u] = tr_post[post[u]];
      }
    }
    // the bundle's own trace, once per event (read by on_post, which runs after this launch)
    if (head_key >= 0 && lane == 0) {
      if (!DELAYS) p = tr_pre[head_key];
      p.a = decayed(p, t, P.taupre, inv_pre) + dApre;
      p.t = (R)t;
      tr_pre[head_key] = p;
    }
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
      R w = 0;
      if (at[u] >= 0) {
        w = wt[u];
        W[at[u]] = dclip(w + decayed(q[u], t, P.taupost, inv_post), wmin, wmax);
      }
      if (P.pre_adds_weight && 32 * u < len)  // warp-uniform
        add_to_target<R, AGG>(T, post[u], w, at[u] >= 0);
    }
  });
}

// on_post: every synapse of each neuron of the target population that spiked this step,
// reached through the transposed (post-sorted) index.  Key: the type of the bundle keys.
template <typename R, typename Key>
__global__ void __launch_bounds__(kDeliverBlock)
deliver_stdp_post_kernel(ProjDev P, const int64_t* __restrict__ clock, int k, double dt) {
  const int64_t ts = clock[0] + k;
  const double t = (double)ts * dt;
  const int slot = ring_slot(ts, P.post_ring_len);
  const double inv_pre = 1.0 / P.taupre, inv_post = 1.0 / P.taupost;
  let_next_launch_start();
  asm volatile("" ::"r"(slot), "l"(P.post_off), "l"(P.key_of), "d"(t), "d"(inv_pre),
               "d"(inv_post));   // in registers before the wait
  previous_launch_done();
  const int nspk = P.post_ring_cnt[slot];
  const int32_t* spikes = P.post_ring_idx + (int64_t)slot * P.post_src_n;
  R* __restrict__ W = static_cast<R*>(P.stdp_w);
  const Trace<R>* __restrict__ tr_pre = static_cast<const Trace<R>*>(P.tr_pre);
  Trace<R>* __restrict__ tr_post = static_cast<Trace<R>*>(P.tr_post);
  const R dApost = (R)P.dApost, wmin = (R)P.wmin, wmax = (R)P.wmax;
  const int lane = threadIdx.x & 31;
  const int64_t items = (int64_t)nspk * P.post_chunks;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t it = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); it < items;
       it += warps) {
    const int sp = items <= INT32_MAX ? (int)((uint32_t)it / (uint32_t)P.post_chunks)
                                      : (int)(it / P.post_chunks);
    const int ch = (int)(it - (int64_t)sp * P.post_chunks);
    const int32_t j = spikes[sp];
    const int64_t b0 = P.post_off[j] + (int64_t)ch * kChunk;
    int64_t b1 = P.post_off[j + 1];
    if (b1 > b0 + kChunk) b1 = b0 + kChunk;
    // the lane's (up to) kChunk/32 synapses of the item, all loaded before any is updated so
    // that their loads are in flight together (distinct weights: no ordering between them)
    static_assert(kChunk % 32 == 0, "an item is whole rounds of the warp");
    constexpr int kPer = kChunk / 32;
    R wt[kPer];
    Trace<R> p[kPer];
    int64_t at[kPer];
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
      const int64_t r = b0 + lane + 32 * u;
      // post-grouped weights: weight r itself (contiguous); otherwise its synapse's
      at[u] = r < b1 ? (P.rec_of ? r : (int64_t)__ldg(P.post_syn + r)) : -1;
      if (at[u] >= 0) {
        wt[u] = W[at[u]];
        p[u] = tr_pre[__ldg(static_cast<const Key*>(P.key_of) + r)];
      }
    }
    if (ch == 0 && lane == 0) {
      Trace<R> q = tr_post[j];
      q.a = decayed(q, t, P.taupost, inv_post) + dApost;
      q.t = (R)t;
      tr_post[j] = q;
    }
#pragma unroll
    for (int u = 0; u < kPer; ++u)
      if (at[u] >= 0)
        W[at[u]] = dclip(wt[u] + decayed(p[u], t, P.taupre, inv_pre), wmin, wmax);
  }
}

// CTAs of a delivery with `group` lanes per work item: more lanes than eight leave a warp fewer items.
unsigned deliver_grid(const Proj& pr, int group) {
  const int64_t want = (pr.dev.src_n * (int64_t)pr.dev.chunks) * std::max(group / 8, 1) / 64 + 1;
  const int64_t cap = 4 * kNumSMs;
  return (unsigned)(want < cap ? want : cap);
}

template <typename R, bool HAS_W, bool AGG, int GROUP>
cudaError_t launch_add_g(const ProjBatch& B, dim3 g, bool warp_prefix, size_t smem,
                         const int64_t* clock, int k, cudaStream_t s, bool chained) {
  if (warp_prefix) smem = 0;
  if (g.y == 1) {
    const AddBatch<1> one{{B.p[0]}};
    return warp_prefix
               ? launch_kernel(deliver_add_batch_kernel<R, HAS_W, AGG, true, GROUP, 1>, g,
                               kDeliverBlock, smem, s, chained, one, clock, k)
               : launch_kernel(deliver_add_batch_kernel<R, HAS_W, AGG, false, GROUP, 1>, g,
                               kDeliverBlock, smem, s, chained, one, clock, k);
  }
  return warp_prefix
             ? launch_kernel(deliver_add_batch_kernel<R, HAS_W, AGG, true, GROUP, kMaxProjBatch>,
                             g, kDeliverBlock, smem, s, chained, B, clock, k)
             : launch_kernel(deliver_add_batch_kernel<R, HAS_W, AGG, false, GROUP, kMaxProjBatch>,
                             g, kDeliverBlock, smem, s, chained, B, clock, k);
}

// Lanes per work item: 2, 4, 8, 16 or 32.
template <typename R, bool HAS_W, bool AGG>
cudaError_t launch_add(const ProjBatch& B, dim3 g, bool wp, size_t smem, const int64_t* clock,
                       int k, cudaStream_t s, int group, bool chained) {
  if (group == 32) return launch_add_g<R, HAS_W, AGG, 32>(B, g, wp, smem, clock, k, s, chained);
  if (group == 16) return launch_add_g<R, HAS_W, AGG, 16>(B, g, wp, smem, clock, k, s, chained);
  if (group == 4) return launch_add_g<R, HAS_W, AGG, 4>(B, g, wp, smem, clock, k, s, chained);
  if (group == 2) return launch_add_g<R, HAS_W, AGG, 2>(B, g, wp, smem, clock, k, s, chained);
  return launch_add_g<R, HAS_W, AGG, 8>(B, g, wp, smem, clock, k, s, chained);
}

template <typename R>
cudaError_t launch_add_r(const ProjBatch& B, dim3 g, bool hw, bool ag, bool wp, size_t smem,
                         const int64_t* clock, int k, cudaStream_t s, int group, bool chained) {
  if (hw)
    return ag ? launch_add<R, true, true>(B, g, wp, smem, clock, k, s, group, chained)
              : launch_add<R, true, false>(B, g, wp, smem, clock, k, s, group, chained);
  return ag ? launch_add<R, false, true>(B, g, wp, smem, clock, k, s, group, chained)
            : launch_add<R, false, false>(B, g, wp, smem, clock, k, s, group, chained);
}

// ---- on_pre accumulated in the distributed shared memory of thread-block clusters -------
// One L2 atomic per event bounds the scattered delivery at high event rates.  Here every
// cluster of kClusterCtas CTAs holds a private copy of the target variables the batch adds
// into (slots of the padded target population laid end to end, one slice per CTA's shared
// memory), adds its share of the events there (remote shared-memory atomics within the
// cluster), and after a cluster barrier adds its non-zero partial sums to the targets with
// one vector atomic per four elements.  The sums are regrouped (partial sums per cluster),
// so results equal the scattered form's up to rounding.  float32 only.
constexpr int kClusterCtas = 8;

struct ClusterAcc {
  float* slot_ptr[3];            // target array of each slot
  int32_t slot_of_var[3];        // slot of variable v (v, ge, gi), -1 if none
  int32_t n_slots;
  int32_t slice;                 // floats per CTA (a multiple of 4)
  int64_t n;                     // padded target population size (a multiple of 128)
};

template <bool HAS_W, bool WARP_PREFIX, int GROUP>
__global__ void __launch_bounds__(kDeliverBlock)
deliver_cluster_kernel(const __grid_constant__ ProjBatch B,
                       const __grid_constant__ ClusterAcc A, const int64_t* __restrict__ clock,
                       int k, int pref_ints) {
  extern __shared__ __align__(16) float s_dyn[];
  int* s_pref = reinterpret_cast<int*>(s_dyn);
  float* s_acc = s_dyn + pref_ints;          // pref_ints is a multiple of 4
  cg::cluster_group cl = cg::this_cluster();
  const unsigned rank = cl.block_rank();
  for (int i = 4 * threadIdx.x; i < A.slice; i += 4 * blockDim.x)
    *reinterpret_cast<float4*>(s_acc + i) = make_float4(0.f, 0.f, 0.f, 0.f);
  cl.sync();
  const AddDev& P = B.p[blockIdx.y];
  const int64_t ts = clock[0] + k;
  const float* __restrict__ W = static_cast<const float*>(P.w);
  const int64_t warp0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const int glane = (threadIdx.x & 31) % GROUP;
  MemberCache<float> mc;
  for_each_due_item<WARP_PREFIX, GROUP>(P, ts, warp0, nwarps, s_pref,
                                        [&](int64_t b0, int64_t b1, int64_t len, int32_t pre,
                                            int64_t) {
    member_lookup<float>(P, pre, mc);
    const int v = mc.target == P.targets[0] ? 0 : (mc.target == P.targets[1] ? 1 : 2);
    const int64_t base = (int64_t)A.slot_of_var[v] * A.n;
    for (int64_t off = 0; off < len; off += kAddUnroll * GROUP) {
      int32_t post[kAddUnroll];
      float w[kAddUnroll];
      bool ok[kAddUnroll];
#pragma unroll
      for (int u = 0; u < kAddUnroll; ++u) {
        const int64_t s = b0 + off + u * GROUP + glane;
        ok[u] = s < b1;
        post[u] = ok[u] ? __ldg(P.post + s) : 0;
        w[u] = mc.w;
        if constexpr (HAS_W) w[u] = ok[u] ? __ldg(W + s) : 0.f;
      }
#pragma unroll
      for (int u = 0; u < kAddUnroll; ++u) {
        if (!ok[u]) continue;
        const int64_t flat = base + post[u];
        const unsigned r = (unsigned)(flat / A.slice);
        float* dst = cl.map_shared_rank(s_acc, r);
        atomicAdd(dst + (flat - (int64_t)r * A.slice), w[u]);
      }
    }
  });
  cl.sync();
  // this CTA's slice of the cluster's partial sums into the targets
  const int64_t lo = (int64_t)rank * A.slice;
  const int64_t total = (int64_t)A.n_slots * A.n;
  for (int i = 4 * threadIdx.x; i < A.slice; i += 4 * blockDim.x) {
    const int64_t flat = lo + i;
    if (flat >= total) break;
    const float4 x = *reinterpret_cast<const float4*>(s_acc + i);
    if (x.x == 0.f && x.y == 0.f && x.z == 0.f && x.w == 0.f) continue;
    const int slot = (int)(flat / A.n);
    atomicAdd(reinterpret_cast<float4*>(A.slot_ptr[slot] + (flat - (int64_t)slot * A.n)), x);
  }
}

// Whether a batch can accumulate in clusters, and its accumulator layout (slice <= 200 KB).
bool cluster_layout(const Proj* const* prs, int n, ClusterAcc* A) {
  if (prs[0]->dtype != B2B_F32) return false;
  uint8_t mask = 0;
  for (int i = 0; i < n; ++i) {
    if (prs[i]->dst_pop != prs[0]->dst_pop || prs[i]->dev.aggregate) return false;
    mask |= prs[i]->var_mask;
  }
  *A = ClusterAcc{};
  A->n = 0;
  int ns = 0;
  for (int v = 0; v < 3; ++v) {
    A->slot_of_var[v] = -1;
    if (mask & (1u << v)) {
      A->slot_of_var[v] = ns;
      A->slot_ptr[ns] = static_cast<float*>(prs[0]->dev.targets[v]);
      ++ns;
    }
  }
  if (mask & ~7u || ns == 0) return false;
  A->n_slots = ns;
  A->n = prs[0]->dst_n;                     // every projection targets the same population
  const int64_t total = (int64_t)ns * A->n;
  A->slice = (int32_t)(((total + 4 * kClusterCtas - 1) / (4 * kClusterCtas)) * 4);
  return (int64_t)A->slice * 4 <= 200 * 1024;
}

// Clusters of the cluster kernel that are resident together for `smem` bytes per CTA
// (queried once per shared-memory size).
unsigned resident_clusters(const void* kern, size_t smem) {
  static std::mutex mu;
  static std::vector<std::pair<size_t, int>> cache;
  std::lock_guard<std::mutex> lock(mu);
  for (auto& c : cache)
    if (c.first == smem) return (unsigned)c.second;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(kClusterCtas * 64);
  cfg.blockDim = dim3(kDeliverBlock);
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = kClusterCtas;
  attr.val.clusterDim.y = 1;
  attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  int clusters = 0;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
          cudaSuccess ||
      cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg) != cudaSuccess) {
    clusters = 0;
    cudaGetLastError();   // the refusal's error must not be reported by the next launch
  }
  cache.emplace_back(smem, clusters);
  return (unsigned)clusters;
}

template <bool HAS_W, int GROUP>
cudaError_t launch_cluster_g(const ProjBatch& B, const ClusterAcc& A, unsigned clusters,
                             bool wp, int pref_ints, size_t smem, const int64_t* clock, int k,
                             cudaStream_t s, int n) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(kClusterCtas * clusters, (unsigned)n);
  cfg.blockDim = dim3(kDeliverBlock);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = kClusterCtas;
  attr.val.clusterDim.y = 1;
  attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  if (wp) {
    auto kern = deliver_cluster_kernel<HAS_W, true, GROUP>;
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    return cudaLaunchKernelEx(&cfg, kern, B, A, clock, k, pref_ints);
  }
  auto kern = deliver_cluster_kernel<HAS_W, false, GROUP>;
  cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  return cudaLaunchKernelEx(&cfg, kern, B, A, clock, k, pref_ints);
}

template <typename R>
cudaError_t launch_stdp_pre(const ProjDev& P, unsigned grid, bool ag, bool wp, size_t smem,
                            const int64_t* clock, int k, double dt, cudaStream_t s,
                            bool chained) {
  auto launch = [&](auto kernel) {
    return launch_kernel(kernel, dim3(grid), kDeliverBlock, wp ? 0 : smem, s, chained, P, clock, k,
                         dt);
  };
  if (P.nd == 1)
    return ag ? launch(deliver_stdp_pre_kernel<R, true, true, false>)
              : launch(deliver_stdp_pre_kernel<R, false, true, false>);
  if (wp)
    return ag ? launch(deliver_stdp_pre_kernel<R, true, true, true>)
              : launch(deliver_stdp_pre_kernel<R, false, true, true>);
  return ag ? launch(deliver_stdp_pre_kernel<R, true, false, true>)
            : launch(deliver_stdp_pre_kernel<R, false, false, true>);
}

}  // namespace

AddDev add_dev(const Proj& pr) {
  const ProjDev& D = pr.dev;
  AddDev A{};
  A.src_ring_cnt = D.src_ring_cnt;
  A.src_ring_idx = D.src_ring_idx;
  A.src_n = D.src_n;
  A.src_ring_len = D.src_ring_len;
  A.dmin = D.dmin;
  A.nd = D.nd;
  A.chunks = D.chunks;
  A.src_lo = D.src_lo;
  A.src_hi = D.src_hi;
  A.off = D.off;
  A.post = D.post;
  A.w = D.w;
  for (int v = 0; v < 3; ++v) A.targets[v] = D.targets[v];
  A.n_mem = D.n_mem;
  A.mem_hi = D.mem_hi;
  A.mem_var = D.mem_var;
  A.mem_w = D.mem_w;
  A.w_scalar = D.w_scalar;
  A.in_var[0] = pr.target_var;
  A.in_w[0] = D.w_scalar;
  if (D.n_mem > 1 && D.n_mem <= kInlineMembers)
    for (int m = 0; m < D.n_mem; ++m) {
      if (m < kInlineMembers - 1) A.in_hi[m] = (int32_t)pr.mem_hi[m];
      A.in_var[m] = pr.mem_var[m];
      A.in_w[m] = D.mem_w ? pr.mem_w[m] : D.w_scalar;
    }
  return A;
}

// A work item is a bundle (up to kChunk synapses): as many lanes as keep most of them busy, so
// that short bundles leave lanes to other items and long ones need few dependent rounds.
// Measured, us per step at 2 / 4 / 8 / 16 / 32 lanes: 80 synapses per bundle (CUBA 4000) 8.81 /
// 7.28 / 6.46 / 6.00 / 5.53; 40 (1e5 -> 1e5 at 300 Hz, 4 CTAs per SM) 54.0 / 51.8 / 52.2 / 49.8 /
// 55.7; 12 (2e4 -> 3e4) 7.83 / 7.25 / 6.74 / 7.48 / 8.15; 6 (40 merged COBAHH networks, 4 CTAs
// per SM) 17.1 / 16.8 / 17.4 / 20.2 / 24.0.
int delivery_lanes(double mean_bundle) {
  return mean_bundle >= 64 ? 32 : mean_bundle >= 24 ? 16 : mean_bundle >= 8 ? 8 : 4;
}

// The pending delivery runs beside the update and, in a step of few events, is mostly latency: wide
// items spread them over more warps.  In a step of many, lanes that a short bundle leaves idle are what it
// takes longer by (deliver_pending_body has more in the quiet steps).  us per step of the chained grid at
// 4 / 8 / 16 lanes in both, at 12 and 220 Hz (LIF f32, synapses per bundle): 4000 neurons (4) 2.82 / 2.76 /
// 2.75 and 2.93 / 2.88 / 2.93, 8000 (4) - / 2.90 / 2.86 and - / 3.36 / 4.19; 20,000 (4) 2.98 / 2.90 / 2.88 and 3.3 /
// 4.4 / 5.8, (15) 3.46 / 3.03 / 2.98 and 4.8 / 4.9 / 5.9, (50) 4.66 / 3.83 / 3.33 and 11.2 / 9.7 / 10.2; 60,000
// (8) 3.42 / 3.30 / 3.30 and 5.6 / 7.2 / 9.9, (25) 4.25 / 3.78 / 3.43 and 10.7 / 11.0 / 10.9; 100,000 (4) 3.14 /
// 3.10 / 3.28 and 7.8 / 12.3 / 19.5, (15) 3.88 / 3.46 / 3.41 and 11.1 / 12.0 / 17.2, (50) 6.72 / 5.20 / 4.30 and
// 25.7 / 23.9 / 24.1; two launches of 220,000 (15) 5.27 / 4.83 / 5.04 and 17.4 / 18.9 / 25.7, 300,000 (15) 6.48 /
// 6.22 / 7.60 and 20.4 / 23.5 / 33.8, (25) 7.23 / 6.45 / 7.83 and 26.8 / 30.1 / 36.0, 700,000 (8) 8.89 / 9.24 / 9.97
// and 38.0 / 53.2 / 82.6; merged networks of 613,000 (4-5) 12.5 / 13.7 / 17.2 at their own rates.
int pending_lanes(double mean_bundle, int64_t n) {
  const bool is_long = mean_bundle >= kLongBundle;
  if (n <= 10000) return mean_bundle < 8 ? 8 : 16;
  if (n < 250000) return mean_bundle < 10 ? 4 : is_long && n < kPendingLarge ? 16 : 8;
  return is_long ? 8 : 4;
}

// Chained, a delivery's CTAs take their places while the update's still run, where one has ended
// first, and stay uneven over the SMs.  Up to here the launch hidden is worth more: STDP 1e4 -> 1e3
// (1e7 synapses) 21.2 -> 21.1 us per step, STDP 3,001 -> 257 (8e5) 9.5 -> 8.8; 1e5 -> 1e5 at 300 Hz
// (1e8) 50.6 -> 59.5.
bool chained_delivery(int64_t n_syn) { return n_syn <= (int64_t)1 << 25; }

cudaError_t launch_proj_add_batch(const Proj* const* prs, int n, const int64_t* clock, int k,
                                  cudaStream_t s, const AddTune* tune, bool chained) {
  if (n <= 0 || n > kMaxProjBatch) return cudaErrorInvalidValue;
  if (counted_in_use(prs, n, tune)) {
    cudaError_t e = cudaSuccess;
    for (int i = 0; i < n && e == cudaSuccess; ++i)
      e = launch_counted(*prs[i], clock, k, s, chained || i > 0);
    return e;
  }
  ProjBatch B{};
  unsigned grid = 1;
  int nd = 1;
  int64_t n_syn = 0;
  for (int i = 0; i < n; ++i) {
    n_syn += prs[i]->n_syn;
    B.p[i] = add_dev(*prs[i]);
    nd = std::max(nd, (int)prs[i]->dev.nd);
  }
  const bool wp = nd <= kWarpPrefixMaxDelays;
  const size_t smem = sizeof(int) * (size_t)(nd + 1);
  double mean = 0;
  int64_t most = -1;
  for (int i = 0; i < n; ++i)
    if (prs[i]->n_syn > most) {
      most = prs[i]->n_syn;
      mean = prs[i]->mean_bundle;
    }
  const int group = tune && tune->group > 0 ? tune->group : delivery_lanes(mean);
  for (int i = 0; i < n; ++i) grid = std::max(grid, deliver_grid(*prs[i], group));
  ClusterAcc A;
  if (tune && tune->cluster && cluster_layout(prs, n, &A)) {
    const int pref_ints = ((nd + 1 + 3) / 4) * 4;
    const size_t csmem = sizeof(float) * ((size_t)pref_ints + A.slice);
    const unsigned clusters =
        resident_clusters((const void*)deliver_cluster_kernel<false, true, 8>, csmem);
    if (clusters > 0) {
      const bool hw = prs[0]->dev.w != nullptr;
      switch (group) {
        case 4:
          return hw ? launch_cluster_g<true, 4>(B, A, clusters, wp, pref_ints, csmem, clock, k, s, n)
                    : launch_cluster_g<false, 4>(B, A, clusters, wp, pref_ints, csmem, clock, k, s, n);
        case 16:
          return hw ? launch_cluster_g<true, 16>(B, A, clusters, wp, pref_ints, csmem, clock, k, s, n)
                    : launch_cluster_g<false, 16>(B, A, clusters, wp, pref_ints, csmem, clock, k, s, n);
        case 32:
          return hw ? launch_cluster_g<true, 32>(B, A, clusters, wp, pref_ints, csmem, clock, k, s, n)
                    : launch_cluster_g<false, 32>(B, A, clusters, wp, pref_ints, csmem, clock, k, s, n);
        default:
          return hw ? launch_cluster_g<true, 8>(B, A, clusters, wp, pref_ints, csmem, clock, k, s, n)
                    : launch_cluster_g<false, 8>(B, A, clusters, wp, pref_ints, csmem, clock, k, s, n);
      }
    }
  }
  if (tune && tune->grid > 0) grid = (unsigned)tune->grid;
  const dim3 g(grid, (unsigned)n);
  chained = chained && chained_delivery(n_syn);
  const bool hw = prs[0]->dev.w != nullptr;
  const bool ag = prs[0]->dev.aggregate != 0;
  return prs[0]->dtype == B2B_F32
             ? launch_add_r<float>(B, g, hw, ag, wp, smem, clock, k, s, group, chained)
             : launch_add_r<double>(B, g, hw, ag, wp, smem, clock, k, s, group, chained);
}

bool add_batch_cluster_capable(const Proj* const* prs, int n) {
  ClusterAcc A;
  return n > 0 && n <= kMaxProjBatch && cluster_layout(prs, n, &A);
}

cudaError_t launch_proj_pre(const Proj& pr, const int64_t* clock, int k, double dt,
                            int32_t* status, cudaStream_t s, bool chained) {
  (void)status;
  if (pr.effect == B2B_EFFECT_ADD) {
    const Proj* one = &pr;
    return launch_proj_add_batch(&one, 1, clock, k, s, nullptr, chained);
  }
  if (pr.effect != B2B_EFFECT_STDP) return cudaErrorInvalidValue;
  const ProjDev& P = pr.dev;
  chained = chained && chained_delivery(pr.n_syn);
  const unsigned grid = deliver_grid(pr, 8);
  const bool wp = P.nd <= kWarpPrefixMaxDelays;
  const size_t smem = sizeof(int) * (size_t)(P.nd + 1);
  const bool ag = P.aggregate != 0;
  return pr.dtype == B2B_F32
             ? launch_stdp_pre<float>(P, grid, ag, wp, smem, clock, k, dt, s, chained)
             : launch_stdp_pre<double>(P, grid, ag, wp, smem, clock, k, dt, s, chained);
}

cudaError_t launch_proj_post(const Proj& pr, const int64_t* clock, int k, double dt,
                             int32_t* status, cudaStream_t s, bool chained) {
  (void)status;
  if (pr.effect != B2B_EFFECT_STDP) return cudaSuccess;
  const ProjDev& P = pr.dev;
  int64_t want = (P.post_src_n * (int64_t)P.post_chunks) / 8 + 1;
  const unsigned grid = (unsigned)(want < 4 * kNumSMs ? want : 4 * kNumSMs);
  auto launch = [&](auto kernel) {
    return launch_kernel(kernel, dim3(grid), kDeliverBlock, 0, s, chained, P, clock, k, dt);
  };
  if (wide_keys(P.src_n * (int64_t)P.nd))
    return pr.dtype == B2B_F32 ? launch(deliver_stdp_post_kernel<float, int64_t>)
                               : launch(deliver_stdp_post_kernel<double, int64_t>);
  return pr.dtype == B2B_F32 ? launch(deliver_stdp_post_kernel<float, int32_t>)
                             : launch(deliver_stdp_post_kernel<double, int32_t>);
}

}  // namespace b2b
