// Additive delivery of a heavily driven projection by counting.
//
// deliver_add_batch_kernel (propagate.cu) makes one L2 atomic per synaptic event, and the chip
// takes 1.3 to 1.5e11 of them per second to scattered float32 targets (3e6 onto 1e5 targets in
// 20.6 us), however the work is laid out.  Where every Synapses object adds one weight, an event
// need only be counted: each SM counts its share of the events per target in 16 bits of its own
// shared memory (an atomic there takes a bank's cycle), adds four neighbouring targets' counts at
// once to the sums of all SMs in L2 (one coalesced 64-bit reduction), and a second launch adds the
// weight as often as it was counted.  The additions are those the atomics would make, one by one
// in float, so the result is the same bit for bit.
//
// 1e5 -> 1e5 at 300 Hz (6e6 events per step onto two variables, 40 synapses per bundle): a step
// 49.0 -> 30.5 us.  Of the 22 us that the count takes, by a CTA's clock, 1.3 go to the prefix over
// the delays, 2 to the spikes, 3 to the bundles, 9 to the targets and their counts (34 MB of
// scattered 160-byte bundles from DRAM; without the counts themselves the reads take the same) and
// 4.5 to the sums; zeroing the counts overlaps the launch before.
#include <algorithm>

#include "delivery.cuh"

namespace b2b {
namespace {

constexpr int kCountBlock = 1024;              // one CTA per SM
// shared memory beyond half an SM's keeps a second CTA off the SM while the launch before ends
constexpr size_t kCountMinSmem = 118 * 1024;
constexpr int kListItems = 2048;                // work items listed at a time
// below the counts: the list (place, length), its end, the prefix over the delays' spikes
constexpr int kCountMaxDelays = 64;
constexpr size_t kCountSideSmem = 9 * kListItems + 16 + 4 * (kCountMaxDelays + 4);
static_assert(kChunk <= 255, "an item's length is a byte");
constexpr int kApplyBlock = 256;
constexpr int kMaxSharedBytes = 227 * 1024;

// Class (target variable) of presynaptic neuron pre.
__device__ __forceinline__ int class_of(const AddDev& P, int32_t pre) {
  int var = P.in_var[0];
#pragma unroll
  for (int m = 1; m < kInlineMembers; ++m)
    if (m < P.n_mem && pre >= P.in_hi[m - 1]) var = P.in_var[m];
  return var;
}

// CTAs [cta_lo[c], cta_lo[c + 1]) share the due items among them and count those that add into
// variable var[c].  In rounds of up to four items per thread: each thread finds its items' spikes
// and bundles (two dependent reads, all threads' together) and lists those of the class; then GROUP
// lanes take an item from the list, U reads in flight per lane and the next item's before this
// one's are counted.  Taken 32 items to a warp without the list, every warp waited for its own
// chain of reads (a step 40.2 us instead of 30.5); asking the L2 for the targets as the items are
// listed made the list slower by what the reads gained (32.6 to 35).
template <int GROUP, int U>
__global__ void __launch_bounds__(kCountBlock, 1)
count_events_kernel(const __grid_constant__ CountedDev D, const int64_t* __restrict__ clock,
                    int k) {
  extern __shared__ __align__(16) uint8_t smem[];
  constexpr int kItems = 4;                     // per thread and round
  constexpr int kGroups = kCountBlock / GROUP;
  const AddDev& P = D.add;
  const int64_t ts = clock[0] + k;
  int c = 0;
#pragma unroll
  for (int i = 1; i < 3; ++i)
    if ((int)blockIdx.x >= D.cta_lo[i]) c = i;
  const int rank = (int)blockIdx.x - D.cta_lo[c], ncta = D.cta_lo[c + 1] - D.cta_lo[c];
  const int var = D.var[c], per_round = D.per_round[c];
  const int lane = threadIdx.x & 31;
  const int grp = threadIdx.x / GROUP, glane = threadIdx.x % GROUP;
  int64_t* list_at = reinterpret_cast<int64_t*>(smem);
  uint8_t* list_len = smem + 8 * kListItems;
  int* listed = reinterpret_cast<int*>(smem + 9 * kListItems);
  int* s_pref = listed + 4;
  uint32_t* cnt = reinterpret_cast<uint32_t*>(smem + kCountSideSmem);
  uint4* cnt16 = reinterpret_cast<uint4*>(cnt);
  for (int i = threadIdx.x; i < (D.words + 1) / 2; i += kCountBlock)
    cnt16[i] = make_uint4(0, 0, 0, 0);
  if (threadIdx.x == 0) *listed = 0;
  __syncthreads();
  let_next_launch_start();
  previous_launch_done();
  const int64_t items = (int64_t)due_prefix_block(P.src_ring_cnt, P.src_ring_len, ts, P.dmin,
                                                  P.nd, P.src_lo, P.src_hi, s_pref) * P.chunks;
  const int base = ring_slot(ts, P.src_ring_len);
  // every ncta-th 32 items: the newest spikes' bundles, which no step before has brought into the
  // caches, fall to all CTAs alike
  const int64_t blocks = (items + 31) / 32;
  const int64_t end = blocks > rank ? ((blocks - rank - 1) / ncta + 1) * 32 : 0;
  auto count = [&](int32_t post) { atomicAdd(cnt + (post >> 1), 1u << ((post & 1) * 16)); };
  for (int64_t lo = 0; lo < end; lo += per_round) {
    const int here = (int)min((int64_t)per_round, end - lo);
    int32_t pre[kItems];
    int di[kItems], ch[kItems];
#pragma unroll
    for (int u = 0; u < kItems; ++u) {
      const int at = u * kCountBlock + (int)threadIdx.x;
      pre[u] = -1;
      if (u * kCountBlock >= here) continue;    // the same for the whole CTA
      const int64_t mine = lo + at;
      const int64_t it = ((mine >> 5) * ncta + rank) * 32 + (mine & 31);
      const bool have = at < here && it < items;
      const int sp = !have ? 0
                     : P.chunks == 1 ? (int)it
                     : items <= INT32_MAX ? (int)((uint32_t)it / (uint32_t)P.chunks)
                                          : (int)(it / P.chunks);
      ch[u] = have ? (int)(it - (int64_t)sp * P.chunks) : 0;
      int kk = 0;
      di[u] = find_delay_block(s_pref, P.nd, sp, &kk);
      if (have)
        pre[u] = P.src_ring_idx[(int64_t)ring_back(base, P.dmin + di[u], P.src_ring_len) * P.src_n
                                + kk];
    }
    int64_t b0[kItems], b1[kItems];
#pragma unroll
    for (int u = 0; u < kItems; ++u) {
      b0[u] = b1[u] = 0;
      if (pre[u] >= 0 && class_of(P, pre[u]) == var) {
        const int64_t key = (int64_t)pre[u] * P.nd + di[u];
        b0[u] = P.off[key] + (int64_t)ch[u] * kChunk;
        b1[u] = P.off[key + 1];
      }
    }
#pragma unroll
    for (int u = 0; u < kItems; ++u) {
      if (u * kCountBlock >= here) continue;
      const int len = (int)max((int64_t)0, min(b1[u] - b0[u], (int64_t)kChunk));
      const unsigned mine = __ballot_sync(kFull, len > 0);
      int place = 0;
      if (lane == 0 && mine) place = atomicAdd(listed, __popc(mine));
      place = __shfl_sync(kFull, place, 0) + __popc(mine & ((1u << lane) - 1));
      if (len == 0) continue;
      const int32_t* p = P.post + b0[u];
      if (place < kListItems) {
        list_at[place] = b0[u];
        list_len[place] = (uint8_t)len;
      } else {                                  // more of the class than expected
        for (int o = 0; o < len; ++o) count(__ldg(p + o));
      }
    }
    __syncthreads();
    const int n = min(*listed, kListItems);
    struct Item {
      const int32_t* p;
      int len;
      int32_t post[U];
    };
    auto load = [&](int r) {
      Item a;
      a.len = r < n ? list_len[r] : 0;
      a.p = P.post + (r < n ? list_at[r] : 0);
#pragma unroll
      for (int u = 0; u < U; ++u)
        a.post[u] = u * GROUP + glane < a.len ? __ldg(a.p + u * GROUP + glane) : -1;
      return a;
    };
    Item a = load(grp);
    for (int r = grp; r < n; r += kGroups) {
      const Item b = load(r + kGroups);
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (a.post[u] >= 0) count(a.post[u]);
      if constexpr (GROUP * U < kChunk)
        for (int o = GROUP * U + glane; o < a.len; o += GROUP) count(__ldg(a.p + o));
      a = b;
    }
    __syncthreads();
    if (threadIdx.x == 0) *listed = 0;
    __syncthreads();
  }
  __syncthreads();
  // every CTA starts elsewhere, so that few add to one word at a time (25,000 words from 148
  // CTAs: 12.4 -> 10.7 us)
  const unsigned long long* mine = reinterpret_cast<const unsigned long long*>(cnt);
  const int at = (int)((int64_t)D.words * rank / ncta);
  for (int i = threadIdx.x; i < D.words; i += kCountBlock) {
    const int j = i + at < D.words ? i + at : i + at - D.words;
    const unsigned long long v = mine[j];
    if (v) atomicAdd(D.sums[c] + j, v);
  }
}

__device__ __forceinline__ float add_once(float x, float w) {
  float r;   // as a reduction to global memory does: subnormal results are zero
  asm("add.rn.ftz.f32 %0, %1, %2;" : "=f"(r) : "f"(x), "f"(w));
  return r;
}
__device__ __forceinline__ double add_once(double x, double w) { return x + w; }

// target += w, as often as counted; the sums are zero again afterwards.
template <typename R>
__global__ void __launch_bounds__(kApplyBlock)
apply_counts_kernel(const __grid_constant__ CountedDev D) {
  const int64_t i = (int64_t)blockIdx.x * kApplyBlock + threadIdx.x;
  const int c = blockIdx.y;
  uint16_t* sum = reinterpret_cast<uint16_t*>(D.sums[c]) + i;
  R* x = static_cast<R*>(D.target[c]) + i;
  const R w = (R)D.w[c];
  previous_launch_done();
  let_next_launch_start();
  if (i >= D.n) return;
  const int n = *sum;
  if (n == 0) return;
  R v = *x;
  for (int e = 0; e < n; ++e) v = add_once(v, w);
  *x = v;
  *sum = 0;
}

// In-degrees of all targets, and their largest.
__global__ void in_degree_kernel(const int32_t* __restrict__ post, int64_t n_syn, uint32_t* deg) {
  for (int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; s < n_syn;
       s += (int64_t)gridDim.x * blockDim.x)
    atomicAdd(deg + post[s], 1u);
}
__global__ void largest_kernel(uint32_t* deg, int64_t n) {
  uint32_t m = 0;
  for (int64_t i = threadIdx.x; i < n; i += blockDim.x) m = max(m, deg[i]);
  m = __reduce_max_sync(kFull, m);
  if ((threadIdx.x & 31) == 0) atomicMax(deg + n, m);
}

size_t count_smem(int32_t words) {
  return std::max(kCountMinSmem, kCountSideSmem + 16 * (size_t)((words + 1) / 2));
}

template <int GROUP, int U>
cudaError_t launch_count(const CountedDev& D, const int64_t* clock, int k, cudaStream_t s,
                         bool chained) {
  const size_t smem = count_smem(D.words);
  // (a property of the function on this device: the same limit for every network)
  cudaError_t e = cudaFuncSetAttribute(count_events_kernel<GROUP, U>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       kMaxSharedBytes);
  if (e != cudaSuccess) return e;
  return launch_kernel(count_events_kernel<GROUP, U>, dim3(D.cta_lo[3]), kCountBlock, smem, s,
                       chained, D, clock, k);
}

}  // namespace

bool counted_in_use(const Proj* const* prs, int n, const AddTune* tune) {
  if (tune && (tune->group > 0 || tune->grid > 0 || tune->cluster)) return false;
  for (int i = 0; i < n; ++i)
    if (!prs[i]->counted_ok) return false;
  return true;
}

bool counted_fits(int64_t n_targets, int32_t n_delays) {
  const int64_t words = (n_targets + 3) / 4;
  return n_delays <= kCountMaxDelays && words < (1 << 20) && count_smem((int32_t)words) <= (size_t)kMaxSharedBytes;
}

cudaError_t largest_in_degree(const int32_t* d_post, int64_t n_syn, int64_t n_targets,
                              int64_t* largest, cudaStream_t s) {
  uint32_t* deg = nullptr;
  cudaError_t e = cudaMalloc(&deg, 4 * (size_t)(n_targets + 1));
  if (e != cudaSuccess) return e;
  uint32_t m = 0;
  e = cudaMemsetAsync(deg, 0, 4 * (size_t)(n_targets + 1), s);
  if (e == cudaSuccess) {
    in_degree_kernel<<<8 * kNumSMs, 256, 0, s>>>(d_post, n_syn, deg);
    largest_kernel<<<1, 1024, 0, s>>>(deg, n_targets);
    e = cudaMemcpyAsync(&m, deg + n_targets, 4, cudaMemcpyDeviceToHost, s);
  }
  const cudaError_t f = cudaStreamSynchronize(s);
  cudaFree(deg);
  *largest = m;
  return e != cudaSuccess ? e : f;
}

// Lanes per item narrower than deliver_add_batch_kernel's: every group has two items' reads in
// flight, and 8 lanes of 8 reads fill up better than 16 of 4 (40 synapses per bundle 30.5 against
// 32.3 us per step, 20 per bundle 21.8 against 26.0).
cudaError_t launch_counted(const Proj& pr, const int64_t* clock, int k, cudaStream_t s,
                           bool chained) {
  CountedDev D = pr.counted;
  D.add = add_dev(pr);                       // the rings and the state as they are now
  for (int c = 0; c < D.n_class; ++c) D.target[c] = D.add.targets[D.var[c]];
  cudaError_t e = pr.mean_bundle >= 64   ? launch_count<32, 4>(D, clock, k, s, chained)
                  : pr.mean_bundle >= 16 ? launch_count<8, 8>(D, clock, k, s, chained)
                                         : launch_count<8, 2>(D, clock, k, s, chained);
  if (e != cudaSuccess) return e;
  const dim3 grid((unsigned)((D.n + kApplyBlock - 1) / kApplyBlock), (unsigned)D.n_class);
  return pr.dtype == B2B_F32
             ? launch_kernel(apply_counts_kernel<float>, grid, kApplyBlock, 0, s, true, D)
             : launch_kernel(apply_counts_kernel<double>, grid, kApplyBlock, 0, s, true, D);
}

}  // namespace b2b
