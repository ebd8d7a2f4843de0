// Fused per-neuron kernels: state update + refractoriness + threshold + reset + spikespace
// compaction, one launch per population and step.
//
// The reference runs these as separate code objects, each a separate launch over all N
// neurons: `_run_kernel_<group>_stateupdater` (brian2cuda/templates/common_group.cu:108-160),
// an eventspace reset kernel (templates/threshold.cu:50-75), the thresholder that appends
// spikes with one global atomicAdd per spike (threshold.cu:19-45), and the resetter over
// the spiking indices (templates/reset.cu:3-27).  Here a thread owns E consecutive neurons:
// E = 4 for large populations (each state array read with one 128-bit access, two for
// float64), E = 1 when the population is too small to fill the GPU that way.  A warp
// compacts its spikes with shuffles and reserves its output range with a single atomicAdd on
// the step's slot of the spike-history ring (the Poisson kernel, whose every warp may have
// spikes in every step, does this per CTA instead).
//
// The reset is applied in the same pass when no synaptic effect of the population writes a
// variable the reset writes; otherwise `late_reset` defers it to a kernel that runs after
// the synaptic delivery, preserving Brian2's schedule (groups, thresholds, synapses,
// resets).
#include <algorithm>
#include <cmath>
#include <type_traits>

#include "neuron_common.cuh"
#include "pending_body.cuh"

namespace b2b {

namespace {
// Adds the input delivered during the previous step (fold buffer of variable v, the row that
// step k-1 of the chunk filled) into pack X and returns the pack's address in the buffer, to be
// cleared after the update's stores; no-op when the population has no fold buffer for v.  The
// row goes by the step's place in its chunk (both rows are empty between chunks), a launch
// argument, so its load does not wait for the clock's.
// COUNTED: the buffer holds event counts, each one addition of the group's weight.
template <typename R, int E, bool COUNTED = false>
__device__ __forceinline__ R* fold_in(const PopDev& P, int v, int k, int64_t q,
                                      Pack<R, E>& X) {
  if (!P.fold[v]) return nullptr;
  R* a = static_cast<R*>(P.fold[v]) + (int64_t)((k & 1) ^ 1) * P.n;
  const Pack<R, E> A = load_pack<R, E>(a, q);
  if constexpr (COUNTED) {
    const R w = (R)P.fold_gw[3 * group_of<E>(P, q) + v];
#pragma unroll
    for (int e = 0; e < E; ++e)
      for (int c = (int)A.x[e]; c > 0; --c) X.x[e] += w;
    return a;
  }
#pragma unroll
  for (int e = 0; e < E; ++e) X.x[e] += A.x[e];
  return a;
}

// The same from event counts (the fused step): count additions of the variable's weight one by
// one, which rounds as the delivery's own additions would; nothing to clear where no event came.
template <typename R, int E>
__device__ __forceinline__ int32_t* fold_counts(const PopDev& P, int v, int k, int64_t q,
                                                Pack<R, E>& X) {
  if (!P.fold[v]) return nullptr;
  int32_t* a = static_cast<int32_t*>(P.fold[v]) + (int64_t)((k & 1) ^ 1) * P.n + E * q;
  const R w = (R)P.fold_w[v];
  int32_t n[E];
  if constexpr (E == 2) {
    const int2 c = *reinterpret_cast<const int2*>(a);
    n[0] = c.x;
    n[1] = c.y;
  } else {
    n[0] = a[0];
  }
  int32_t any = 0;
#pragma unroll
  for (int e = 0; e < E; ++e) {
    any |= n[e];
    for (int32_t c = n[e]; c > 0; --c) X.x[e] += w;
  }
  return any ? a : nullptr;
}
template <int E>
__device__ __forceinline__ void clear_counts(int32_t* a) {
  if (!a) return;
#pragma unroll
  for (int e = 0; e < E; ++e) a[e] = 0;
}

template <typename R, int E>
__device__ __forceinline__ void fold_clear(R* a, int64_t q) {
  if (!a) return;
  Pack<R, E> z;
#pragma unroll
  for (int e = 0; e < E; ++e) z.x[e] = (R)0;
  store_pack<R, E>(a, q, z);
}

// ---- LIF, exact integration ------------------------------------------------------------
// INPUTS: the population has TimedArray or PoissonInput inputs (compiled out otherwise).
// The work of CTA `blk` of the update (blockDim.x threads, E neurons each).
// FUSED: the step's delivery is part of it (fused_step_kernel): the input pending from the step
// before comes as event counts, and the CTA's spikes go through emit(q, fl, ts, slot).
// CHAINED: the kernel may be launched chained (launch_kernel).  NEXT: the next launch may start
// after the wait rather than at the top, so that its CTAs spread over SMs that the launch before
// has left (pair_step_kernel before a delivery, STDP 3,001 -> 257: 9.06 -> 8.78 us per step).
template <typename R, int E, bool INPUTS, bool FUSED = false, bool CHAINED = false,
          bool NEXT = false, bool COUNTED = false, class Emit = int>
__device__ __forceinline__ void lif_step_body(const PopDev& P, const int64_t* __restrict__ clock,
                                              int k, double dt, int32_t* status, int64_t blk,
                                              Emit emit = 0) {
  const int64_t ts = clock[0] + k;
  const double t = (double)ts * dt;
  const double inv_dt = 1.0 / dt;
  const int slot = ring_slot(ts, P.ring_len);
  const int64_t nthr = P.n / E;
  const int64_t q = blk * blockDim.x + threadIdx.x;
  unsigned fl = 0;
  const LifDev* prm = static_cast<const LifDev*>(P.params);
  const int grp = q < nthr ? group_of<E>(P, q) : 0;
  const LifDev g = prm[grp];
  if constexpr (CHAINED) previous_launch_done();
  if constexpr (NEXT) let_next_launch_start();
  if (q < nthr) {
    const GroupInputs* gin = INPUTS ? P.inputs + grp : nullptr;
    const bool after_reset = INPUTS && gin->pin.after_reset;
    const R Vt = (R)g.Vt, Vr = (R)g.Vr;
    const bool refr = g.ref_steps >= 0;
    Pack<R, E> V = load_pack<R, E>(P.var[B2B_VAR_V], q);
    Pack<R, E> GE = load_pack<R, E>(P.var[B2B_VAR_GE], q);
    Pack<R, E> GI = load_pack<R, E>(P.var[B2B_VAR_GI], q);
    Pack<R, E> LS;
    if (refr) LS = load_pack<R, E>(P.var[B2B_VAR_LASTSPIKE], q);
    R *fge = nullptr, *fgi = nullptr;
    int32_t *cge = nullptr, *cgi = nullptr;
    if constexpr (FUSED) {
      cge = fold_counts<R, E>(P, B2B_VAR_GE, k, q, GE);
      cgi = fold_counts<R, E>(P, B2B_VAR_GI, k, q, GI);
    } else {
      fge = fold_in<R, E, COUNTED>(P, B2B_VAR_GE, k, q, GE);
      fgi = fold_in<R, E, COUNTED>(P, B2B_VAR_GI, k, q, GI);
    }
    uint32_t NRout = 0;
#pragma unroll
    for (int e = 0; e < E; ++e) {
      R ge = GE.x[e], gi = GI.x[e];
      bool nr = true;
      if (refr) nr = past_refractory(t - (double)LS.x[e], dt, inv_dt, g.ref_steps);
      R vn = lif_advance<R>(g, V.x[e], ge, gi, nr,
                            INPUTS ? timed_input<R>(gin->ta, ts, E * q + e - g.offset) : R(0));
      GE.x[e] = ge;
      GI.x[e] = gi;
      const int64_t local = E * q + e - g.offset;
      const bool valid = local < g.n;
      bool reset_now = false;
      if (g.has_threshold && valid && vn > Vt && nr) {
        nr = false;
        if (refr) LS.x[e] = (R)t;
        reset_now = g.has_reset && !P.late_reset;
        fl |= 1u << e;
      }
      // PoissonInputs act in the synapses slot: after the threshold, and before the reset
      // unless the schedule resets first
      if (reset_now && after_reset) vn = Vr;
      if (INPUTS && gin->pin.count && valid)
        add_poisson_inputs<R>(gin->pin, ts, local, vn, GE.x[e], GI.x[e]);
      if (reset_now && !after_reset) vn = Vr;
      V.x[e] = vn;
      NRout |= (nr ? 1u : 0u) << (8 * e);
    }
    store_pack<R, E>(P.var[B2B_VAR_V], q, V);
    store_pack<R, E>(P.var[B2B_VAR_GE], q, GE);
    store_pack<R, E>(P.var[B2B_VAR_GI], q, GI);
    if (refr) {
      if (fl) store_pack<R, E>(P.var[B2B_VAR_LASTSPIKE], q, LS);   // changes only on a spike
      store_flags<E>(P.var[B2B_VAR_NOT_REFRACTORY], q, NRout);
    }
    if constexpr (FUSED) {
      clear_counts<E>(cge);
      clear_counts<E>(cgi);
    } else {
      fold_clear<R, E>(fge, q);
      fold_clear<R, E>(fgi, q);
    }
  }
  if constexpr (FUSED) emit(q, fl, ts, slot);
  else emit_spikes_warp<E>(P, q, fl, ts, slot, status);
  clear_next_slot(P, ts, blk);
}

template <typename R, int E, bool INPUTS, bool COUNTED>
__global__ void __launch_bounds__(kBlock)
lif_step_kernel(PopDev P, const int64_t* __restrict__ clock, int k, double dt,
                int32_t* status) {
  lif_step_body<R, E, INPUTS, false, false, false, COUNTED>(P, clock, k, dt, status, blockIdx.x);
}

// ---- Hodgkin-Huxley (COBAHH), exponential Euler (hh_advance) ------------------------
template <typename R, int E, bool INPUTS, bool FUSED = false, bool CHAINED = false,
          bool NEXT = false, bool COUNTED = false, class Emit = int>
__device__ __forceinline__ void hh_step_body(const PopDev& P, const int64_t* __restrict__ clock,
                                             int k, double dt, int32_t* status, int64_t blk,
                                             Emit emit = 0) {
  const int64_t ts = clock[0] + k;
  const double t = (double)ts * dt;
  const double inv_dt = 1.0 / dt;
  const int slot = ring_slot(ts, P.ring_len);
  const int64_t nthr = P.n / E;
  const int64_t q = blk * blockDim.x + threadIdx.x;
  unsigned fl = 0;
  const HhDev* prm = static_cast<const HhDev*>(P.params);
  const int grp = q < nthr ? group_of<E>(P, q) : 0;
  const HhRun<R> g = hh_run(prm[grp], R());
  if constexpr (CHAINED) previous_launch_done();
  if constexpr (NEXT) let_next_launch_start();
  if (q < nthr) {
    const GroupInputs* gin = INPUTS ? P.inputs + grp : nullptr;
    const R Vthr = (R)g.Vthr, dtR = (R)dt;
    const bool refr = g.ref_steps >= 0;
    Pack<R, E> V = load_pack<R, E>(P.var[B2B_VAR_V], q);
    Pack<R, E> M = load_pack<R, E>(P.var[B2B_VAR_M], q);
    Pack<R, E> H = load_pack<R, E>(P.var[B2B_VAR_H], q);
    Pack<R, E> N = load_pack<R, E>(P.var[B2B_VAR_N], q);
    Pack<R, E> GE = load_pack<R, E>(P.var[B2B_VAR_GE], q);
    Pack<R, E> GI = load_pack<R, E>(P.var[B2B_VAR_GI], q);
    Pack<R, E> LS;
    if (refr) LS = load_pack<R, E>(P.var[B2B_VAR_LASTSPIKE], q);
    R *fge = nullptr, *fgi = nullptr;
    int32_t *cge = nullptr, *cgi = nullptr;
    if constexpr (FUSED) {
      cge = fold_counts<R, E>(P, B2B_VAR_GE, k, q, GE);
      cgi = fold_counts<R, E>(P, B2B_VAR_GI, k, q, GI);
    } else {
      fge = fold_in<R, E, COUNTED>(P, B2B_VAR_GE, k, q, GE);
      fgi = fold_in<R, E, COUNTED>(P, B2B_VAR_GI, k, q, GI);
    }
    uint32_t NRout = 0;
#pragma unroll
    for (int e = 0; e < E; ++e) {
      bool nr = true;
      if (refr) nr = past_refractory(t - (double)LS.x[e], dt, inv_dt, g.ref_steps);
      const int64_t local = E * q + e - g.offset;
      R vn = hh_advance<R>(g, V.x[e], M.x[e], H.x[e], N.x[e], GE.x[e], GI.x[e], dtR,
                           INPUTS ? timed_input<R>(gin->ta, ts, local) : R(0));
      const bool valid = local < g.n;
      if (valid && vn > Vthr && nr) {
        nr = false;
        if (refr) LS.x[e] = (R)t;
        fl |= 1u << e;
      }
      if (INPUTS && gin->pin.count && valid)
        add_poisson_inputs<R>(gin->pin, ts, local, vn, GE.x[e], GI.x[e]);
      V.x[e] = vn;
      NRout |= (nr ? 1u : 0u) << (8 * e);
    }
    store_pack<R, E>(P.var[B2B_VAR_V], q, V);
    store_pack<R, E>(P.var[B2B_VAR_M], q, M);
    store_pack<R, E>(P.var[B2B_VAR_H], q, H);
    store_pack<R, E>(P.var[B2B_VAR_N], q, N);
    store_pack<R, E>(P.var[B2B_VAR_GE], q, GE);
    store_pack<R, E>(P.var[B2B_VAR_GI], q, GI);
    if (refr) {
      if (fl) store_pack<R, E>(P.var[B2B_VAR_LASTSPIKE], q, LS);   // changes only on a spike
      store_flags<E>(P.var[B2B_VAR_NOT_REFRACTORY], q, NRout);
    }
    if constexpr (FUSED) {
      clear_counts<E>(cge);
      clear_counts<E>(cgi);
    } else {
      fold_clear<R, E>(fge, q);
      fold_clear<R, E>(fgi, q);
    }
  }
  if constexpr (FUSED) emit(q, fl, ts, slot);
  else emit_spikes_warp<E>(P, q, fl, ts, slot, status);
  clear_next_slot(P, ts, blk);
}

// The same with a neuron's v, m, h and n in four warps of the CTA (warp 4 g + r: variable r of the
// CTA's neurons 32 g .. 32 g + 31): in a population that does not fill the GPU the update is one
// thread's chain of exponentials and quotients, and the four equations are independent given the
// state at the start of the step.  A barrier between the loads and the stores keeps that state.
// Float64, us per step of the update alone, one thread per neuron / here: 4000 neurons 4.12 / 2.89,
// 8000 4.24 / 3.09, 20,000 4.48 / 3.52, 40,000 4.92 / 5.33 (the added warps are work there);
// float32, whose hardware exponentials are short, 4000 neurons 2.17 / 2.33, so it is not used.
template <typename R>
__device__ __forceinline__ int64_t split_neuron(int64_t blk) {
  return blk * (blockDim.x >> 2) + 32 * (threadIdx.x >> 7) + (threadIdx.x & 31);
}
template <typename R, bool FUSED = false, bool CHAINED = false, bool NEXT = false,
          class Emit = int>
__device__ __forceinline__ void hh_split_body(const PopDev& P, const int64_t* __restrict__ clock,
                                              int k, double dt, int32_t* status, int64_t blk,
                                              Emit emit = 0) {
  const int64_t ts = clock[0] + k;
  const int slot = ring_slot(ts, P.ring_len);
  const int role = (threadIdx.x >> 5) & 3;
  const int64_t q = split_neuron<R>(blk);
  const bool mine = q < P.n;
  const R dtR = (R)dt;
  HhRun<R> g{};
  if (mine) g = hh_run(static_cast<const HhDev*>(P.params)[group_of<1>(P, q)], R());
  if constexpr (CHAINED) previous_launch_done();
  if constexpr (NEXT) let_next_launch_start();
  // the state at the start of the step: all of it for the membrane's warp (role 0), v and its own
  // gate for the others
  R v = 0, m = 0, h = 0, n = 0, ls = 0, x = 0;
  R* const X =
      static_cast<R*>(P.var[role == 1 ? B2B_VAR_M : role == 2 ? B2B_VAR_H : B2B_VAR_N]);
  Pack<R, 1> GE{}, GI{};
  R *fge = nullptr, *fgi = nullptr;
  int32_t *cge = nullptr, *cgi = nullptr;
  if (mine) {
    v = static_cast<const R*>(P.var[B2B_VAR_V])[q];
    if (role == 0) {
      m = static_cast<const R*>(P.var[B2B_VAR_M])[q];
      h = static_cast<const R*>(P.var[B2B_VAR_H])[q];
      n = static_cast<const R*>(P.var[B2B_VAR_N])[q];
      GE = load_pack<R, 1>(P.var[B2B_VAR_GE], q);
      GI = load_pack<R, 1>(P.var[B2B_VAR_GI], q);
      ls = static_cast<const R*>(P.var[B2B_VAR_LASTSPIKE])[q];
      if constexpr (FUSED) {
        cge = fold_counts<R, 1>(P, B2B_VAR_GE, k, q, GE);
        cgi = fold_counts<R, 1>(P, B2B_VAR_GI, k, q, GI);
      } else {
        fge = fold_in<R, 1>(P, B2B_VAR_GE, k, q, GE);
        fgi = fold_in<R, 1>(P, B2B_VAR_GI, k, q, GI);
      }
    } else {
      x = X[q];
    }
  }
  __syncthreads();   // every thread of the CTA, whatever its role
  unsigned fl = 0;
  if (mine && role == 0) {
    const double t = (double)ts * dt;
    const bool refr = g.ref_steps >= 0;
    bool nr = true;
    if (refr) nr = past_refractory(t - (double)ls, dt, 1.0 / dt, g.ref_steps);
    const R vn = hh_membrane<R>(g, v, m, h, n, GE.x[0], GI.x[0], dtR);
    if (q - g.offset < g.n && vn > (R)g.Vthr && nr) {
      nr = false;
      if (refr) static_cast<R*>(P.var[B2B_VAR_LASTSPIKE])[q] = (R)t;
      fl = 1u;
    }
    static_cast<R*>(P.var[B2B_VAR_V])[q] = vn;
    static_cast<R*>(P.var[B2B_VAR_GE])[q] = (R)g.De * GE.x[0];
    static_cast<R*>(P.var[B2B_VAR_GI])[q] = (R)g.Di * GI.x[0];
    if (refr) static_cast<uint8_t*>(P.var[B2B_VAR_NOT_REFRACTORY])[q] = nr ? 1 : 0;
    if constexpr (FUSED) {
      clear_counts<1>(cge);
      clear_counts<1>(cgi);
    } else {
      fold_clear<R, 1>(fge, q);
      fold_clear<R, 1>(fgi, q);
    }
  } else if (mine) {
    if (role == 1) x = hh_gate_m<R>((R)g.VT, v, x, dtR);
    else if (role == 2) x = hh_gate_h<R>((R)g.VT, v, x, dtR);
    else x = hh_gate_n<R>((R)g.VT, v, x, dtR);
    X[q] = x;
  }
  if constexpr (FUSED) emit(q, fl, ts, slot);
  else emit_spikes_warp<1>(P, q, fl, ts, slot, status);
  clear_next_slot(P, ts, blk);
}

template <typename R>
__global__ void __launch_bounds__(kBlock)
hh_split_kernel(PopDev P, const int64_t* __restrict__ clock, int k, double dt, int32_t* status) {
  hh_split_body<R>(P, clock, k, dt, status, blockIdx.x);
}

template <typename R, int E, bool INPUTS, bool COUNTED>
__global__ void __launch_bounds__(kBlock)
hh_step_kernel(PopDev P, const int64_t* __restrict__ clock, int k, double dt,
               int32_t* status) {
  hh_step_body<R, E, INPUTS, false, false, false, COUNTED>(P, clock, k, dt, status, blockIdx.x);
}

// ---- one launch per step (nets of the two-launch form, pending.cu) --------------------
// The update of step t and the delivery of step t into the pending input are independent
// (pending.cu); here they are one grid: CTAs [0, n_upd) do the per-step update (one neuron
// per thread, folding in the input pending from step t-1), the CTAs after them deliver the
// bundles due at step t into acc[t & 1] (t counted from the chunk's start).  Consecutive steps are consecutive launches on one
// stream, so one launch boundary orders step t+1 after both halves of step t, where the two
// concurrent launches need a boundary each and dependencies across two streams.
// E = 0: a HH neuron's variables in four warps (hh_split_body).
template <typename R, int KIND, int E, int GROUP, int NP>
__global__ void __launch_bounds__(kBlock, E <= 1 ? (sizeof(R) == 4 ? 5 : 4) : 3)
one_launch_step_kernel(const __grid_constant__ PopDev U,
                       const __grid_constant__ PendingArgs<NP> F,
                       const int64_t* __restrict__ clock, int k, double dt, int32_t* status,
                       int n_upd) {
  // chained launches (programmatic dependent launch): the next step's CTAs come in as this one's
  // leave, and each reads its parameters, the clock and its group's constants before it waits for
  // the previous step's grid to complete; without that launch attribute both are no-ops
  let_next_launch_start();
  if ((int)blockIdx.x < n_upd) {
    if constexpr (E == 0)
      hh_split_body<R, false, true>(U, clock, k, dt, status, blockIdx.x);
    else if constexpr (KIND == KIND_HH)
      hh_step_body<R, E, false, false, true>(U, clock, k, dt, status, blockIdx.x);
    else
      lif_step_body<R, E, false, false, true>(U, clock, k, dt, status, blockIdx.x);
  } else {
    deliver_pending_body<R, true, GROUP, NP, true>(F, clock, k, (int64_t)blockIdx.x - n_upd,
                                             (int64_t)gridDim.x - n_upd, nullptr);
  }
}

// use(kernel, projections its parameters hold) with the one-launch kernel of a population at e
// neurons per thread (0: four threads per neuron), `group` lanes per work item and n_proj projections.
template <typename R, int KIND, int E, class Use>
cudaError_t with_one_launch_e(int group, int n_proj, Use use) {
  auto pick = [&](auto lanes) {
    constexpr int G = decltype(lanes)::value;
    return n_proj == 1 ? use(one_launch_step_kernel<R, KIND, E, G, 1>,
                             std::integral_constant<int, 1>{})
                       : use(one_launch_step_kernel<R, KIND, E, G, kMaxProjBatch>,
                             std::integral_constant<int, kMaxProjBatch>{});
  };
  if (group == 16) return pick(std::integral_constant<int, 16>{});
  if (group == 4) return pick(std::integral_constant<int, 4>{});
  if (group == 2) return pick(std::integral_constant<int, 2>{});
  return pick(std::integral_constant<int, 8>{});
}
template <class Use>
cudaError_t with_one_launch(const Pop& pop, int e, int group, int n_proj, Use use) {
  const bool f32 = pop.dtype == B2B_F32;
  if (pop.kind == KIND_HH) {
    if (e == 0) return with_one_launch_e<double, KIND_HH, 0>(group, n_proj, use);
    if (e == 2)
      return f32 ? with_one_launch_e<float, KIND_HH, 2>(group, n_proj, use)
                 : with_one_launch_e<double, KIND_HH, 2>(group, n_proj, use);
    return f32 ? with_one_launch_e<float, KIND_HH, 1>(group, n_proj, use)
               : with_one_launch_e<double, KIND_HH, 1>(group, n_proj, use);
  }
  if (e == 2)
    return f32 ? with_one_launch_e<float, KIND_LIF, 2>(group, n_proj, use)
               : with_one_launch_e<double, KIND_LIF, 2>(group, n_proj, use);
  return f32 ? with_one_launch_e<float, KIND_LIF, 1>(group, n_proj, use)
             : with_one_launch_e<double, KIND_LIF, 1>(group, n_proj, use);
}

// ---- update and delivery of a step without delays as one launch ------------------------
// Synapses without delays deliver the step's own spikes, so the per-step form runs the update
// and then a delivery launch that waits for it.  Where a variable's events all carry one
// weight, counting them separates the two: a CTA that finds spikes among its neurons adds 1 to
// the targets' counts for this step (row k & 1) as soon as it has updated them, whether the
// targets' own CTAs have updated theirs or not, and the update of the next step adds the weight
// count times before it integrates.  The additions and their order per target are those of the
// two launches, so the state is the same bit for bit.  Between chunks the last step's counts are
// added in (fold_counts_kernel).  CUBA 4000, float64: 6.1 -> 3.3 us per step, the launches chained
// (unchained 3.8, and 4.0 with the bundle bounds and member tables loaded after the spike).
//
// SHARE: a bundle longer than one round of its warp's loads (kFusedAlone) goes on a list in shared
// memory, which all warps of the CTA work off after the update.  Walked by its own warp alone / shared,
// us per step: LIF f32 4000 with 1000 synapses per neuron at 12 Hz 6.35 / 4.19, at 220 Hz 12.9 / 7.6;
// 100,000 with 40 and 10 neurons of 100,000 9.1 / 5.2.
constexpr int kFusedListed = 128;
template <typename R, int KIND, int E, bool SHARE>
__global__ void __launch_bounds__(kBlock)
fused_step_kernel(const __grid_constant__ PopDev U, const __grid_constant__ FusedDev F,
                  const int64_t* __restrict__ clock, int k, double dt, int32_t* status) {
  constexpr int kMine = E > 0 ? E : 1;          // neurons per thread
  constexpr int kAhead = 2;                     // projections whose bundle bounds are loaded ahead
  let_next_launch_start();
  struct Listed {
    const int32_t* post;
    int32_t len, var;
  };
  __shared__ Listed s_list[SHARE ? kFusedListed : 1];
  __shared__ int s_listed;
  if constexpr (SHARE) {
    if (threadIdx.x == 0) s_listed = 0;
    __syncthreads();
  }
  // the bundle bounds of this thread's neurons are loaded with its group's constants, so that a
  // spike's delivery starts at its targets
  const int64_t q0 = E > 0 ? (int64_t)blockIdx.x * blockDim.x + threadIdx.x
                           : split_neuron<R>(blockIdx.x);
  int64_t off[kAhead][kMine + 1];
#pragma unroll
  for (int p = 0; p < kAhead; ++p)
#pragma unroll
    for (int e = 0; e <= kMine; ++e)
      off[p][e] = p < F.n_proj && q0 < U.n / kMine ? __ldg(F.proj[p].off + kMine * q0 + e) : 0;
  // every warp delivers its own spikes, one after the other, its lanes over a bundle's targets
  auto deliver = [&](int64_t q, unsigned fl) {
    const int lane = threadIdx.x & 31;
    const int64_t row = (int64_t)(k & 1) * U.n;
#pragma unroll
    for (int e = 0; e < kMine; ++e) {
      for (unsigned m = __ballot_sync(kFull, (fl >> e) & 1u); m; m &= m - 1) {
        const int src = __ffs(m) - 1;
        const int32_t pre = (int32_t)(kMine * __shfl_sync(kFull, q, src) + e);
        for (int p = 0; p < F.n_proj; ++p) {
          const ProjDev& J = F.proj[p];
          int64_t b0, b1;
          if (p < kAhead) {
            b0 = __shfl_sync(kFull, p == 0 ? off[0][e] : off[1][e], src);
            b1 = __shfl_sync(kFull, p == 0 ? off[0][e + 1] : off[1][e + 1], src);
          } else {
            b0 = __ldg(J.off + pre);
            b1 = __ldg(J.off + pre + 1);
          }
          if (b0 == b1) continue;
          int var = F.var[p][0];
          if (J.n_mem > kFusedMembers) {
            var = J.mem_var[member_of(J, pre)];
          } else {
#pragma unroll
            for (int mm = 1; mm < kFusedMembers; ++mm)
              if (mm < J.n_mem && pre >= F.hi[p][mm - 1]) var = F.var[p][mm];
          }
          int32_t* c = F.cnt[var] + row;
          if (SHARE && b1 - b0 > kFusedAlone) {
            int at = 0;
            if (lane == 0) at = atomicAdd(&s_listed, 1);
            at = __shfl_sync(kFull, at, 0);
            if (at < kFusedListed) {   // (a full list: the warp adds by itself)
              if (lane == 0) s_list[at] = {J.post + b0, (int32_t)(b1 - b0), var};
              continue;
            }
          }
          // four rounds' targets are loaded before their additions
          for (int64_t s = b0 + lane; s < b1; s += 128) {
            int32_t post[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) post[u] = s + 32 * u < b1 ? __ldg(J.post + s + 32 * u) : -1;
#pragma unroll
            for (int u = 0; u < 4; ++u)
              if (post[u] >= 0) atomicAdd(c + post[u], 1);
          }
        }
      }
    }
  };
  auto emit = [&](int64_t q, unsigned fl, int64_t ts, int slot) {
    emit_spikes_warp<kMine>(U, q, fl, ts, slot, status, [&]() { deliver(q, fl); });
  };
  if constexpr (E == 0)
    hh_split_body<R, true, true>(U, clock, k, dt, status, blockIdx.x, emit);
  else if constexpr (KIND == KIND_HH)
    hh_step_body<R, E, false, true, true>(U, clock, k, dt, status, blockIdx.x, emit);
  else
    lif_step_body<R, E, false, true, true>(U, clock, k, dt, status, blockIdx.x, emit);
  if constexpr (SHARE) {
    __syncthreads();
    const int listed = min(s_listed, kFusedListed);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const int64_t row = (int64_t)(k & 1) * U.n;
    for (int i = 0; i < listed; ++i) {
      const Listed b = s_list[i];
      int32_t* c = F.cnt[b.var] + row;
      // the bundles' pieces of 128 targets start at another warp each; two pieces' targets are
      // loaded before their additions
      const int first = (warp + i) % warps * 128 + lane, ahead = warps * 128;
      for (int s = first; s < b.len; s += 2 * ahead) {
        int32_t post[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const int at = s + 32 * (u & 3) + (u >> 2) * ahead;
          post[u] = at < b.len ? __ldg(b.post + at) : -1;
        }
#pragma unroll
        for (int u = 0; u < 8; ++u)
          if (post[u] >= 0) atomicAdd(c + post[u], 1);
      }
    }
  }
}

// Adds the counts of the chunk's last step (row `row`) into the target variables.
template <typename R>
__global__ void fold_counts_kernel(const __grid_constant__ PopDev U, int row) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int v = B2B_VAR_GE; v <= B2B_VAR_GI; ++v) {
    if (!U.fold[v]) continue;
    R* X = static_cast<R*>(U.var[v]);
    for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < U.n; q += stride) {
      Pack<R, 1> x{{X[q]}};
      if (int32_t* a = fold_counts<R, 1>(U, v, row ^ 1, q, x)) {
        X[q] = x.x[0];
        a[0] = 0;
      }
    }
  }
}

template <typename R, int KIND, int E>
cudaError_t launch_fused_e(const PopDev& U, const FusedDev& F, unsigned grid, int block,
                           bool chained, const int64_t* clock, int k, double dt, int32_t* status,
                           cudaStream_t s) {
  return F.share ? launch_kernel(fused_step_kernel<R, KIND, E, true>, dim3(grid), block, 0, s,
                                 chained, U, F, clock, k, dt, status)
                 : launch_kernel(fused_step_kernel<R, KIND, E, false>, dim3(grid), block, 0, s,
                                 chained, U, F, clock, k, dt, status);
}
template <typename R, int KIND>
cudaError_t launch_fused_rk(const PopDev& U, const FusedDev& F, int e, unsigned grid, int block,
                            bool chained, const int64_t* clock, int k, double dt,
                            int32_t* status, cudaStream_t s) {
  if constexpr (KIND == KIND_HH && sizeof(R) == 8)
    if (e == 0)
      return launch_fused_e<R, KIND, 0>(U, F, grid, block, chained, clock, k, dt, status, s);
  if (e == 2)
    return launch_fused_e<R, KIND, 2>(U, F, grid, block, chained, clock, k, dt, status, s);
  return launch_fused_e<R, KIND, 1>(U, F, grid, block, chained, clock, k, dt, status, s);
}

// Large HH populations: a persistent grid (resident CTAs only) walks the population in
// strides, and every thread loads the state of its next four neurons before it updates the
// current four, so the loads of one pack overlap the arithmetic of the previous one.  The
// per-neuron arithmetic is hh_step_kernel's.
template <typename R>
struct HhPack {
  Pack<R, 4> V, M, H, N, GE, GI, LS;
  int grp;
};

// lastspike is loaded whatever the group's refractoriness (every HH population holds it):
// deciding on the group's flag first would make the prefetch wait for the group id and the
// group's constants, two dependent loads, when a population holds many groups.
template <typename R>
__device__ __forceinline__ void hh_pack_load(const PopDev& P, int64_t q, HhPack<R>& s) {
  s.grp = group_of<4>(P, q);
  s.V = load_pack<R, 4>(P.var[B2B_VAR_V], q);
  s.M = load_pack<R, 4>(P.var[B2B_VAR_M], q);
  s.H = load_pack<R, 4>(P.var[B2B_VAR_H], q);
  s.N = load_pack<R, 4>(P.var[B2B_VAR_N], q);
  s.GE = load_pack<R, 4>(P.var[B2B_VAR_GE], q);
  s.GI = load_pack<R, 4>(P.var[B2B_VAR_GI], q);
  s.LS = load_pack<R, 4>(P.var[B2B_VAR_LASTSPIKE], q);
}

template <typename R, bool INPUTS, bool COUNTED>
__global__ void __launch_bounds__(kBlock, 2)
hh_stream_kernel(PopDev P, const int64_t* __restrict__ clock, int k, double dt,
                 int32_t* status) {
  const int64_t ts = clock[0] + k;
  const double t = (double)ts * dt;
  const double inv_dt = 1.0 / dt;
  const int slot = ring_slot(ts, P.ring_len);
  const int64_t nthr = P.n / 4;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  const int64_t iters = (nthr + stride - 1) / stride;   // the same for every thread
  const HhDev* prm = static_cast<const HhDev*>(P.params);
  const R dtR = (R)dt;
  int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  HhPack<R> cur;
  if (q < nthr) hh_pack_load<R>(P, q, cur);
  for (int64_t it = 0; it < iters; ++it, q += stride) {
    HhPack<R> nxt;
    if (q + stride < nthr) hh_pack_load<R>(P, q + stride, nxt);
    unsigned fl = 0;
    if (q < nthr) {
      const HhRun<R> g = hh_run(prm[cur.grp], R());
      const GroupInputs* gin = INPUTS ? P.inputs + cur.grp : nullptr;
      const bool refr = g.ref_steps >= 0;
      R* fge = fold_in<R, 4, COUNTED>(P, B2B_VAR_GE, k, q, cur.GE);
      R* fgi = fold_in<R, 4, COUNTED>(P, B2B_VAR_GI, k, q, cur.GI);
      uint32_t NRout = 0;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        bool nr = true;
        if (refr) nr = past_refractory(t - (double)cur.LS.x[e], dt, inv_dt, g.ref_steps);
        const int64_t local = 4 * q + e - g.offset;
        R vn = hh_advance<R>(g, cur.V.x[e], cur.M.x[e], cur.H.x[e], cur.N.x[e],
                             cur.GE.x[e], cur.GI.x[e], dtR,
                             INPUTS ? timed_input<R>(gin->ta, ts, local) : R(0));
        const bool valid = local < g.n;
        if (valid && vn > (R)g.Vthr && nr) {
          nr = false;
          if (refr) cur.LS.x[e] = (R)t;
          fl |= 1u << e;
        }
        if (INPUTS && gin->pin.count && valid)
          add_poisson_inputs<R>(gin->pin, ts, local, vn, cur.GE.x[e], cur.GI.x[e]);
        cur.V.x[e] = vn;
        NRout |= (nr ? 1u : 0u) << (8 * e);
      }
      store_pack<R, 4>(P.var[B2B_VAR_V], q, cur.V);
      store_pack<R, 4>(P.var[B2B_VAR_M], q, cur.M);
      store_pack<R, 4>(P.var[B2B_VAR_H], q, cur.H);
      store_pack<R, 4>(P.var[B2B_VAR_N], q, cur.N);
      store_pack<R, 4>(P.var[B2B_VAR_GE], q, cur.GE);
      store_pack<R, 4>(P.var[B2B_VAR_GI], q, cur.GI);
      if (refr) {
        if (fl) store_pack<R, 4>(P.var[B2B_VAR_LASTSPIKE], q, cur.LS);   // changes on a spike
        store_flags<4>(P.var[B2B_VAR_NOT_REFRACTORY], q, NRout);
      }
      fold_clear<R, 4>(fge, q);
      fold_clear<R, 4>(fgi, q);
    }
    emit_spikes_warp<4>(P, q, fl, ts, slot, status);
    cur = nxt;
  }
  clear_next_slot(P, ts);
}

// ---- PoissonGroup: spike when u < rate*dt, u read in place from the bulk buffer ---------
// (the numbers of a chunk are drawn before it: they are read ahead of the previous launch's end)
template <typename R, int E, bool INPUTS>
__device__ __forceinline__ void poisson_step_body(const PopDev& P,
                                                  const int64_t* __restrict__ clock, int k,
                                                  double dt, int32_t* status, int64_t blk) {
  const int64_t ts = clock[0] + k;
  const int slot = ring_slot(ts, P.ring_len);
  const int64_t nthr = P.n / E;
  const int64_t q = blk * blockDim.x + threadIdx.x;
  unsigned fl = 0;
  if (q < nthr) {
    const PoissonDev* prm = static_cast<const PoissonDev*>(P.params);
    const int grp = group_of<E>(P, q);
    const PoissonDev g = prm[grp];
    const GroupInputs* gin = INPUTS ? P.inputs + grp : nullptr;
    const R thr = (R)g.p_spike;
    const R* row = static_cast<const R*>(P.rng) + (int64_t)k * P.n;
    Pack<R, E> U = load_pack<R, E>(row, q);
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const int64_t local = E * q + e - g.offset;
      const bool valid = local < g.n;
      // a TimedArray gives the rate in Hz (PoissonGroup(rates='ta(t)')): u < rate dt
      const R th = INPUTS && gin->ta.val
                       ? (R)((double)timed_input<R>(gin->ta, ts, local) * dt) : thr;
      if (valid && U.x[e] < th) fl |= 1u << e;
    }
  }
  previous_launch_done();
  let_next_launch_start();
  emit_spikes<E>(P, q, fl, ts, slot, status);
  clear_next_slot(P, ts, blk);
}

template <typename R, int E, bool INPUTS>
__global__ void __launch_bounds__(kBlock)
poisson_step_kernel(PopDev P, const int64_t* __restrict__ clock, int k, double dt,
                    int32_t* status) {
  poisson_step_body<R, E, INPUTS>(P, clock, k, dt, status, blockIdx.x);
}

// ---- SpikeGeneratorGroup: entries sorted by step, one CTA ---------------------------------
// Entries of the sorted a[0, n) below key, by a whole warp: 32 probes per round, so that 1e6
// entries take 4 dependent loads instead of a binary search's 20.
__device__ __forceinline__ int64_t warp_lower_bound(const int64_t* __restrict__ a, int64_t n,
                                                    int64_t key) {
  const int lane = threadIdx.x & 31;
  int64_t lo = 0, hi = n;                       // the answer lies in [lo, hi]
  while (lo < hi) {                             // warp-uniform
    const int64_t step = (hi - lo + 31) / 32;
    const int64_t at = lo + lane * step;
    const int below = __popc(__ballot_sync(kFull, at < hi && a[at] < key));
    if (below == 0) return lo;
    hi = min(hi, lo + below * step);
    lo += (below - 1) * step + 1;
  }
  return lo;
}

__device__ __forceinline__ void spikegen_step_body(const PopDev& P,
                                                   const int64_t* __restrict__ clock, int k,
                                                   int32_t* status) {
  const int64_t ts = clock[0] + k;
  const int slot = ring_slot(ts, P.ring_len);
  __shared__ int64_t s_bound[2];
  __shared__ unsigned long long s_mbase;
  if (threadIdx.x < 64) {
    // with a period, step ts emits the entries of bin ts mod period
    // (brian2cuda/templates/spikegenerator.cu:42-49); one warp per bound
    const int64_t bin = P.sg_period > 0 ? ts % P.sg_period : ts;
    const int64_t b = warp_lower_bound(P.sg_step, P.sg_n, bin + (threadIdx.x >> 5));
    if ((threadIdx.x & 31) == 0) s_bound[threadIdx.x >> 5] = b;
  }
  __syncthreads();
  previous_launch_done();
  let_next_launch_start();
  const int64_t s_lo = s_bound[0], cnt = s_bound[1] - s_bound[0];
  if (threadIdx.x == 0) {
    P.ring_cnt[slot] = (int)cnt;
    P.ring_cnt[ring_slot(ts + 1, P.ring_len)] = 0;
    if (P.mon_cnt) s_mbase = atomicAdd(P.mon_cnt, (unsigned long long)cnt);
  }
  __syncthreads();
  int32_t* out = P.ring_idx + (int64_t)slot * P.n;
  for (int64_t r = threadIdx.x; r < cnt; r += blockDim.x) {
    const int32_t idx = P.sg_idx[s_lo + r];
    out[r] = idx;
    if (P.mon_cnt) {
      const unsigned long long mp = s_mbase + (unsigned long long)r;
      if (mp < (unsigned long long)P.mon_cap) {
        P.mon_idx[mp] = idx;
        P.mon_step[mp] = ts;
      } else {
        set_status(status, B2B_ERR_QUEUE_OVERFLOW);
      }
    }
  }
}

__global__ void spikegen_step_kernel(PopDev P, const int64_t* __restrict__ clock, int k,
                                     int32_t* status) {
  spikegen_step_body(P, clock, k, status);
}

// ---- two populations in one launch ---------------------------------------------------------
// A source population (Poisson or spike generator) and the LIF or HH population it drives, the
// two of an ordinary driven network: CTAs [0, n_first) update the first, the others the second.
// Launched side by side on two streams they cost a step a fork and a join, and the launches after
// the join cannot be chained.  Poisson and LIF with STDP, us per step, two launches -> one and
// chained: 1e4 -> 1e3 22.4 -> 20.9, 3,001 -> 257 (f64) 10.3 -> 8.8.
// EB = 0: a HH neuron's variables in four warps.
template <int KA, typename RA, int KB, typename RB, int EB>
__global__ void __launch_bounds__(kBlock)
pair_step_kernel(const __grid_constant__ PopDev A, const __grid_constant__ PopDev B,
                 const int64_t* __restrict__ clock, int k, double dt, int32_t* status,
                 int n_first) {
  if ((int)blockIdx.x < n_first) {
    if constexpr (KA == KIND_POISSON)
      poisson_step_body<RA, 2, false>(A, clock, k, dt, status, blockIdx.x);
    else
      spikegen_step_body(A, clock, k, status);
  } else {
    const int64_t blk = (int64_t)blockIdx.x - n_first;
    if constexpr (EB == 0) hh_split_body<RB, false, true, true>(B, clock, k, dt, status, blk);
    else if constexpr (KB == KIND_HH)
      hh_step_body<RB, EB, false, false, true, true>(B, clock, k, dt, status, blk);
    else
      lif_step_body<RB, EB, false, false, true, true>(B, clock, k, dt, status, blk);
  }
}

// ---- reset after synaptic delivery (Brian2's 'resets' slot) -------------------------------
template <typename R>
__global__ void lif_late_reset_kernel(PopDev P, const int64_t* __restrict__ clock, int k) {
  const int64_t ts = clock[0] + k;
  const int slot = ring_slot(ts, P.ring_len);
  let_next_launch_start();
  previous_launch_done();
  const int cnt = P.ring_cnt[slot];
  const int32_t* idx = P.ring_idx + (int64_t)slot * P.n;
  const LifDev* prm = static_cast<const LifDev*>(P.params);
  R* V = static_cast<R*>(P.var[B2B_VAR_V]);
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < cnt; r += gridDim.x * blockDim.x) {
    const int32_t i = idx[r];
    const LifDev& g = prm[P.vec_group ? P.vec_group[i >> 2] : 0];
    if (g.has_reset) V[i] = (R)g.Vr;
  }
}

// Float64 HH populations below this size run hh_split_body.
constexpr int64_t kSplitNeurons = 32000;
// Neurons per thread and threads per CTA of a population's update: the autotuner's choice, else
// by kind, type and size.  Small populations are bound by one neuron's chain of loads and
// arithmetic, so every neuron gets a thread, in CTAs of 128 that spread over more SMs; once a
// thread per neuron is more than a wave of CTAs, the per-thread work (the clock, the group's
// constants, the addresses) counts and two, then four neurons share it.  Measured, us per step
// at 1 / 2 / 4 neurons per thread of 128 (256: 1-8 % slower): HH f32 20,000 2.48 / 2.75 / 3.27,
// 100,000 3.16 / 3.18 / 3.70 (two are 5 % faster beside a delivery), 220,000 4.59 / 3.94 /
// 4.18, 300,000 5.41 / 5.09 / 4.67, 600,000 8.61 / 7.50 / 7.12; LIF f32 100,000 2.96 / 2.93 /
// 3.12, 300,000 4.71 / 3.45 / 3.44, 600,000 7.06 / 5.47 / 4.29; LIF f64 100,000 2.94 / 3.15 /
// 3.65, 150,000 3.40 / 3.28 / 3.72, 600,000 7.92 / 6.96 / 8.24; HH f64 (two or more
// serialise its exponentials) 8000-450,000: one; Poisson 100,000 2.69 / 2.65 / 2.65, 300,000
// 3.42 / 3.10 / 3.03.
struct UpdateShape {
  int e, block;
  bool split;                     // a HH neuron's variables in four warps (hh_split_body; e = 1)
};
// Beside a delivery (beside: the update of the two launches) HH f32 keeps two: 460,000 9.83 ->
// 9.11 us per step, 613,000 12.5 -> 11.7.
UpdateShape update_shape(const Pop& pop, int64_t n, bool beside = false) {
  const bool f32 = pop.dtype == B2B_F32;
  int e = 1;
  if (pop.kind == KIND_HH && pop.tune_e == 0 && !pop.inputs && !f32 && n < kSplitNeurons)
    return {1, pop.tune_block > 0 ? pop.tune_block : 128, true};
  if (pop.kind == KIND_POISSON) e = n >= 200000 ? 4 : 2;
  else if (f32) e = n >= 280000 && !(beside && pop.kind == KIND_HH) ? 4 : (n >= 90000 ? 2 : 1);
  else if (pop.kind == KIND_LIF) e = n >= 130000 ? 2 : 1;
  return {pop.tune_e > 0 ? pop.tune_e : e, pop.tune_block > 0 ? pop.tune_block : 128, false};
}

// Neurons per thread of the forms that deliver as well (0: four threads per neuron).
int one_launch_e(const UpdateShape& shape) { return shape.split ? 0 : shape.e >= 2 ? 2 : 1; }

// CTAs of an update of n neurons at e neurons per thread (0: four threads per neuron).
unsigned update_grid(const UpdateShape& shape, int e, int64_t n) {
  const int64_t threads = e == 0 ? 4 * n : n / e;
  return (unsigned)((threads + shape.block - 1) / shape.block);
}

template <int E, bool IN, bool CNT>
cudaError_t launch_e(const Pop& pop, const PopDev& P, const int64_t* clock, int k, double dt,
                     int32_t* status, cudaStream_t s) {
  const int block = update_shape(pop, P.n).block;   // <= kBlock (the same beside a delivery)
  const unsigned grid = (unsigned)((P.n / E + block - 1) / block);
  const bool f32 = pop.dtype == B2B_F32;
  switch (pop.kind) {
    case KIND_LIF:
      if (f32) lif_step_kernel<float, E, IN, CNT><<<grid, block, 0, s>>>(P, clock, k, dt, status);
      else lif_step_kernel<double, E, IN, CNT><<<grid, block, 0, s>>>(P, clock, k, dt, status);
      break;
    case KIND_HH:
      if (E == 4 && f32) {
        // resident CTAs only (2 per SM of 256 threads by the launch bounds); float64 keeps
        // one pack per thread (two packs of doubles do not fit the register budget)
        const unsigned g2 = std::min<unsigned>(grid, 2 * kNumSMs * (kBlock / block));
        hh_stream_kernel<float, IN, CNT><<<g2, block, 0, s>>>(P, clock, k, dt, status);
      } else if (f32) {
        hh_step_kernel<float, E, IN, CNT><<<grid, block, 0, s>>>(P, clock, k, dt, status);
      } else {
        hh_step_kernel<double, E, IN, CNT><<<grid, block, 0, s>>>(P, clock, k, dt, status);
      }
      break;
    case KIND_POISSON:
      if (f32) poisson_step_kernel<float, E, IN><<<grid, block, 0, s>>>(P, clock, k, dt, status);
      else poisson_step_kernel<double, E, IN><<<grid, block, 0, s>>>(P, clock, k, dt, status);
      break;
    default:
      return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

template <int KA, typename RA>
cudaError_t launch_pair_a(const Pop& a, const Pop& b, int block, int eb, const int64_t* clock,
                          int k, double dt, int32_t* status, cudaStream_t s, bool chained) {
  const unsigned first = KA == KIND_SPIKEGEN ? 1 : (unsigned)((a.dev.n / 2 + block - 1) / block);
  const int64_t threads = eb == 0 ? 4 * b.dev.n : b.dev.n / eb;
  const unsigned grid = first + (unsigned)((threads + block - 1) / block);
  auto launch = [&](auto kernel) {
    return launch_kernel(kernel, dim3(grid), block, 0, s, chained, a.dev, b.dev, clock, k, dt,
                         status, (int)first);
  };
  const bool f32 = b.dtype == B2B_F32;
  if (b.kind == KIND_HH) {
    if (eb == 0) return launch(pair_step_kernel<KA, RA, KIND_HH, double, 0>);
    if (!f32) return launch(pair_step_kernel<KA, RA, KIND_HH, double, 1>);
    return eb == 2 ? launch(pair_step_kernel<KA, RA, KIND_HH, float, 2>)
                   : launch(pair_step_kernel<KA, RA, KIND_HH, float, 1>);
  }
  if (f32)
    return eb == 2 ? launch(pair_step_kernel<KA, RA, KIND_LIF, float, 2>)
                   : launch(pair_step_kernel<KA, RA, KIND_LIF, float, 1>);
  return eb == 2 ? launch(pair_step_kernel<KA, RA, KIND_LIF, double, 2>)
                 : launch(pair_step_kernel<KA, RA, KIND_LIF, double, 1>);
}

}  // namespace

cudaError_t launch_pop_step(const Pop& pop, const int64_t* clock, int k, double dt,
                            int32_t* status, cudaStream_t s) {
  return launch_pop_step_dev(pop, pop.dev, clock, k, dt, status, s);
}

bool update_is_split(const Pop& pop) { return update_shape(pop, pop.dev.n).split; }

bool pair_supported(const Pop& a, const Pop& b) {
  for (const Pop* p : {&a, &b})
    if (p->inputs || p->surr_img || p->tune_e != 0 || p->tune_block != 0) return false;
  const UpdateShape sa = update_shape(a, a.dev.n), sb = update_shape(b, b.dev.n);
  return (a.kind == KIND_SPIKEGEN || (a.kind == KIND_POISSON && sa.e == 2)) &&
         (b.kind == KIND_LIF || b.kind == KIND_HH) && sb.e <= 2;
}

cudaError_t launch_pair_step(const Pop& a, const Pop& b, const int64_t* clock, int k, double dt,
                             int32_t* status, cudaStream_t s, bool chained) {
  const UpdateShape sb = update_shape(b, b.dev.n);
  const int eb = sb.split ? 0 : sb.e;
  if (a.kind == KIND_SPIKEGEN)
    return launch_pair_a<KIND_SPIKEGEN, float>(a, b, sb.block, eb, clock, k, dt, status, s,
                                               chained);
  if (a.dtype == B2B_F32)
    return launch_pair_a<KIND_POISSON, float>(a, b, sb.block, eb, clock, k, dt, status, s,
                                              chained);
  return launch_pair_a<KIND_POISSON, double>(a, b, sb.block, eb, clock, k, dt, status, s, chained);
}

cudaError_t launch_pop_step_dev(const Pop& pop, const PopDev& dev, const int64_t* clock, int k,
                                double dt, int32_t* status, cudaStream_t s) {
  if (pop.kind == KIND_HH && pop.surr_img) return launch_hh_surrogate(pop, clock, k, dt, status, s);
  if (pop.kind == KIND_MODEL)   // the generated model's own kernel, from its shared object
    return (cudaError_t)pop.model_launch(&dev, clock, k, dt, status, s, pop.dtype, 0);
  if (pop.kind == KIND_SPIKEGEN) {
    spikegen_step_kernel<<<1, kBlock, 0, s>>>(pop.dev, clock, k, status);
    return cudaGetLastError();
  }
  const UpdateShape shape =
      update_shape(pop, pop.dev.n, dev.fold[B2B_VAR_GE] || dev.fold[B2B_VAR_GI]);
  const int e = shape.e;
  if (shape.split) {
    hh_split_kernel<double>
        <<<update_grid(shape, 0, dev.n), shape.block, 0, s>>>(dev, clock, k, dt, status);
    return cudaGetLastError();
  }
  auto launch = [&](auto in, auto counted) {
    constexpr bool IN = decltype(in)::value, CNT = decltype(counted)::value;
    if (e == 4) return launch_e<4, IN, CNT>(pop, dev, clock, k, dt, status, s);
    if (e == 2) return launch_e<2, IN, CNT>(pop, dev, clock, k, dt, status, s);
    return launch_e<1, IN, CNT>(pop, dev, clock, k, dt, status, s);
  };
  using T = std::true_type;
  using N = std::false_type;
  if (dev.fold_gw) return pop.inputs ? launch(T{}, T{}) : launch(N{}, T{});
  return pop.inputs ? launch(T{}, N{}) : launch(N{}, N{});
}

bool one_launch_supported(const Pop& pop, const PendingDev& F) {
  return (pop.kind == KIND_LIF || pop.kind == KIND_HH) && !pop.inputs && !pop.surr_img &&
         F.nd_max <= kWarpPrefixMaxDelays;
}

cudaError_t launch_one_launch_step(const Pop& pop, const PopDev& U, const PendingDev& F,
                                   int deliver_ctas, bool chained, const int64_t* clock, int k,
                                   double dt, int32_t* status, cudaStream_t s) {
  if (!one_launch_supported(pop, F) || deliver_ctas < 1) return cudaErrorInvalidValue;
  // the update half takes the population's shape (neurons per thread 1 or 2, 128 or 256
  // threads per CTA); the delivery half the same threads per CTA, deliver_ctas counted in
  // CTAs of kBlock threads
  const UpdateShape shape = update_shape(pop, U.n);
  const int e = one_launch_e(shape), block = shape.block;
  const int n_upd = (int)update_grid(shape, e, U.n);
  const unsigned grid = (unsigned)(n_upd + (int64_t)deliver_ctas * kBlock / block);
  return with_one_launch(pop, e, F.group, F.n_proj, [&](auto kernel, auto np) {
    return launch_kernel(kernel, dim3(grid), block, 0, s, chained, U,
                         pending_args<decltype(np)::value>(F), clock, k, dt, status, n_upd);
  });
}

// A step with many events is as long as its delivery, which the SMs' delivering warps bound; in a quiet
// one the launch is over sooner if the next step's CTAs find room beside it, so up to there the
// delivering CTAs are as many as leave it (half of what an SM holds), at least 1.5 per SM.  Where the update alone leaves the next step no room, they are as many as
// run in one wave, as the bundles need them: two per SM for short ones of LIF, 2.5, and three for long
// (16 lanes each), which are worth them beyond the wave as well.  Up to 10,000 neurons a step has too few
// events.  us per step at 1.5 / 2 / 2.5 / 3 CTAs per SM, at 12 and 220 Hz: LIF f32 (synapses per neuron over 20
// delays) 4000 (80) 2.75 / 2.95 / - / 3.24 and 2.93 / 3.05 / - / 3.36; 12,000 (80) 2.96 / 2.88 / 3.12 / 3.21 and 3.6 /
// 3.6 / 3.7 / 3.8; 20,000 (1000) 3.33 / 3.35 / - / 3.50 and 10.2 / 8.0 / - / 8.2; 35,000 (80) 2.90 / 3.18 / 3.14 / 3.13 and
// 6.5 / 5.9 / 5.4 / 4.9; 45,000 (80) 3.14 / 3.14 / 3.13 / 3.17 and 5.6 / 5.2 / 4.6 / 4.4; 68,000 (80) 3.14 / 3.16 / 3.21 /
// 3.31 and 6.8 / 6.6 / 6.0 / 5.7, (300) 3.18 / 3.26 / 3.33 / 3.37 and 11.2 / 11.2 / 9.6 / 8.5; 60,000 (1000) 3.95 / 3.81 / - /
// 3.95 and 25.8 / 20.5 / - / 15.4; 100,000 (two neurons per thread) (300) 3.43 / 3.46 / - / 3.95 and 15.2 / 12.0 / - /
// 10.0, (1000) 4.51 / 4.30 / - / 4.71 and 31.3 / 24.1 / - / 19.5; 150,000 (1000) 5.38 / 5.13 / - / 5.12 and 37.6 / 36.2 /
// - / 27.1.  COBAHH f32 12,500 2.91 / 2.89 / 2.93 / 2.99, 18,786 2.75 / 2.46 / 2.75 / 2.81, 28,603 2.84 / 2.59 / 2.70 /
// 2.77, 36,000 2.56 / 2.77 / 2.87 / 2.88, 50,186 3.00 / 3.02 / 3.10 / 3.11, 70,001 3.33 / 3.40 / 3.27 / 3.24, 85,000 3.59 /
// 3.44 / 3.36 / 3.37; f64 20,000 3.25 / 3.46 / 3.58 / 3.61.
int builtin_one_launch_grid(const Pop& pop, const PendingDev& F, double mean_bundle, int sms) {
  const int64_t n = pop.dev.n;
  int halves = 3;
  if (n > 10000) {
    const UpdateShape shape = update_shape(pop, n);
    const int e = one_launch_e(shape);
    int resident = 0;
    with_one_launch(pop, e, F.group, F.n_proj, [&](auto kernel, auto) {
      return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident, kernel, shape.block, 0);
    });
    const int64_t update = update_grid(shape, e, n);
    // halves of a CTA of kBlock threads per SM that fit beside the update in `slots` CTAs
    auto beside = [&](double slots) {
      return (int)std::floor(2 * (slots - (double)update) * shape.block / kBlock / sms);
    };
    const bool lif = pop.kind == KIND_LIF;
    const bool is_long = lif && mean_bundle >= kLongBundle;
    const int with_next = beside(0.5 * resident * sms);
    const int one_wave = beside((double)resident * sms);
    const bool large = lif ? n > 40000 : update > 3 * sms;
    if (large) halves = std::min(one_wave, is_long ? 6 : lif && mean_bundle < 10 ? 4 : 5);
    else halves = is_long ? 4 : std::min(with_next, 4);
    if (is_long && n >= 90000) halves = 6;
    halves = std::max(halves, 3);
  }
  return halves * sms / 2;
}

// Its warps deliver as well, so a thread per neuron pays up to one wave of CTAs of 128 (us per step at
// 1 / 2 neurons per thread, LIF f32, 80 synapses per neuron at 12 and 220 Hz: 100,000 3.89 / 4.13 and
// 6.14 / 6.82, 150,000 4.18 / 4.35 and 7.18 / 8.40, 200,000 5.72 / 4.89 and 9.33 / 10.1; f64 140,000
// with 130 synapses 4.56 / 5.46; HH f32 140,000 4.87 / 5.44, 180,000 6.08 / 5.53).
constexpr int64_t kFusedOneEach = 150000;
cudaError_t launch_fused_step(const Pop& pop, const PopDev& U, const FusedDev& F, bool chained,
                              const int64_t* clock, int k, double dt, int32_t* status,
                              cudaStream_t s) {
  UpdateShape shape = update_shape(pop, U.n);
  if (pop.tune_e == 0 && U.n <= kFusedOneEach) shape.e = 1;
  const int e = one_launch_e(shape), b = shape.block;
  const unsigned grid = update_grid(shape, e, U.n);
  const bool f32 = pop.dtype == B2B_F32;
  if (pop.kind == KIND_HH)
    return f32 ? launch_fused_rk<float, KIND_HH>(U, F, e, grid, b, chained, clock, k, dt, status, s)
               : launch_fused_rk<double, KIND_HH>(U, F, e, grid, b, chained, clock, k, dt, status,
                                                  s);
  return f32 ? launch_fused_rk<float, KIND_LIF>(U, F, e, grid, b, chained, clock, k, dt, status, s)
             : launch_fused_rk<double, KIND_LIF>(U, F, e, grid, b, chained, clock, k, dt, status,
                                                 s);
}

cudaError_t launch_fold_counts(const Pop& pop, const PopDev& U, int k_last, cudaStream_t s) {
  const unsigned grid =
      (unsigned)std::min<int64_t>((U.n + kBlock - 1) / kBlock, 4 * kNumSMs);
  if (pop.dtype == B2B_F32) fold_counts_kernel<float><<<grid, kBlock, 0, s>>>(U, k_last & 1);
  else fold_counts_kernel<double><<<grid, kBlock, 0, s>>>(U, k_last & 1);
  return cudaGetLastError();
}

cudaError_t launch_pop_late_reset(const Pop& pop, const int64_t* clock, int k, cudaStream_t s,
                                  bool chained) {
  if (pop.kind == KIND_MODEL)
    return (cudaError_t)pop.model_launch(&pop.dev, clock, k, 0.0, nullptr, s, pop.dtype, 1);
  if (pop.kind != KIND_LIF) return cudaSuccess;
  const dim3 grid(2 * kNumSMs);
  return pop.dtype == B2B_F32
             ? launch_kernel(lif_late_reset_kernel<float>, grid, kBlock, 0, s, chained, pop.dev,
                             clock, k)
             : launch_kernel(lif_late_reset_kernel<double>, grid, kBlock, 0, s, chained, pop.dev,
                             clock, k);
}

namespace {
__global__ void tick_kernel(int64_t* clock, int steps) { clock[0] += steps; }
}  // namespace

cudaError_t launch_tick(int64_t* clock, int steps, cudaStream_t s) {
  tick_kernel<<<1, 1, 0, s>>>(clock, steps);
  return cudaGetLastError();
}

}  // namespace b2b
