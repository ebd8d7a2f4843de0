// Batched Hines solver for multicompartment (SpatialNeuron) HH neurons.
//
// Reference: brian2cuda/templates/spatialstateupdate.cu runs, per SpatialNeuron and step,
// five launches: channel update (108-113), `_tridiagsolve<<<branches, 1>>>` (128-192,
// Thomas algorithm with three right-hand sides per section), `_coupling<<<1, 1>>>` (202-307,
// the Hines elimination over the section tree on a single thread), `_combine<<<branches,
// 1>>>` (316-351) and `_currents` (359-387).  One neuron is one code object, so a batch of
// neurons costs five launches per neuron per step.
//
// The method (domain decomposition of the backward-Euler cable equation), restated from the
// mathematics: compartment j couples to compartment j-1 of its section through the axial
// conductance g[j] (0 at a section's first compartment), a section's first and last
// compartments to its start and end nodes through g0 and gn.  Per section, three
// tridiagonal solves with one matrix give x* (both node voltages 0) and the responses u_start,
// u_end to a unit voltage at either node, so that v = x* + V_start u_start + V_end u_end;
// Kirchhoff's current law at the nodes (node 0: the sealed start of the root section, node
// s+1: the end of section s) gives a tree-shaped system in the node voltages.
//
// Here one CTA owns one neuron and keeps it on chip across a chunk of steps (the state of its
// compartments in registers, everything the phases exchange in shared memory); the only
// global traffic inside the chunk is the soma spike count.  Per step: compartment-parallel
// channels, section-parallel tridiagonal solves, node-parallel assembly of the node
// equations, then elimination (each node pulls in its children) and substitution level by
// level over the section tree (nodes of equal depth are independent), and a
// compartment-parallel combination.
//
// A step is a chain of latencies (an SM holds 2-5 neurons), so each phase is written for its
// chain: operands that do not depend on the previous link are loaded ahead of it, a node's
// children are read without branches (a dummy child adds 0), and a node's four numbers are
// two 16-byte pairs.  Cycles per step of a 375-compartment, 15-level neuron alone on its SM,
// before / after (clock64 in a copy of the kernel, float64 channels): channels 6450 / 3170,
// sections 3310 / 2340, node equations 1000 / 880, elimination 14190 / 2370, substitution 6300 /
// 1350, combination 810 / 220.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <new>
#include <vector>

#include "kernels_common.cuh"

namespace b2b {
namespace {

constexpr int kHinesBlock = 256;
constexpr int kHinesMaxStepsPerLaunch = 1000;
constexpr int kHinesWide = 512;      // threads per CTA when every neuron has an SM to itself
constexpr int kHinesMaxInRegs = 1024;  // largest neuron whose state the registers hold
constexpr int kHinesSmallCtas = 5;   // CTAs per SM whose images the small class's would fit

struct HinesDev {
  int32_t n_neurons;
  int32_t nc_max, ns_max, nlev_max;
  const int64_t* comp_off;
  const int32_t* sec_off;
  const int32_t* lvl_base;
  // per compartment: matrix row without the membrane conductance (low couples j to j-1, up
  // couples j to j+1; both 0 across section boundaries)
  const double *low, *diag, *up;
  const int32_t* sec_of_comp;
  const int32_t *sec_start, *sec_end, *sec_pnode;
  // per section: node couplings, and the right-hand side of the unit-node solves at the
  // first (-g0/area) and last (-gn/area) compartment
  const double *g0, *gn, *rhs_first, *rhs_last;
  const int32_t* child_off;   // per node (global node index = sec_off[b] + b + i), global edges
  const int32_t* child_sec;   // neuron-local section index per edge
  // per node slot, nodes sorted by depth: neuron-local indices times 16 (byte offsets of 16-byte
  // entries) of {node, end nodes of its first and second child section (node ns + 1, a dummy,
  // where there is none), parent node}; and the edges of its further children, first | end << 16
  const int4* level_rec;
  const int32_t* more_rec;
  // per neuron at lvl_base[b]: offsets into level_rec of its groups of at most 32 nodes of one
  // depth, and their end
  const int32_t* level_off;
  double* v;
  void *m, *h, *n;
  double* Ic;
  const double* soma_I;       // per neuron injected current / soma area (A/m^2)
  int32_t* spikes;
  int32_t* above;
  double Cm, dt, El, EK, ENa, gl, gNa, gK, Vthr;
  // neuron of CTA k: neurons by decreasing estimated cost, so that the CTAs the block
  // scheduler starts last (when fewer than all neurons fit on the GPU at once) are the
  // shortest
  const int32_t* order;
};

template <typename RC>
__device__ __forceinline__ RC hh_expeuler(RC x, RC a, RC b, RC dt) {
  const RC A = -(a + b);
  const RC BA = a / A;
  return -BA + (BA + x) * dexp(A * dt);
}

// x / c for a literal c, correctly rounded: the product with the rounded reciprocal, corrected
// by its residual (P. Markstein, "Computation of elementary functions on the IBM RISC System/6000
// processor", 1990: with 1/c correctly rounded one fused residual step rounds the quotient
// correctly).  Three operations without a branch, where the general quotient's range checks
// keep the exponentials around it from overlapping.  The last place may differ where the residual is
// inexact (|x| below 2^-101 in float32, 2^-968 in float64: its last place is below the smallest
// subnormal number) and above 3e38 (kept uncorrected, as the residual may overflow), of values whose
// exponentials are 1, 0 or infinite.
template <typename RC>
__device__ __forceinline__ RC div_lit(RC x, double c) {
  const RC b = (RC)c, y = (RC)(1.0 / (double)b);
  const RC q = x * y;
  const RC r = dfma(-q, b, x);
  return fabs(q) <= (RC)3e38 ? dfma(r, y, q) : q;
}

// Hodgkin-Huxley 1952 rates (examples/compartmental/hh_with_spikes_cuda.py:41-46), v in
// volts measured from rest, rates in 1/s; x/(exp(x/a) - 1) forms through z_over_expm1.
template <typename RC>
__device__ __forceinline__ void hh_gates(RC v, RC dt, RC& m, RC& h, RC& n) {
  const RC am = (RC)1000 * z_over_expm1(div_lit<RC>((RC)25e-3 - v, 10e-3));
  const RC bm = (RC)4000 * dexp(div_lit<RC>(-v, 18e-3));
  const RC ah = (RC)70 * dexp(div_lit<RC>(-v, 20e-3));
  const RC bh = (RC)1000 / (dexp(div_lit<RC>((RC)30e-3 - v, 10e-3)) + (RC)1);
  const RC an = (RC)100 * z_over_expm1(div_lit<RC>((RC)10e-3 - v, 10e-3));
  const RC bn = (RC)125 * dexp(div_lit<RC>(-v, 80e-3));
  m = hh_expeuler(m, am, bm, dt);
  h = hh_expeuler(h, ah, bh, dt);
  n = hh_expeuler(n, an, bn, dt);
}

// 1/x for a finite, normal, nonzero x: the reciprocal unit's approximation refined by two
// Newton-Raphson steps (y <- y + y (1 - x y), each step doubling the correct bits), within
// an ulp or two of the correctly rounded quotient.  The solver's serial chains (the pivots of
// a section, the node system level by level) take one reciprocal per link; the IEEE
// division's longer sequence made them several times longer.
__device__ __forceinline__ double recip(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  double e = fma(-x, y, 1.0);
  y = fma(y, e, y);
  e = fma(-x, y, 1.0);
  return fma(y, e, y);
}

// KC: compartments per thread whose state (v, the gates, the constant matrix diagonal) lives in
// registers, the matrix couplings then in shared memory; 0: neurons of any size, the state in
// shared memory and the matrix read through the read-only cache.  BS threads per CTA; MINB: CTAs
// per SM the register budget is sized for (hines_variant).
template <typename RC, int KC, int BS, int MINB>
__global__ void __launch_bounds__(BS, MINB)
hines_kernel(HinesDev H, int n_steps, int write_currents) {
  extern __shared__ __align__(16) uint8_t sm[];
  const int b = H.order[blockIdx.x];
  const int tid = threadIdx.x;
  const int64_t c0 = H.comp_off[b];
  const int nc = (int)(H.comp_off[b + 1] - c0);
  const int s0 = H.sec_off[b];
  const int ns = H.sec_off[b + 1] - s0;
  const int nB = ns + 1;                     // nodes; node nB is the dummy child
  const int nb0 = s0 + b;
  const int l0 = H.lvl_base[b];
  const int nlev = H.lvl_base[b + 1] - l0 - 1;
  const int NC = H.nc_max, NS = H.ns_max, ND = H.ns_max + 2;

  int4* REC = reinterpret_cast<int4*>(sm);                    // level records
  // a node's equation {diagonal, right-hand side}, after its elimination {1 / diagonal,
  // right-hand side}, at last the right-hand side the node's voltage; and its coefficient in
  // its parent's equation and the parent's in its own
  double2* EQ = reinterpret_cast<double2*>(REC + ND);
  double2* IT = EQ + ND;
  // per compartment: the membrane solve's {diagonal, right-hand side}, after the forward pass
  // {eliminated super-diagonal, right-hand side}, at last {u_end, x*}; and u_start
  double2* DX = IT + ND;
  double2* LU = DX + NC;                                      // KC > 0: {low, up} couplings
  double* US = reinterpret_cast<double*>(LU + (KC > 0 ? NC : 0));
  double* G0 = US + NC;
  double* GN = G0 + NS;
  double* RF = GN + NS;
  double* RL = RF + NS;
  double* Vs = RL + NS;                                       // KC == 0: the state
  RC* Ms = reinterpret_cast<RC*>(Vs + (KC > 0 ? 0 : NC));
  RC* Hs = Ms + (KC > 0 ? 0 : NC);
  RC* Ns = Hs + (KC > 0 ? 0 : NC);
  int32_t* SST = reinterpret_cast<int32_t*>(Ns + (KC > 0 ? 0 : NC));
  int32_t* SEN = SST + NS;
  int32_t* SPN = SEN + NS;
  int32_t* CSEC = SPN + NS;
  int32_t* MORE = CSEC + NS;   // edges of a node's children past the second, first | end << 16
  int32_t* LOFF = MORE + ND;

  constexpr int K1 = KC > 0 ? KC : 1;
  double vr[K1], dr[K1];
  RC mr[K1], hr[K1], nr[K1];
  int32_t nodes[K1];           // start node | section << 16 of each compartment
  // every compartment of this thread: f(j, its register slot)
  auto for_comps = [&](auto f) {
    if constexpr (KC > 0) {
#pragma unroll
      for (int c = 0; c < KC; ++c)
        if (tid + c * BS < nc) f(tid + c * BS, c);
    } else {
      for (int j = tid; j < nc; j += BS) f(j, 0);
    }
  };

  for (int s = tid; s < ns; s += BS) {
    SST[s] = H.sec_start[s0 + s];
    SEN[s] = H.sec_end[s0 + s];
    SPN[s] = H.sec_pnode[s0 + s];
    G0[s] = H.g0[s0 + s];
    GN[s] = H.gn[s0 + s];
    RF[s] = H.rhs_first[s0 + s];
    RL[s] = H.rhs_last[s0 + s];
  }
  const int e0 = H.child_off[nb0];
  for (int e = tid; e < ns; e += BS) CSEC[e] = H.child_sec[e0 + e];
  bool more = false;           // some node has more than two children
  for (int k = tid; k < nB; k += BS) {
    REC[k] = H.level_rec[nb0 + k];
    MORE[k] = H.more_rec[nb0 + k];
    more |= (MORE[k] & 0xffff) != (int)((unsigned)MORE[k] >> 16);
  }
  if (tid == 0) {
    EQ[nB] = make_double2(1.0, 0.0);
    IT[nB] = make_double2(0.0, 0.0);
    IT[0] = make_double2(0.0, 0.0);
  }
  for (int L = tid; L <= nlev; L += BS) LOFF[L] = H.level_off[l0 + L];
  const bool any_more = __syncthreads_or(more);
  {
    const RC* gm = static_cast<const RC*>(H.m);
    const RC* gh = static_cast<const RC*>(H.h);
    const RC* gn = static_cast<const RC*>(H.n);
    for_comps([&](int j, int c) {
      if constexpr (KC > 0) {
        vr[c] = H.v[c0 + j];
        mr[c] = gm[c0 + j];
        hr[c] = gh[c0 + j];
        nr[c] = gn[c0 + j];
        dr[c] = H.diag[c0 + j];
        LU[j] = make_double2(H.low[c0 + j], H.up[c0 + j]);
        const int s = H.sec_of_comp[c0 + j];
        nodes[c] = SPN[s] | s << 16;
      } else {
        Vs[j] = H.v[c0 + j];
        Ms[j] = gm[c0 + j];
        Hs[j] = gh[c0 + j];
        Ns[j] = gn[c0 + j];
      }
    });
  }

  const double cdt = H.Cm / H.dt;
  const double Isoma = H.soma_I[b];
  const RC dtR = (RC)H.dt;
  int above = H.above[b];
  int spikes = 0;

  for (int step = 0; step < n_steps; ++step) {
    // (1) channels: conductance and current at the start of the step, then the gates
    for_comps([&](int j, int c) {
      const double v = KC > 0 ? vr[c] : Vs[j];
      RC m = KC > 0 ? mr[c] : Ms[j], h = KC > 0 ? hr[c] : Hs[j], n = KC > 0 ? nr[c] : Ns[j];
      const double md = (double)m, hd = (double)h, nd = (double)n;
      const double gna = H.gNa * (md * md * md * hd);
      const double gk = H.gK * (nd * nd * nd * nd);
      const double gtot = H.gl + gna + gk;
      double I0 = H.gl * H.El + gna * H.ENa + gk * H.EK;
      if (j == 0) I0 += Isoma;
      DX[j] = make_double2((KC > 0 ? dr[c] : __ldg(H.diag + c0 + j)) - gtot, -cdt * v - I0);
      hh_gates<RC>((RC)v, dtR, m, h, n);
      if constexpr (KC > 0) {
        mr[c] = m; hr[c] = h; nr[c] = n;
      } else {
        Ms[j] = m; Hs[j] = h; Ns[j] = n;
      }
    });
    __syncthreads();
    // (2) per section, one pass of forward elimination (reciprocal pivot) and back
    // substitution for the three right-hand sides.  The pivots are one chain per section:
    // the next compartment's operands are loaded ahead of it (clamped, not branched) and what
    // is passed along stays in registers.  u_end is 0 before the last compartment of the
    // forward pass; the couplings into a section's first and out of its last compartment are 0.
    for (int s = tid; s < ns; s += BS) {
      const int j0 = SST[s], last = SEN[s] - 1;
      auto couplings = [&](int j) {
        return KC > 0 ? LU[j] : make_double2(__ldg(H.low + c0 + j), __ldg(H.up + c0 + j));
      };
      double2 lu = couplings(j0), dx = DX[j0];
      double rs = RF[s];
      const double rl = RL[s];
      double cprev = 0.0, xprev = 0.0, sprev = 0.0, piv = 0.0;
#pragma unroll 2
      for (int j = j0; j <= last; ++j) {
        const int jn = min(j + 1, last);
        const double2 lun = couplings(jn), dxn = DX[jn];
        piv = recip(dx.x - lu.x * cprev);
        cprev = lu.y * piv;
        xprev = (dx.y - lu.x * xprev) * piv;
        sprev = (rs - lu.x * sprev) * piv;
        DX[j] = make_double2(cprev, xprev);   // the diagonal is not needed again
        US[j] = sprev;
        lu = lun;
        dx = dxn;
        rs = 0.0;
      }
      double eprev = rl * piv;
      DX[last].x = eprev;
      int j = max(last - 1, j0);
      dx = DX[j];
      double us = US[j];
#pragma unroll 2
      for (j = last - 1; j >= j0; --j) {
        const int jn = max(j - 1, j0);
        const double2 dxn = DX[jn];
        const double un = US[jn];
        xprev = dx.y - dx.x * xprev;
        sprev = us - dx.x * sprev;
        eprev = -(dx.x * eprev);
        DX[j] = make_double2(eprev, xprev);
        US[j] = sprev;
        dx = dxn;
        us = un;
      }
    }
    __syncthreads();
    // (3) node equations: node i's current balance in its own voltage, its parent node's
    // and its children's end nodes' (stored with the child node)
    for (int k = tid; k < nB; k += BS) {
      const int4 r = REC[k];
      const int i = r.x >> 4;
      double dn, rh;
      if (i == 0) {
        // the root's start takes the voltage of the root's first compartment
        const int f = SST[0];
        dn = US[f] - 1.0;
        rh = -DX[f].y;
        IT[1].x = DX[f].x;
      } else {
        const int s = i - 1, l = SEN[s] - 1;
        const double2 ex = DX[l];
        dn = GN[s] * (1.0 - ex.x);
        IT[i].y = -GN[s] * US[l];
        rh = GN[s] * ex.y;
        auto child = [&](int cn) {   // cn: the child section's end node
          const int f = SST[cn - 1];
          const double g = G0[cn - 1];
          const double2 exf = DX[f];
          dn += g * (1.0 - US[f]);
          IT[cn].x = -g * exf.x;
          rh += g * exf.y;
        };
        if ((r.y >> 4) < nB) child(r.y >> 4);
        if ((r.z >> 4) < nB) child(r.z >> 4);
        if (any_more)
          for (int e = MORE[k] & 0xffff; e < (int)((unsigned)MORE[k] >> 16); ++e)
            child(CSEC[e] + 1);
      }
      EQ[i] = make_double2(dn, rh);
    }
    __syncthreads();
    // (4)-(5) the node system on the first warp alone, group by group of at most 32 nodes of
    // one depth, with warp barriers.  Records hold byte offsets into EQ and IT and are loaded
    // two groups ahead, what else does not depend on the group before it one ahead; the dummy
    // child of a node with fewer than two subtracts 0.
    if (tid < 32) {
      char* const eqb = reinterpret_cast<char*>(EQ);
      char* const itb = reinterpret_cast<char*>(IT);
      auto eq_at = [&](int off) -> double2& { return *reinterpret_cast<double2*>(eqb + off); };
      auto it_at = [&](int off) -> double2& { return *reinterpret_cast<double2*>(itb + off); };
      // (4) elimination, deepest group first: each node takes in its children's equations in
      // the children's order
      int hi = nB, lo = LOFF[nlev - 1], lo1 = LOFF[max(nlev - 2, 0)];
      if (!any_more) {
        int4 r = REC[min(lo + tid, nB - 1)], rn = REC[min(lo1 + tid, nB - 1)];
        double2 eq = eq_at(r.x), ia = it_at(r.y), ib = it_at(r.z);
        for (int L = nlev - 1; L >= 0; --L) {
          const double2 a = eq_at(r.y), c = eq_at(r.z);
          const int lo2 = LOFF[max(L - 2, 0)];
          const double2 eqn = eq_at(rn.x), ian = it_at(rn.y), ibn = it_at(rn.z);
          const int4 rnn = REC[min(lo2 + tid, nB - 1)];
          const double fa = ia.x * a.x, fb = ib.x * c.x;
          double dn = eq.x, rh = eq.y;
          dn -= fa * ia.y;
          rh -= fa * a.y;
          dn -= fb * ib.y;
          rh -= fb * c.y;
          const double inv = recip(dn);   // the node's equation is final here
          if (lo + tid < hi) eq_at(r.x) = make_double2(inv, rh);
          __syncwarp();
          r = rn; eq = eqn; ia = ian; ib = ibn; rn = rnn;
          hi = lo; lo = lo1; lo1 = lo2;
        }
      } else {
        for (int L = nlev - 1; L >= 0; --L) {
          const int k = LOFF[L] + tid;
          if (k < LOFF[L + 1]) {
            const int4 r = REC[k];
            double2 eq = eq_at(r.x);
            auto take = [&](int off) {
              const double2 it = it_at(off), c = eq_at(off);
              const double f = it.x * c.x;
              eq.x -= f * it.y;
              eq.y -= f * c.y;
            };
            take(r.y);
            take(r.z);
            for (int e = MORE[k] & 0xffff; e < (int)((unsigned)MORE[k] >> 16); ++e)
              take(16 * (CSEC[e] + 1));
            eq_at(r.x) = make_double2(recip(eq.x), eq.y);
          }
          __syncwarp();
        }
      }
      // (5) substitution, root first: the right-hand side becomes the node voltage
      if (tid == 0) EQ[0].y = EQ[0].y * EQ[0].x;
      lo = LOFF[min(1, nlev)];
      hi = LOFF[min(2, nlev)];
      int hi1 = LOFF[min(3, nlev)];
      int4 r = REC[min(lo + tid, nB - 1)], rn = REC[min(hi + tid, nB - 1)];
      double2 eq = eq_at(r.x);
      double toward = it_at(r.x).y;
      __syncwarp();
      for (int L = 1; L < nlev; ++L) {
        const double vp = eq_at(r.w).y;
        const double2 eqn = eq_at(rn.x);
        const double towardn = it_at(rn.x).y;
        const int hi2 = LOFF[min(L + 3, nlev)];
        const int4 rnn = REC[min(hi1 + tid, nB - 1)];
        if (lo + tid < hi) eq_at(r.x).y = (eq.y - toward * vp) * eq.x;
        __syncwarp();
        r = rn; eq = eqn; toward = towardn; rn = rnn;
        lo = hi; hi = hi1; hi1 = hi2;
      }
    }
    __syncthreads();
    // (6) v = x* + V_start u_start + V_end u_end; capacitive current
    const bool last_step = step == n_steps - 1;
    for_comps([&](int j, int c) {
      int pn, s;
      if constexpr (KC > 0) {
        pn = nodes[c] & 0xffff;
        s = nodes[c] >> 16;
      } else {
        s = __ldg(H.sec_of_comp + c0 + j);
        pn = SPN[s];
      }
      const double2 ex = DX[j];
      const double vn = ex.y + EQ[pn].y * US[j] + EQ[s + 1].y * ex.x;
      const double v = KC > 0 ? vr[c] : Vs[j];
      if (last_step && write_currents) H.Ic[c0 + j] = H.Cm * (vn - v) / H.dt;
      if constexpr (KC > 0) vr[c] = vn; else Vs[j] = vn;
    });
    // no barrier: a thread owns the same compartments here and in the next step's channel
    // phase (and thread 0 owns compartment 0); the next step's first barrier orders the rest
    if (tid == 0) {
      const int ab = (KC > 0 ? vr[0] : Vs[0]) > H.Vthr ? 1 : 0;
      if (ab && !above) ++spikes;
      above = ab;
    }
  }
  RC* wm = static_cast<RC*>(H.m);
  RC* wh = static_cast<RC*>(H.h);
  RC* wn = static_cast<RC*>(H.n);
  for_comps([&](int j, int c) {
    H.v[c0 + j] = KC > 0 ? vr[c] : Vs[j];
    wm[c0 + j] = KC > 0 ? mr[c] : Ms[j];
    wh[c0 + j] = KC > 0 ? hr[c] : Hs[j];
    wn[c0 + j] = KC > 0 ? nr[c] : Ns[j];
  });
  if (tid == 0) {
    H.spikes[b] += spikes;
    H.above[b] = above;
  }
}

// Shared memory of a neuron's image of nlev node groups (in_regs: its compartments' state is in
// registers).
size_t hines_smem(int nc, int ns, int nlev, int rc_size, bool in_regs) {
  const size_t ND = (size_t)ns + 2;
  return 48 * ND + sizeof(double) * ((in_regs ? 5 : 4) * (size_t)nc + 4 * (size_t)ns) +
         (in_regs ? 0 : rc_size * 3 * (size_t)nc) +
         sizeof(int32_t) * (4 * (size_t)ns + ND + (size_t)nlev + 1);
}

using HinesKernel = void (*)(HinesDev, int, int);

// The kernel and its threads per CTA for a class of neurons of up to nc compartments.
struct HinesVariant {
  HinesKernel kern;
  int block;
};
template <typename RC, int KC, int BS, int MINB>
HinesVariant variant() {
  return {hines_kernel<RC, KC, BS, MINB>, BS};
}
// Neurons that have an SM each are pure latency: 512 threads, so that fewer compartments share a
// thread (61 neurons of up to 400 compartments, float64 channels: 10.2 -> 5.3 us per step with
// the rest of the kernel's chains, 15.3 before both).  Otherwise as many neurons per SM as
// registers and shared memory allow cover each other's chains: the float32 variant of 1024
// compartments at 4 per SM with a few spills 20.2, at 3 without 21.6 us per step (1024 neurons of
// 200-1000 compartments); those of up to 768 at 5 per SM 13.4, at 4 12.1 (200-400 compartments).
template <typename RC>
HinesVariant hines_variant(int nc, bool one_per_sm) {
  constexpr bool f32 = sizeof(RC) == 4;
  if (one_per_sm) {
    if (nc <= kHinesWide) return variant<RC, 1, kHinesWide, 1>();
    if (nc <= 2 * kHinesWide) return variant<RC, 2, kHinesWide, 1>();
    return variant<RC, 0, kHinesBlock, 3>();
  }
  switch ((nc + kHinesBlock - 1) / kHinesBlock) {
    case 1: return variant<RC, 1, kHinesBlock, 4>();
    case 2: return variant<RC, 2, kHinesBlock, 4>();
    case 3: return variant<RC, 3, kHinesBlock, f32 ? 4 : 3>();
    case 4: return variant<RC, 4, kHinesBlock, f32 ? 4 : 3>();
    default: return variant<RC, 0, kHinesBlock, 3>();
  }
}

}  // namespace
}  // namespace b2b

struct b2b_hines {
  b2b_net* net = nullptr;
  b2b::HinesDev dev{};
  int channel_dtype = B2B_F32;
  int64_t n_comp = 0;
  int32_t n_neurons = 0;
  size_t smem = 0;
  // Neurons whose shared-memory image fits five CTAs per SM run as a second launch of their
  // own size beside the others (on stream2, forked from and joined to the net's stream), so
  // that small neurons do not reserve the largest neuron's shared memory.
  int32_t n_large = 0;                   // CTAs of the first launch (all neurons when 1 class)
  b2b::HinesVariant var{}, var_small{};   // kernels of the two classes
  b2b::HinesDev dev_small{};
  size_t smem_small = 0;
  cudaStream_t stream2 = nullptr;
  cudaEvent_t ev_fork = nullptr, ev_join = nullptr;
  std::vector<double> soma_area;
  std::vector<void*> allocs;
  std::string err;
};

using namespace b2b;

namespace {

template <typename T>
cudaError_t upload(b2b_hines* h, const T** dst, const std::vector<T>& src) {
  T* d = nullptr;
  cudaError_t e = cudaMalloc((void**)&d, sizeof(T) * std::max<size_t>(src.size(), 1));
  if (e != cudaSuccess) return e;
  h->allocs.push_back(d);
  if (!src.empty()) e = cudaMemcpy(d, src.data(), sizeof(T) * src.size(), cudaMemcpyHostToDevice);
  *dst = d;
  return e;
}

}  // namespace

extern "C" {

b2b_status b2b_hines_create(b2b_net* net, int32_t n_neurons, const int64_t* comp_off,
                            const int32_t* sec_off, const int32_t* sec_start,
                            const int32_t* sec_end, const int32_t* sec_parent,
                            const double* diameter, const double* length,
                            const b2b_hines_params* p, b2b_hines** out) {
  if (!net || !out || !p || n_neurons <= 0 || !comp_off || !sec_off || !sec_start || !sec_end ||
      !sec_parent || !diameter || !length)
    return B2B_ERR_INVALID_ARG;
  if (p->channel_dtype != B2B_F32 && p->channel_dtype != B2B_F64) return B2B_ERR_INVALID_ARG;
  if (!(p->Cm > 0) || !(p->Ri > 0)) return B2B_ERR_INVALID_ARG;
  if (cudaSetDevice(net->cfg.device) != cudaSuccess) return B2B_ERR_CUDA;
  *out = nullptr;
  const double dt = net->cfg.dt;
  try {
    if (comp_off[0] != 0 || sec_off[0] != 0) return B2B_ERR_INVALID_ARG;
    const int64_t n_comp = comp_off[n_neurons];
    const int32_t n_sec = sec_off[n_neurons];
    std::vector<double> low(n_comp, 0.0), diag(n_comp, 0.0), upr(n_comp, 0.0);
    std::vector<int32_t> soc(n_comp), sst(n_sec), sen(n_sec), spn(n_sec);
    std::vector<double> g0(n_sec), gn(n_sec), rfirst(n_sec), rlast(n_sec);
    std::vector<int32_t> child_off, child_sec, more_rec, level_off, lvl_base;
    std::vector<int4> level_rec;
    // r: cross section over half the length; g: axial conductance into c from c - 1
    std::vector<double> area(n_comp), rl(n_comp), g(n_comp + 1, 0.0);
    std::vector<double> soma_area(n_neurons);
    std::vector<int> nlev_of(n_neurons, 0);
    int nc_max = 0, ns_max = 0, nlev_max = 0;
    const double Ri = p->Ri, Cm = p->Cm;
    for (int b = 0; b < n_neurons; ++b) {
      const int64_t c0 = comp_off[b], c1 = comp_off[b + 1];
      const int s0 = sec_off[b], s1 = sec_off[b + 1];
      const int nc = (int)(c1 - c0), ns = s1 - s0;
      if (nc <= 0 || ns <= 0 || nc > (1 << 20)) return B2B_ERR_INVALID_ARG;
      // 16-bit node and edge indices; so many sections exceed a CTA's shared memory anyway
      if (ns >= 32766) return B2B_ERR_UNSUPPORTED;
      nc_max = std::max(nc_max, nc);
      ns_max = std::max(ns_max, ns);
      // morphology checks: sections contiguous, in topological order, root first
      if (sec_start[s0] != 0 || sec_parent[s0] != -1 || sec_end[s1 - 1] != nc)
        return B2B_ERR_INVALID_ARG;
      for (int s = 0; s < ns; ++s) {
        if (sec_end[s0 + s] <= sec_start[s0 + s]) return B2B_ERR_INVALID_ARG;
        if (s > 0 && sec_start[s0 + s] != sec_end[s0 + s - 1]) return B2B_ERR_INVALID_ARG;
        if (s > 0 && (sec_parent[s0 + s] < 0 || sec_parent[s0 + s] >= s)) return B2B_ERR_INVALID_ARG;
      }
      for (int64_t c = c0; c < c1; ++c) {
        if (!(diameter[c] > 0) || !(length[c] > 0)) return B2B_ERR_INVALID_ARG;
        area[c] = M_PI * diameter[c] * length[c];
        rl[c] = M_PI * diameter[c] * diameter[c] / (2.0 * length[c]);
      }
      soma_area[b] = area[c0];
      // matrix rows (the cable matrix of spatialstateupdate.cu:36-77)
      std::vector<char> first_of_sec(nc, 0);
      for (int s = 0; s < ns; ++s) first_of_sec[sec_start[s0 + s]] = 1;
      for (int64_t c = c0; c < c1; ++c)
        g[c] = first_of_sec[c - c0] ? 0.0 : 1.0 / (Ri * (1.0 / rl[c - 1] + 1.0 / rl[c]));
      g[c1] = 0.0;
      for (int64_t c = c0; c < c1; ++c) {
        low[c] = g[c] / area[c];
        upr[c] = g[c + 1] / area[c];
        diag[c] = -(Cm / dt) - (g[c] + g[c + 1]) / area[c];
      }
      for (int s = 0; s < ns; ++s) {
        const int64_t first = c0 + sec_start[s0 + s];
        const int64_t last = c0 + sec_end[s0 + s] - 1;
        g0[s0 + s] = rl[first] / Ri;
        gn[s0 + s] = rl[last] / Ri;
        diag[first] -= g0[s0 + s] / area[first];
        diag[last] -= gn[s0 + s] / area[last];
        rfirst[s0 + s] = -g0[s0 + s] / area[first];
        rlast[s0 + s] = -gn[s0 + s] / area[last];
        sst[s0 + s] = sec_start[s0 + s];
        sen[s0 + s] = sec_end[s0 + s];
        spn[s0 + s] = s == 0 ? 0 : sec_parent[s0 + s] + 1;
        for (int64_t c = first; c <= last; ++c) soc[c] = s;
      }
      // nodes: node 0 = sealed start of the root, node s+1 = end of section s
      const int nB = ns + 1;
      std::vector<std::vector<int>> kids(nB);
      kids[0].push_back(0);
      for (int s = 1; s < ns; ++s) kids[spn[s0 + s]].push_back(s);
      std::vector<int> depth(nB, 0);
      for (int s = 0; s < ns; ++s) depth[s + 1] = depth[spn[s0 + s]] + 1;
      const int edge_base = (int)child_sec.size();
      std::vector<int> first_edge(nB + 1);
      for (int i = 0; i < nB; ++i) {
        child_off.push_back((int)child_sec.size());
        first_edge[i] = (int)child_sec.size() - edge_base;
        for (int s : kids[i]) child_sec.push_back(s);
      }
      first_edge[nB] = (int)child_sec.size() - edge_base;
      std::vector<int> order(nB);
      for (int i = 0; i < nB; ++i) order[i] = i;
      std::stable_sort(order.begin(), order.end(), [&](int a, int c) { return depth[a] < depth[c]; });
      lvl_base.push_back((int)level_off.size());
      for (int i : order) {
        const std::vector<int>& ch = kids[i];
        const int ca = ch.size() > 0 ? ch[0] + 1 : nB, cb = ch.size() > 1 ? ch[1] + 1 : nB;
        const int more = std::min(first_edge[i] + 2, first_edge[i + 1]);
        level_rec.push_back(
            make_int4(16 * i, 16 * ca, 16 * cb, i == 0 ? 0 : 16 * spn[s0 + i - 1]));
        more_rec.push_back(more | first_edge[i + 1] << 16);
      }
      // groups of at most 32 nodes (one per lane of the warp that walks them) of one depth
      int groups = 0;
      for (int k = 0; k < nB; ++groups) {
        level_off.push_back(k);
        const int first = k;
        while (k < nB && k - first < 32 && depth[order[k]] == depth[order[first]]) ++k;
      }
      level_off.push_back(nB);
      nlev_of[b] = groups;
      nlev_max = std::max(nlev_max, groups);
    }
    child_off.push_back((int)child_sec.size());
    lvl_base.push_back((int)level_off.size());

    const int rc = p->channel_dtype == B2B_F32 ? 4 : 8;
    // neurons beyond the register variants' size put the whole batch on the general one
    const bool in_regs = nc_max <= kHinesMaxInRegs;
    int sms = kNumSMs;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, net->cfg.device);
    const bool one_per_sm = n_neurons <= sms;   // latency alone counts: wide CTAs, one class
    const size_t smem = hines_smem(nc_max, ns_max, nlev_max, rc, in_regs);
    int dev_smem = 0;
    cudaDeviceGetAttribute(&dev_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, net->cfg.device);
    if ((int64_t)smem > dev_smem) return B2B_ERR_UNSUPPORTED;

    b2b_hines* h = new b2b_hines();
    h->net = net;
    h->channel_dtype = p->channel_dtype;
    h->n_comp = n_comp;
    h->n_neurons = n_neurons;
    h->smem = smem;
    h->soma_area = soma_area;
    HinesDev& D = h->dev;
    D.n_neurons = n_neurons;
    D.nc_max = nc_max;
    D.ns_max = ns_max;
    D.nlev_max = nlev_max;
    D.Cm = Cm; D.dt = dt; D.El = p->El; D.EK = p->EK; D.ENa = p->ENa; D.gl = p->gl;
    D.gNa = p->gNa; D.gK = p->gK; D.Vthr = p->Vthr;
    std::vector<int64_t> co(comp_off, comp_off + n_neurons + 1);
    std::vector<int32_t> so(sec_off, sec_off + n_neurons + 1);
    cudaError_t e = cudaSuccess;
    auto up = [&](auto** dst, const auto& src) {
      if (e == cudaSuccess) e = upload(h, dst, src);
    };
    up(&D.comp_off, co); up(&D.sec_off, so); up(&D.lvl_base, lvl_base);
    up(&D.low, low); up(&D.diag, diag); up(&D.up, upr); up(&D.sec_of_comp, soc);
    up(&D.sec_start, sst); up(&D.sec_end, sen); up(&D.sec_pnode, spn);
    up(&D.g0, g0); up(&D.gn, gn); up(&D.rhs_first, rfirst); up(&D.rhs_last, rlast);
    up(&D.child_off, child_off); up(&D.child_sec, child_sec);
    up(&D.level_rec, level_rec); up(&D.more_rec, more_rec); up(&D.level_off, level_off);
    // cost of a neuron's step: the node system walks its levels on one warp, the
    // compartment-parallel phases grow with its size
    std::vector<int32_t> order(n_neurons);
    std::vector<double> cost(n_neurons);
    for (int b = 0; b < n_neurons; ++b) {
      order[b] = b;
      cost[b] = 1000.0 * (lvl_base[b + 1] - lvl_base[b] - 1) +
                15.0 * (double)(comp_off[b + 1] - comp_off[b]);
    }
    // two classes by shared-memory image: those that fit five CTAs per SM (whose registers allow
    // four), and the rest; each class in decreasing order of cost, the large class first
    int sm_bytes = 0, reserved = 0;
    cudaDeviceGetAttribute(&sm_bytes, cudaDevAttrMaxSharedMemoryPerMultiprocessor, net->cfg.device);
    cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, net->cfg.device);
    const size_t small_cap = sm_bytes > 0 ? (size_t)(sm_bytes / kHinesSmallCtas - reserved) : 0;
    std::vector<char> small(n_neurons, 0);
    int n_small = 0;
    for (int b = 0; b < n_neurons; ++b) {
      const int nc = (int)(comp_off[b + 1] - comp_off[b]), ns = sec_off[b + 1] - sec_off[b];
      small[b] = hines_smem(nc, ns, nlev_of[b], rc, in_regs) <= small_cap ? 1 : 0;
      n_small += small[b];
    }
    if (n_small == 0 || n_small == n_neurons || smem <= small_cap || one_per_sm)
      std::fill(small.begin(), small.end(), 0);   // one class, one launch
    std::stable_sort(order.begin(), order.end(), [&](int32_t a, int32_t c) {
      if (small[a] != small[c]) return small[a] < small[c];
      return cost[a] > cost[c];
    });
    int n_large = 0, ncs = 0, nss = 0, nls = 0, ncl = 0, nsl = 0, nll = 0;
    for (int b = 0; b < n_neurons; ++b) {
      const int nc = (int)(comp_off[b + 1] - comp_off[b]), ns = sec_off[b + 1] - sec_off[b];
      if (small[b]) {
        ncs = std::max(ncs, nc); nss = std::max(nss, ns); nls = std::max(nls, nlev_of[b]);
      } else {
        ++n_large;
        ncl = std::max(ncl, nc); nsl = std::max(nsl, ns); nll = std::max(nll, nlev_of[b]);
      }
    }
    up(&D.order, order);
    h->n_large = n_large;
    if (n_large < n_neurons) {
      // the large class's image bounds its own arrays; the small class has its own bounds
      D.nc_max = ncl; D.ns_max = nsl; D.nlev_max = nll;
      h->smem = hines_smem(ncl, nsl, nll, rc, in_regs);
      h->smem_small = hines_smem(ncs, nss, nls, rc, in_regs);
      if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&h->stream2, cudaStreamNonBlocking);
      if (e == cudaSuccess) e = cudaEventCreateWithFlags(&h->ev_fork, cudaEventDisableTiming);
      if (e == cudaSuccess) e = cudaEventCreateWithFlags(&h->ev_join, cudaEventDisableTiming);
    }
    std::vector<double> zeros_d(n_comp, 0.0), zero_I(n_neurons, 0.0);
    std::vector<int32_t> zeros_i(n_neurons, 0);
    const double* cv = nullptr;
    up(&cv, zeros_d); D.v = const_cast<double*>(cv);
    up(&cv, zeros_d); D.Ic = const_cast<double*>(cv);
    up(&D.soma_I, zero_I);
    const int32_t* ci = nullptr;
    up(&ci, zeros_i); D.spikes = const_cast<int32_t*>(ci);
    up(&ci, zeros_i); D.above = const_cast<int32_t*>(ci);
    for (void** g : {&D.m, &D.h, &D.n}) {
      if (e != cudaSuccess) break;
      e = cudaMalloc(g, rc * std::max<int64_t>(n_comp, 1));
      if (e == cudaSuccess) { h->allocs.push_back(*g); e = cudaMemset(*g, 0, rc * n_comp); }
    }
    if (n_large < n_neurons) {
      // the small class: the same arrays, its own bounds and its part of the order
      h->dev_small = D;
      h->dev_small.nc_max = ncs; h->dev_small.ns_max = nss; h->dev_small.nlev_max = nls;
      h->dev_small.order = D.order + n_large;
    }
    // in a batch of the general variant both classes run it
    auto pick = [&](int nc) {
      if (!in_regs) nc = nc_max;
      return rc == 4 ? hines_variant<float>(nc, one_per_sm) : hines_variant<double>(nc, one_per_sm);
    };
    h->var = pick(D.nc_max);
    h->var_small = pick(n_large < n_neurons ? ncs : D.nc_max);
    // the limit is a property of the kernel, shared by every batch that runs it: the device's
    for (HinesKernel k : {h->var.kern, h->var_small.kern})
      if (e == cudaSuccess)
        e = cudaFuncSetAttribute((const void*)k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 dev_smem);
    if (e != cudaSuccess) {
      b2b_hines_destroy(h);
      return e == cudaErrorMemoryAllocation ? B2B_ERR_OOM : B2B_ERR_CUDA;
    }
    net->hines.push_back(h);
    *out = h;
    return B2B_OK;
  } catch (const std::bad_alloc&) {
    return B2B_ERR_OOM;
  }
}

b2b_status b2b_hines_set_current(b2b_hines* h, const double* soma_current) {
  if (!h) return B2B_ERR_INVALID_ARG;
  std::vector<double> I(h->n_neurons, 0.0);
  if (soma_current)
    for (int b = 0; b < h->n_neurons; ++b) I[b] = soma_current[b] / h->soma_area[b];
  cudaSetDevice(h->net->cfg.device);
  cudaError_t e = cudaMemcpy(const_cast<double*>(h->dev.soma_I), I.data(), 8 * I.size(),
                             cudaMemcpyHostToDevice);
  return e == cudaSuccess ? B2B_OK : B2B_ERR_CUDA;
}

static void* hines_var(b2b_hines* h, int32_t var, size_t* es) {
  const size_t rc = h->channel_dtype == B2B_F32 ? 4 : 8;
  switch (var) {
    case 0: *es = 8; return h->dev.v;
    case 1: *es = rc; return h->dev.m;
    case 2: *es = rc; return h->dev.h;
    case 3: *es = rc; return h->dev.n;
    case 4: *es = 8; return h->dev.Ic;
    default: return nullptr;
  }
}

b2b_status b2b_hines_state_set(b2b_hines* h, int32_t var, const void* host, int64_t n) {
  if (!h || !host || n != h->n_comp) return B2B_ERR_INVALID_ARG;
  size_t es = 0;
  void* d = hines_var(h, var, &es);
  if (!d) return B2B_ERR_INVALID_ARG;
  cudaSetDevice(h->net->cfg.device);
  cudaStreamSynchronize(h->net->stream);
  return cudaMemcpy(d, host, es * n, cudaMemcpyHostToDevice) == cudaSuccess ? B2B_OK : B2B_ERR_CUDA;
}

b2b_status b2b_hines_state_get(b2b_hines* h, int32_t var, void* host, int64_t n) {
  if (!h || !host || n != h->n_comp) return B2B_ERR_INVALID_ARG;
  size_t es = 0;
  void* d = hines_var(h, var, &es);
  if (!d) return B2B_ERR_INVALID_ARG;
  cudaSetDevice(h->net->cfg.device);
  return read_array(h->net, host, d, es * n) == cudaSuccess ? B2B_OK : B2B_ERR_CUDA;
}

b2b_status b2b_hines_run(b2b_hines* h, int64_t n_steps) {
  if (!h || n_steps < 0) return B2B_ERR_INVALID_ARG;
  cudaSetDevice(h->net->cfg.device);
  while (n_steps > 0) {
    const int k = (int)std::min<int64_t>(n_steps, kHinesMaxStepsPerLaunch);
    const int wc = n_steps == k ? 1 : 0;
    cudaStream_t s = h->net->stream;
    const bool two = h->n_large < h->n_neurons;
    if (two) {
      if (cudaEventRecord(h->ev_fork, s) != cudaSuccess) return B2B_ERR_CUDA;
      if (cudaStreamWaitEvent(h->stream2, h->ev_fork, 0) != cudaSuccess) return B2B_ERR_CUDA;
    }
    if (h->n_large > 0)
      h->var.kern<<<h->n_large, h->var.block, h->smem, s>>>(h->dev, k, wc);
    if (two)
      h->var_small.kern<<<h->n_neurons - h->n_large, h->var_small.block, h->smem_small,
                          h->stream2>>>(h->dev_small, k, wc);
    if (cudaGetLastError() != cudaSuccess) return B2B_ERR_CUDA;
    if (two) {
      if (cudaEventRecord(h->ev_join, h->stream2) != cudaSuccess) return B2B_ERR_CUDA;
      if (cudaStreamWaitEvent(s, h->ev_join, 0) != cudaSuccess) return B2B_ERR_CUDA;
    }
    h->net->launches += two ? 2 : 1;
    n_steps -= k;
  }
  return B2B_OK;
}

b2b_status b2b_hines_spike_counts(b2b_hines* h, int32_t* host, int32_t n) {
  if (!h || !host || n != h->n_neurons) return B2B_ERR_INVALID_ARG;
  cudaSetDevice(h->net->cfg.device);
  cudaStreamSynchronize(h->net->stream);
  return cudaMemcpy(host, h->dev.spikes, 4 * (size_t)n, cudaMemcpyDeviceToHost) == cudaSuccess
             ? B2B_OK
             : B2B_ERR_CUDA;
}

b2b_status b2b_hines_destroy(b2b_hines* h) {
  if (!h) return B2B_ERR_INVALID_ARG;
  if (h->net) {
    cudaSetDevice(h->net->cfg.device);
    auto& v = h->net->hines;
    v.erase(std::remove(v.begin(), v.end(), h), v.end());
  }
  if (h->stream2) {
    cudaStreamSynchronize(h->stream2);
    cudaStreamDestroy(h->stream2);
  }
  if (h->ev_fork) cudaEventDestroy(h->ev_fork);
  if (h->ev_join) cudaEventDestroy(h->ev_join);
  for (void* a : h->allocs) cudaFree(a);
  delete h;
  return B2B_OK;
}

}  // extern "C"

// ---- the solver's reciprocal and quotients against the IEEE ones --------------------------------
namespace b2b {
namespace {
__global__ void recip_selftest_kernel(const double* __restrict__ x, double* __restrict__ y,
                                      int64_t n) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    y[i] = recip(x[i]);
}
// x / c for the which-th of the rates' constants.
template <typename RC>
__global__ void div_selftest_kernel(int which, const RC* __restrict__ x, RC* __restrict__ y,
                                    int64_t n) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    y[i] = which == 0   ? div_lit<RC>(x[i], 10e-3)
           : which == 1 ? div_lit<RC>(x[i], 18e-3)
           : which == 2 ? div_lit<RC>(x[i], 20e-3)
                        : div_lit<RC>(x[i], 80e-3);
}
}  // namespace
}  // namespace b2b

namespace {
// y[0..n) from x[0..n), host arrays of `es` bytes an element, by launch(device x, device y).
template <class Launch>
b2b_status run_selftest(int32_t device, const void* x, void* y, size_t es, int64_t n,
                        Launch launch) {
  if (!x || !y || n <= 0) return B2B_ERR_INVALID_ARG;
  int prev = -1;
  if (cudaGetDevice(&prev) != cudaSuccess || cudaSetDevice(device) != cudaSuccess)
    return B2B_ERR_CUDA;
  void *dx = nullptr, *dy = nullptr;
  cudaError_t e = cudaMalloc(&dx, es * n);
  if (e == cudaSuccess) e = cudaMalloc(&dy, es * n);
  if (e == cudaSuccess) e = cudaMemcpy(dx, x, es * n, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    launch(dx, dy);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(y, dy, es * n, cudaMemcpyDeviceToHost);
  if (dx) cudaFree(dx);
  if (dy) cudaFree(dy);
  cudaSetDevice(prev);
  return e == cudaSuccess ? B2B_OK : B2B_ERR_CUDA;
}
}  // namespace

extern "C" b2b_status b2b_recip_selftest(int32_t device, const double* x, double* y,
                                         int64_t n) {
  return run_selftest(device, x, y, sizeof(double), n, [&](void* dx, void* dy) {
    b2b::recip_selftest_kernel<<<256, 256>>>(static_cast<double*>(dx), static_cast<double*>(dy),
                                             n);
  });
}

extern "C" b2b_status b2b_div_selftest(int32_t device, int32_t dtype, int32_t which, const void* x,
                                       void* y, int64_t n) {
  if (which < 0 || which > 3 || (dtype != B2B_F32 && dtype != B2B_F64))
    return B2B_ERR_INVALID_ARG;
  return run_selftest(device, x, y, dtype == B2B_F32 ? 4 : 8, n, [&](void* dx, void* dy) {
    if (dtype == B2B_F32)
      b2b::div_selftest_kernel<<<256, 256>>>(which, static_cast<float*>(dx),
                                             static_cast<float*>(dy), n);
    else
      b2b::div_selftest_kernel<<<256, 256>>>(which, static_cast<double*>(dx),
                                             static_cast<double*>(dy), n);
  });
}
