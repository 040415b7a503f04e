// The CG iterations between two reliable updates as one persistent cooperative kernel.
//
// On a small lattice an iteration of the batched solver is nine dependent launches (four hops, two reduction
// finalizers, the decision and bookkeeping kernels, p = r + beta p) of 2.4-10 us each, of which the arithmetic is a
// fraction: at 8^4 with 12 FP16 right-hand sides an iteration took 51 us for hops of 5-7 us, at 12^3x24 in FP64 65 us
// for hops of 15 us.  Here one block per SM runs the iterations in a loop: a hop is a sweep over the block's share of
// the sites, launches become grid barriers, and the scalars of the iteration (alpha, beta, the reliable-update
// decision) are computed by every block from the block partials in the same fixed order, so that all blocks take the
// same branch and only block 0 writes the state back.  The kernel returns as soon as a slot asks for a reliable
// update (or nothing is active any more); the update and its bookkeeping run as the ordinary kernels, and the WHILE
// node of the solve graph launches the kernel again.
//
// The arithmetic of a site is that of the ordinary kernels (hop_fast_kernel, hop_pair_kernel, hop_lanes_kernel and
// their epilogues); the reductions add block partials in another grouping.  Fields are read with ordinary loads
// (SpinorField<P, false>): the phases read what other blocks wrote before a barrier.
//
// Barriers: one counter that every block increments once per barrier, zeroed before the launch; all blocks are
// resident (cooperative launch, one block per SM).  Every wait has an iteration limit; a block whose wait runs out
// sets *err, deactivates all slots and returns, so that the remaining waits run out too.  Launches that find *err set
// deactivate all slots and do nothing else, which ends the solve's loop; wl_solve then starts the solve again with the
// ordinary launches.
// Measured (B200, whole solves to 1e-12, ordinary launches -> this kernel): 12 point sources on 8^4 in FP16 3.97 ->
// 2.66 ms (links staged every sweep 2.93), one even-odd FP32 solve at 16^3x32 10.8 -> 9.1 ms, plain FP64 CG at
// 12^3x24 23.3 -> 20.4 ms, an MD update at 16^3x32 (full-lattice FP32 solve) 11.9 -> 8.6 ms.  What is left of an
// iteration at 16^3x32 is four hops at the L2's rate and latency, five barriers of 1.5-2.6 us and the FP64 updates.
// Measured and not kept: the loads of two (FP32) or four (FP16) hops issued together (spills; 9.8 against 9.5 ms).
#pragma once
#include "wl_site.cuh"

namespace wl {

constexpr int kPersistMaxSlots = 16;
constexpr int kPersistPolls = 1 << 21;  // limit of the polls of one barrier wait (about a microsecond each)

enum PersistKind { PK_SITE = 0, PK_PAIR = 1, PK_LANES = 2 };

template <int S, class LS>
struct PersistArgs {
  Geom g;
  LS links;
  // fields and epilogues stay in parameter space: built in the kernel they would be indexed in local memory
  SpinorField<S, false> p[2], t1[2], y[2], rs[2];
  EpiXpay<SpinorField<S, false>, false> et;  // t1 = -1/2 hop
  EpiXpay<SpinorField<S, false>, true> ey;   // y = M p (D p), |y|^2
  EpiCG<SpinorField<S, false>> ec;           // reads alpha below: r2 = alpha, pAp = 1 for the unpacked forms
  FUpdateP<SpinorField<S, false>> fu;        // reads beta below
  CGScalars sc;
  double *alpha, *beta;  // [n]; every block writes the same values before its own threads read them
  double* partials;  // [2][n][gridDim.x]
  unsigned* arrived; // barrier arrivals of this launch, zero before it
  int* err;
  int n;             // slots, <= kPersistMaxSlots
  int group;
  int polls;         // limit of one barrier wait
  int per;           // sites (PK_SITE, PK_PAIR: whole warps) or warp tiles (PK_LANES) per block
};

struct PersistState {
  double r2[kPersistMaxSlots], rmax2[kPersistMaxSlots], stop2[kPersistMaxSlots];
  double pap[kPersistMaxSlots], r2n[kPersistMaxSlots], beta[kPersistMaxSlots];
  int active[kPersistMaxSlots], iters[kPersistMaxSlots], maxiter[kPersistMaxSlots], status[kPersistMaxSlots];
  int ru[kPersistMaxSlots];
  int go;
  double wsum[32][kPersistMaxSlots + 1];  // per warp and slot: reduced values of the current sweep
};

// One grid barrier; false if its wait ran out.  `target`: arrivals expected by now (kept by the caller).
WL_D bool grid_barrier(unsigned* arrived, unsigned& target, int limit, PersistState& st) {
  target += gridDim.x;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();  // this block's writes (ordered before by the block barrier) are visible before its arrival
    atomicAdd(arrived, 1u);
    unsigned seen = 0;
    int polls = 0;
    do {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(arrived) : "memory");
    } while (seen < target && ++polls < limit);
    st.go = seen >= target;
    __threadfence();
  }
  __syncthreads();
  return st.go != 0;
}

// out[s] = sum over blocks of partials[s][block] for the active slots, in a fixed order (every block gets the same bits)
WL_D void persist_sum(const double* partials, int n, const PersistState& st, double* out) {
  const int lane = threadIdx.x & 31;
  for (int s = threadIdx.x >> 5; s < n; s += blockDim.x >> 5) {
    if (!st.active[s]) continue;
    double v = 0.0;
    for (int b = lane; b < (int)gridDim.x; b += 32) v += __ldcg(partials + (size_t)s * gridDim.x + b);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0) out[s] = v;
  }
  __syncthreads();
}

// Copies whose strides the optimiser cannot see through, made once per site: the addresses k * stride of a stencil are
// then formed where they are used instead of being hoisted out of the sweeps into registers.
template <class SF> WL_D SF opaque_field(const SF& f) {
  SF o = f;
  asm volatile("" : "+r"(o.kstride));
  return o;
}
template <class LF> WL_D LF opaque_links(const LF& l) {
  LF o = l;
  asm volatile("" : "+r"(o.vh));
  return o;
}

// ---------------------------------------------------------------- sweeps
// A sweep covers the block's share of the target sites (parity0 for npar = 1, both parities for npar = 2) and all
// active slots: its warps take (slot, group of sites) items in turn, so that several slots of a small lattice run side
// by side.  One hop through epilogue `epi`; with EPI::kReduce each item's sum goes to st.wsum and the block's sum per
// slot to partials[slot][block], both in a fixed order.

WL_D void sweep_begin(PersistState& st) {
  const int lane = threadIdx.x & 31;
  if (lane < kPersistMaxSlots) st.wsum[threadIdx.x >> 5][lane] = 0.0;
  __syncwarp();
}
// v: this lane's value of an item of slot rhs (uniform per warp)
WL_D void sweep_add(PersistState& st, int rhs, double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) st.wsum[threadIdx.x >> 5][rhs] += v;
}
WL_D void sweep_end(const PersistState& st, int n, double* partials) {
  __syncthreads();
  const int lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  for (int s = threadIdx.x >> 5; s < n; s += warps) {
    double v = lane < warps ? st.wsum[lane][s] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0) partials[(size_t)s * gridDim.x + blockIdx.x] = v;
  }
}

// The items of a block for W sites per warp: calls f(slot, index of the warp's first site, end of the block's share)
template <int W, class A_, class F>
WL_D void for_items(const A_& A, int npar, const PersistState& st, const F& f) {
  const int begin = blockIdx.x * A.per, end = min(begin + A.per, npar * A.g.Vh);
  const int groups = (end - begin + W - 1) / W, warps = blockDim.x >> 5;
  // the slot is a loop variable, uniform over the block, so that addresses keep their slot part in uniform registers;
  // each slot's first group goes to the warp after the one that got the previous slot's last
  int skew = 0;
#pragma unroll 1
  for (int rhs = 0; rhs < A.n; ++rhs) {
    if (!st.active[rhs]) continue;
    int k = (int)(threadIdx.x >> 5) - skew;
    if (k < 0) k += warps;
#pragma unroll 1
    for (; k < groups; k += warps) f(rhs, begin + k * W, end);
    skew = (skew + groups) % warps;
  }
}

template <bool DAG, class A_, class SF, class EPI>
WL_D void sweep_site(const A_& A, const SF (&src)[2], int parity0, int npar, const EPI& epi, PersistState& st,
                     double* partials) {
  const Geom& g = A.g;
  if (EPI::kReduce) sweep_begin(st);
  for_items<32>(A, npar, st, [&](int rhs, int first, int end) {
    const int i = first + (int)(threadIdx.x & 31);
    double v = 0.0;
    if (i < end) {
      const int second = npar == 2 && i >= g.Vh, parity = parity0 ^ second, c = i - second * g.Vh;
      const Site s = site_from_compact(g, parity, c);
      const bool act[1] = {true};
      const auto links = opaque_links(A.links);
      const SF from = opaque_field(src[1 - parity]);
      float2 acc[1][12];
#pragma unroll
      for (int k = 0; k < 12; ++k) acc[0][k] = f2(0.f, 0.f);
      hop_dir_fast<0, DAG, 1>(g, links, from, parity, s, rhs, act, acc);
      hop_dir_fast<1, DAG, 1>(g, links, from, parity, s, rhs, act, acc);
      hop_dir_fast<2, DAG, 1>(g, links, from, parity, s, rhs, act, acc);
      hop_dir_fast<3, DAG, 1>(g, links, from, parity, s, rhs, act, acc);
      Spinor<float> o;
#pragma unroll
      for (int k = 0; k < 12; ++k) o.v[k / 3][k % 3] = {acc[0][k].x, acc[0][k].y};
      v = epi(rhs, parity, (long long)c, o);
    }
    if (EPI::kReduce) sweep_add(st, rhs, v);
  });
  if (EPI::kReduce) sweep_end(st, A.n, partials);
}

template <bool DAG, class A_, class SF, class EPI>
WL_D void sweep_pair(const A_& A, const SF (&src)[2], int parity0, int npar, const EPI& epi, PersistState& st,
                     double* partials) {
  using T = typename SF::real;
  const Geom& g = A.g;
  const int j = threadIdx.x & 1;
  if (EPI::kReduce) sweep_begin(st);
  for_items<16>(A, npar, st, [&](int rhs, int first, int end) {
    const int i = first + (int)((threadIdx.x & 31) >> 1);
    const bool act = i < end;
    const int second = npar == 2 && i >= g.Vh, parity = parity0 ^ second, c = i - second * g.Vh;
    Site s{};
    if (act) s = site_from_compact(g, parity, c);
    cplx<T> o[2][3];
    pair_stencil<DAG>(g, opaque_links(A.links), opaque_field(src[1 - parity]), parity, s, rhs, j, act, o);
    const double v = epi.half(rhs, parity, (unsigned)s.c, j, act, o);
    if (EPI::kReduce) sweep_add(st, rhs, v);
  });
  if (EPI::kReduce) sweep_end(st, A.n, partials);
}

// A warp tile: 32 / R sites x R right-hand sides, its links staged by the warp as in hop_lanes_kernel.
template <int R>
struct WarpLinks {
  SiteLinks link[32 / R];
  int nb[32 / R][8];
};

template <bool DAG, int R, bool HC, bool HA, class A_, class SF, class EPI>
WL_D void sweep_lanes(const A_& A, const SF (&src)[2], int parity0, int npar, const EPI& epi, PersistState& st,
                      double* partials, WarpLinks<R>* links, bool staged) {
  constexpr int SPW = 32 / R;
  const Geom& g = A.g;
  const int lane = threadIdx.x & 31;
  const int groups = (A.n + R - 1) / R, tiles1 = ((g.Vh + SPW - 1) / SPW) * groups;
  const int end = min((int)(blockIdx.x + 1) * A.per, npar * tiles1);
  if (EPI::kReduce) sweep_begin(st);
#pragma unroll 1
  for (int t = blockIdx.x * A.per + (threadIdx.x >> 5); t < end; t += blockDim.x >> 5) {  // uniform per warp
    const int second = npar == 2 && t >= tiles1, parity = parity0 ^ second, tt = t - second * tiles1;
    const int sg = tt / groups, gr = tt - sg * groups, site0 = sg * SPW;
    WarpLinks<R>& L = links[R >= 8 ? parity : 0];
    if (!staged) {
      __syncwarp();
      for (int j = lane; j < 8 * SPW; j += 32) {
        const int sl = j >> 3, q = j & 7;
        if (site0 + sl < g.Vh)
          L.nb[sl][q] = stage_link<HC>(g, A.links, parity, site0 + sl, q >> 1, q & 1, L.link[sl].l[q]);
      }
      __syncwarp();
    }
    const int sl = lane / R, c = site0 + sl, rhs = gr * R + (lane % R);
    double v = 0.0;
    if (c < g.Vh && rhs < A.n && st.active[rhs]) {
      float2 acc[12];
#pragma unroll
      for (int k = 0; k < 12; ++k) acc[k] = f2(0.f, 0.f);
      lane_stencil<DAG, HC, HA>(opaque_field(src[1 - parity]), L.link[sl].l, L.nb[sl], rhs, acc);
      v = epi.packed(rhs, parity, (unsigned)c, acc);
    }
    if (EPI::kReduce) {
#pragma unroll
      for (int off = R; off < 32; off <<= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
      if (lane < R && rhs < A.n) st.wsum[threadIdx.x >> 5][rhs] += v;
    }
  }
  if (EPI::kReduce) sweep_end(st, A.n, partials);
}

// p = r + beta p on the block's share (the sites that its hops wrote)
template <int KIND, int R, class A_, class SF>
WL_D void sweep_update(const A_& A, int npar, PersistState& st, const SF&) {
  const Geom& g = A.g;
  if constexpr (KIND == PK_LANES) {
    constexpr int SPW = 32 / R;
    const int lane = threadIdx.x & 31, groups = (A.n + R - 1) / R, tiles1 = ((g.Vh + SPW - 1) / SPW) * groups;
    const int end = min((int)(blockIdx.x + 1) * A.per, npar * tiles1);
    for (int t = blockIdx.x * A.per + (threadIdx.x >> 5); t < end; t += blockDim.x >> 5) {
      const int parity = npar == 2 && t >= tiles1, tt = t - parity * tiles1, sg = tt / groups;
      const int c = sg * SPW + lane / R, rhs = (tt - sg * groups) * R + lane % R;
      if (c < g.Vh && rhs < A.n && st.active[rhs]) A.fu(rhs, parity, c);
    }
  } else if constexpr (KIND == PK_PAIR) {
    using T = typename SF::real;
    const int j = threadIdx.x & 1;
    for_items<16>(A, npar, st, [&](int rhs, int first, int end) {
      const int i = first + (int)((threadIdx.x & 31) >> 1);
      if (i >= end) return;
      const T be = T(st.beta[rhs]);
      const int parity = npar == 2 && i >= g.Vh, c = i - parity * g.Vh;
      cplx<T> r[2][3], q[2][3];
      half_load(A.rs[parity], rhs, c, j, r);
      half_load(A.p[parity], rhs, c, j, q);
#pragma unroll
      for (int s = 0; s < 2; ++s)
#pragma unroll
        for (int k = 0; k < 3; ++k) q[s][k] = r[s][k] + be * q[s][k];
      half_store(A.p[parity], rhs, c, j, true, q);
    });
  } else {
    for_items<32>(A, npar, st, [&](int rhs, int first, int end) {
      const int i = first + (int)(threadIdx.x & 31);
      if (i >= end) return;
      const int parity = npar == 2 && i >= g.Vh;
      A.fu(rhs, parity, i - parity * g.Vh);
    });
  }
}

// Link slots per warp: one per target parity where two fit, so that a warp with a single tile of each parity (the
// even-odd operator on a lattice of a few thousand sites) stages its links once per launch instead of four times an
// iteration.
constexpr int persist_slots(int R) { return R >= 8 ? 2 : 1; }

// Dynamic shared memory of a block of T threads (PK_LANES: staged links)
template <int KIND, int R, int T>
constexpr size_t persist_smem() {
  return KIND == PK_LANES ? (T / 32) * persist_slots(R) * sizeof(WarpLinks<R>) : 0;
}

// EO (the even-odd operator, four hops) and the full operator (two) are separate instantiations: sharing one function
// their sweeps were merged and spilled (FP64 600 bytes a thread against 120; solves 5-15 % slower).
template <int S, class LS, int KIND, int R, bool HC, bool HA, int T, bool EO>
__global__ void __launch_bounds__(T, 1) cg_persist_kernel(const __grid_constant__ PersistArgs<S, LS> A) {
  using SF = SpinorField<S, false>;
  extern __shared__ __align__(16) unsigned char dyn[];
  __shared__ PersistState st;
  const int tid = threadIdx.x;
  constexpr int npar = EO ? 1 : 2;
  double* part0 = A.partials;
  double* part1 = A.partials + (size_t)A.n * gridDim.x;
  bool mine = false;
  if (tid < A.n) {
    st.r2[tid] = A.sc.r2[tid];
    st.rmax2[tid] = A.sc.rmax2[tid];
    st.stop2[tid] = A.sc.tol2[tid] * A.sc.b2[tid];
    st.active[tid] = A.sc.active[tid];
    st.iters[tid] = A.sc.iters[tid];
    st.maxiter[tid] = A.sc.maxiter[tid];
    st.status[tid] = A.sc.status[tid];
    st.ru[tid] = 0;
    mine = st.active[tid] != 0 && *A.err == 0;
  }
  if (!__syncthreads_or(mine)) {  // nothing to solve, or a wait of an earlier launch ran out: the same in every block
    if (tid < A.n) A.sc.active[tid] = A.sc.ru[tid] = 0;
    return;
  }
  const bool keep = KIND == PK_LANES && R >= 8 && EO && A.per <= T / 32;
  bool staged = false;  // the links of both parities are in shared memory (from the second iteration on)
  const auto hop = [&](auto dag, const SF(&src)[2], int parity0, int np, const auto& epi, double* partials) {
    constexpr bool DAG = decltype(dag)::value;
    if constexpr (KIND == PK_LANES)
      sweep_lanes<DAG, R, HC, HA>(A, src, parity0, np, epi, st, partials,
                                  reinterpret_cast<WarpLinks<R>*>(dyn) + (threadIdx.x >> 5) * persist_slots(R),
                                  staged && keep);
    else if constexpr (KIND == PK_PAIR) sweep_pair<DAG>(A, src, parity0, np, epi, st, partials);
    else sweep_site<DAG>(A, src, parity0, np, epi, st, partials);
  };
  const std::false_type plain{};
  const std::true_type dagger{};
  unsigned target = 0;
  bool ok = true;
  for (;; staged = true) {
    // ---- y = M p (or D p), pAp = |y|^2
    if constexpr (EO) {
      hop(plain, A.p, 1, 1, A.et, nullptr);
      if (!(ok = grid_barrier(A.arrived, target, A.polls, st))) break;
      hop(plain, A.t1, 0, 1, A.ey, part0);
    } else {
      hop(plain, A.p, 0, 2, A.ey, part0);
    }
    if (!(ok = grid_barrier(A.arrived, target, A.polls, st))) break;
    persist_sum(part0, A.n, st, st.pap);
    if (tid < A.n && st.active[tid]) A.alpha[tid] = st.pap[tid] > 0.0 ? st.r2[tid] / st.pap[tid] : 0.0;
    __syncthreads();
    // ---- x_s += alpha p, r_s -= alpha M^dag y, r2n = |r_s|^2
    if constexpr (EO) {
      hop(dagger, A.y, 1, 1, A.et, nullptr);
      if (!(ok = grid_barrier(A.arrived, target, A.polls, st))) break;
      hop(dagger, A.t1, 0, 1, A.ec, part1);
    } else {
      hop(dagger, A.y, 0, 2, A.ec, part1);
    }
    if (!(ok = grid_barrier(A.arrived, target, A.polls, st))) break;
    persist_sum(part1, A.n, st, st.r2n);
    // ---- decision and bookkeeping (cg_decide_kernel, cg_finalize_kernel), the same in every block
    bool trig = false, live = false;
    if (tid < A.n && st.active[tid]) {
      const double r2n = st.r2n[tid], pap = st.pap[tid];
      if (!isfinite(r2n) || !isfinite(pap) || !(pap > 0.0)) {
        st.status[tid] = isfinite(r2n) && isfinite(pap) ? ST_BREAKDOWN : ST_NAN;
        st.active[tid] = 0;
      } else {
        trig = r2n < A.sc.delta2 * st.rmax2[tid] || r2n <= st.stop2[tid] || st.iters[tid] + 1 >= st.maxiter[tid];
        live = true;
      }
    }
    const bool any = __syncthreads_or(trig);
    if (any || !__syncthreads_or(live)) {
      if (tid < A.n) st.ru[tid] = live && (trig || A.group) ? 1 : 0;
      break;
    }
    if (live) {
      const double r2n = st.r2n[tid];
      st.rmax2[tid] = fmax(st.rmax2[tid], r2n);
      st.iters[tid] += 1;
      st.beta[tid] = A.beta[tid] = r2n / st.r2[tid];
      st.r2[tid] = r2n;
    }
    __syncthreads();
    sweep_update<KIND, R>(A, npar, st, SF{});
    if (!(ok = grid_barrier(A.arrived, target, A.polls, st))) break;
  }
  if (!ok) {  // a wait ran out: stop the solve (this launch's stores to the state are not used)
    if (tid < A.n) {
      A.sc.active[tid] = 0;
      A.sc.ru[tid] = 0;
    }
    if (tid == 0) *A.err = 1;
    return;
  }
  if (blockIdx.x == 0 && tid < A.n) {
    A.sc.ru[tid] = st.ru[tid];
    if (A.sc.active[tid]) {
      A.sc.r2[tid] = st.r2[tid];
      A.sc.rmax2[tid] = st.rmax2[tid];
      A.sc.iters[tid] = st.iters[tid];
      A.sc.r2_new[tid] = st.r2n[tid];
      A.sc.pAp[tid] = st.pap[tid];
      A.sc.status[tid] = st.status[tid];
      A.sc.active[tid] = st.active[tid];
    }
  }
}

}  // namespace wl
