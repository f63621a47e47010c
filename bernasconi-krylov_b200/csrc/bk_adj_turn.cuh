// Reverse sweep of the adjoint gradient as turning passes (sm_100a): bk_adjoint.cuh's
// method (psi and lambda through the same inverse steps, the cross terms
// Im <lambda| X_q |psi> read off the butterfly pairs before they are rotated) in the
// passes of bk_alt.cuh: one pass over both statevectors finishes reverse step j - 1 on
// its set of qubits, applies D^dagger and starts step j on the same set. A step costs
// one dual pass up to 2^21 elements (two beyond) instead of two (three), without a
// launch per pass.
//
// A CTA holds the same tile of psi and of lambda (2^12 elements each, 128 KB; 2^10 up to
// 2^18 elements) and keeps 16 elements of both per thread (255 registers, eight warps an
// SM). The cross terms of a round are weighted by (1 + t^2)^-m for the m qubits of the
// step rotated before it; a pass sums two steps' terms, one partial pair per CTA and
// pass, added up in index order by adj_cross_kernel.
//
// Measured on a B200 (reverse us a step, complex64 / complex128): N = 20 17.7 / 28.3, 22
// 64 / 128, 24 253 / 446, against 24.5 / 39, 73 / 186 and 359 / 626 for a launch per pass
// and set; bound by the latency of a tile's rounds at eight warps an SM.
#pragma once
#include "bk_adjoint.cuh"
#include "bk_alt.cuh"

namespace bk {

template <class R>
struct AdjRun {
  CUtensorMap map[2][3];  // psi, lambda: tiles of the A set and of the S sets
  AltSet set[3];
  unsigned char* vec[2];  // psi, lambda
  const uint16_t* E;
  const typename AltPhase<R>::entry* tab;
  const R* tan;        // [T] tangent of reverse step j
  const R* scale;      // [T] exact power of two applied before step j
  const double* lg;    // [T] log2(1 + t^2)
  double* partials;    // [rows][G][2]: a pass's terms of the step it finishes, of the step it starts
  uint32_t n_tiles;
  int n_j, c0;
  int m0;              // qubits rotated at the turn itself (complex64: amplitude bit 0)
  int width[3];        // qubits of each set
  int j0, j1;          // reverse steps [j0, j1)
  int row0;            // partial row of the sweep's pass 0 (a launch's passes have rows of their own)
};

template <class R>
struct AdjPhaseInv;  // D^dagger on both vectors' element
template <>
struct AdjPhaseInv<float> {
  __device__ static void apply(El<float>::T& v, El<float>::T& u, uint32_t e2, const AltTab& t) {
    const float2 H0 = *reinterpret_cast<const float2*>(t.base + (e2 & 0xFFFFu) * t.per_e);
    const float2 H1 = *reinterpret_cast<const float2*>(t.base + (e2 >> 16) * t.per_e);
    const float2 A = make_float2(-H0.x, -H1.x), B = make_float2(-H0.y, -H1.y);
    PhaseV<float>::shear2(v.re, v.im, A, B);
    PhaseV<float>::shear2(v.re, v.im, A, B);
    PhaseV<float>::shear2(u.re, u.im, A, B);
    PhaseV<float>::shear2(u.re, u.im, A, B);
  }
};
template <>
struct AdjPhaseInv<double> {
  __device__ static void apply(El<double>::T& v, El<double>::T& u, uint32_t e, const AltTab& t) {
    const double2 cs = *reinterpret_cast<const double2*>(t.base + e * t.per_e);
    v.v = make_double2(fma(v.v.x, cs.x, v.v.y * cs.y), fma(-v.v.x, cs.y, v.v.y * cs.x));
    u.v = make_double2(fma(u.v.x, cs.x, u.v.y * cs.y), fma(-u.v.x, cs.y, u.v.y * cs.x));
  }
};

struct AdjCtl {
  uint64_t full_bar;
  int stop, inflight;
  double w[16];      // round weights of the pass: [0, 4) finishing, [4, 8) starting; 8, 9: of the lane bit
  double acc[16][2];
};
template <int TB>
struct AdjTurnSmem {
  static constexpr int kLamOff = 16 << TB, kEOff = 32 << TB, kCtlOff = kEOff + (4 << TB), kTabOff = kCtlOff + 512;
  static_assert(sizeof(AdjCtl) <= 512, "the control block's room");
  static int bytes(int n_j, int entry) { return kTabOff + (((n_j + 1) * entry + 127) & ~127) + 1024; }
};

// round r's cross terms and rotations of the set's bits, on both vectors
template <class R, int TB, int KB, int LO, int r>
__device__ __forceinline__ double adj_round(typename El<R>::T (&v)[1 << KB], typename El<R>::T (&u)[1 << KB], R t,
                                            double weight, double lane_weight = 0.0) {
  constexpr int lo = AltPlan<TB, KB>::reg_lo(r);
  CrossAcc<R> ca;
#pragma unroll
  for (int k = 0; k < AltPlan<TB, KB>::act_hi(r); ++k) {
    if (lo + k >= LO) {
#pragma unroll
      for (int j = 0; j < (1 << KB); ++j)
        if (!(j & (1 << k))) ca.pair(v[j], v[j | (1 << k)], u[j], u[j | (1 << k)]);
    }
  }
  double sum = weight * ca.take();
  if constexpr (r == 1 && alt_lane_bit(TB, KB, LO)) {
    // the registers' bits, then the bit across lanes (each thread adds its own ordered term)
#pragma unroll
    for (int k = 0; k < KB; ++k) {
#pragma unroll
      for (int j = 0; j < (1 << KB); ++j)
        if (!(j & (1 << k))) {
          El<R>::bfly(v[j], v[j | (1 << k)], t);
          El<R>::bfly(u[j], u[j | (1 << k)], t);
        }
    }
#pragma unroll
    for (int j = 0; j < (1 << KB); ++j) {
      const typename El<R>::T pv = El<R>::shfl_xor(v[j], 1 << LO), pu = El<R>::shfl_xor(u[j], 1 << LO);
      ca.one(pv, u[j]);
      El<R>::bfly_partner(v[j], pv, t);
      El<R>::bfly_partner(u[j], pu, t);
    }
    sum += weight * lane_weight * ca.take();
  } else {
    alt_rotate<R, TB, KB, LO, r>(v, t);
    alt_rotate<R, TB, KB, LO, r>(u, t);
  }
  return sum;
}
// qubits of a set that round r rotates
__host__ __device__ constexpr int adj_round_bits(int TB, int KB, int LO, int r) {
  const int lo = r == 0 ? TB - KB : r == 1 ? TB - 2 * KB : 0, hi = lo + (r < 2 ? KB : TB - 2 * KB);
  return (hi <= LO ? 0 : hi - (lo > LO ? lo : LO)) + (r == 1 && alt_lane_bit(TB, KB, LO) ? 1 : 0);
}

template <class R, int TB, int KB>
struct AdjCta {
  using PL = AltPlan<TB, KB>;
  using SM = AdjTurnSmem<TB>;
  using E = El<R>;
  static constexpr uint32_t kBytes = 16u << TB;
  const AdjRun<R>& D;
  const AltBarrier& B;
  uint32_t rank, G;
  unsigned char* stage;
  uint32_t parity, epoch;

  __device__ __forceinline__ volatile AdjCtl& ctl() const { return *reinterpret_cast<volatile AdjCtl*>(stage + SM::kCtlOff); }
  __device__ __forceinline__ uint32_t bar() const { return smem_addr(stage) + SM::kCtlOff; }
  __device__ __forceinline__ unsigned char* lam() const { return stage + SM::kLamOff; }
  __device__ __forceinline__ unsigned char* es() const { return stage + SM::kEOff; }
  __device__ __forceinline__ unsigned char* tab() const { return stage + SM::kTabOff; }

  __device__ __forceinline__ void issue(int s, uint32_t tile) {
    if (threadIdx.x == 0 && tile < D.n_tiles && !ctl().stop) {
      const AltSet& S = D.set[s];
      const int mid = (int)(tile & ((1u << S.mid_bits) - 1u)), hi = (int)(tile >> S.mid_bits);
      const int md = S.mid_dim, hd = S.hi_dim;
      fence_proxy_async_shared();
      mbar_arrive_expect_tx(bar(), 2u * kBytes);
#pragma unroll
      for (int x = 0; x < 2; ++x)
        tma_load_5d(smem_addr(stage) + (x ? (uint32_t)SM::kLamOff : 0u), &D.map[x][s], tile_coord(0, md, mid, hd, hi),
                    tile_coord(1, md, mid, hd, hi), tile_coord(2, md, mid, hd, hi), tile_coord(3, md, mid, hd, hi),
                    tile_coord(4, md, mid, hd, hi), bar());
      ctl().inflight = 1;
    }
    __syncwarp();
  }
  __device__ __forceinline__ void wait() {
    for (uint32_t i = 0; i < kWaitPolls; ++i) {
      if (mbar_try_wait(bar(), parity)) {
        parity ^= 1u;
        if (threadIdx.x == 0) ctl().inflight = 0;
        return;
      }
      if (ctl().stop) return;
    }
    ctl().stop = 1;
    atomicCAS(B.err, 0, DEV_TIMEOUT);
    atomicExch(B.abort, 1);
  }
  template <int CP, int H0>
  __device__ __forceinline__ void fetch_e(uint32_t tile) {
    if (tile >= D.n_tiles) return;
    constexpr int RT = alt_turn_round(TB, KB, CP);
    AltE<R, TB, KB, CP, H0, RT>::fetch(D.E, alt_tile_base<TB, CP, H0>(tile),
                                       PL::template base<RT>(threadIdx.x & 31u, threadIdx.x >> 5), smem_addr(es()));
  }
  // the CTA's sums of a pass: [finished step, started step]
  __device__ __forceinline__ void put(int pass, double a, double b) {
    a = warp_sum(a);
    b = warp_sum(b);
    volatile double(&acc)[16][2] = ctl().acc;
    const uint32_t warp = threadIdx.x >> 5;
    if ((threadIdx.x & 31u) == 0) {
      acc[warp][0] = a;
      acc[warp][1] = b;
    }
    __syncthreads();
    if (threadIdx.x < 2u) {
      double x = 0;
      for (int w = 0; w < PL::kWarps; ++w) x += acc[w][threadIdx.x];
      D.partials[2 * ((size_t)(D.row0 + pass) * G + rank) + threadIdx.x] = x;
    }
  }

  // the turning pass that finishes step j - 1 and starts step j on set s; its partial row
  // is `pass` (with three sets the plain pass of step j has its own)
  template <int CP, int H0>
  __device__ __forceinline__ void turn(int s, int j, int pass) {
    constexpr int RT = alt_turn_round(TB, KB, CP), LO = CP == TB ? 0 : CP;
    constexpr int c0 = adj_round_bits(TB, KB, LO, 0), c1 = RT >= 1 ? adj_round_bits(TB, KB, LO, 1) : 0,
                  c2 = RT >= 2 ? adj_round_bits(TB, KB, LO, 2) : 0;
    const bool pre = j > D.j0, post = j < D.j1, phase = post && j > 0;
    const R t_pre = pre ? D.tan[j - 1] : (R)0, t_post = post ? D.tan[j] : (R)0, sc = post ? D.scale[j] : (R)1;
    // weights (1 + t^2)^-m: finishing, the step's earlier passes have rotated the rest of its qubits
    if (threadIdx.x < 8u) {
      const int i = (int)threadIdx.x & 3;
      double w = 0.0;
      if (threadIdx.x < 4u) {
        const int rotated = D.m0 + D.width[0] + D.width[1] + D.width[2] - D.width[s];
        if (pre && i < 3) w = round_weight(rotated + (i > 0 ? c0 : 0) + (i > 1 ? c1 : 0), D.lg[j - 1]);
      } else if (post) {
        // starting: amplitude bit 0 (i = 3), then the rounds from the turn back to round 0
        const int m = i == 3 ? 0 : D.m0 + (i < 2 ? c2 : 0) + (i < 1 ? c1 : 0);
        w = round_weight(m, D.lg[j]);
      }
      ctl().w[threadIdx.x] = w;
      // the lane bit of round 1 comes after its KB register bits
      if (threadIdx.x == 0u) ctl().w[8] = pre ? round_weight(KB, D.lg[j - 1]) : 0.0;
      if (threadIdx.x == 4u) ctl().w[9] = post ? round_weight(KB, D.lg[j]) : 0.0;
    }
    __syncthreads();
    const volatile double(&wt)[16] = ctl().w;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const AltTab P = alt_tab<R>(tab(), phase, (uint32_t)D.c0);
    const uint32_t b0 = PL::template base<0>(lane, warp);
    double fin = 0.0, sta = 0.0;
    unsigned char *sp = stage, *sl = lam();
    for (uint32_t tile = rank; tile < D.n_tiles; tile += G) {
      const uint32_t tile_base = alt_tile_base<TB, CP, H0>(tile);
      typename E::T v[1 << KB], u[1 << KB];
      wait();
      alt_load<R, TB, KB, 0, false>(sp, v, b0);
      alt_load<R, TB, KB, 0, false>(sl, u, b0);
      fin += adj_round<R, TB, KB, LO, 0>(v, u, t_pre, wt[0]);
      auto at_turn = [&](uint32_t base, auto round) {
        constexpr int r = decltype(round)::value;
        cp_async_wait();
#pragma unroll
        for (int q0 = 0; q0 < (1 << KB); q0 += 8) {
          uint32_t ev[8];
          AltE<R, TB, KB, CP, H0, r>::get8(es(), base, q0, ev);
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            AdjPhaseInv<R>::apply(v[q0 + q], u[q0 + q], ev[q], P);
            E::scale(v[q0 + q], sc);  // (no branch around it: 1 in most steps, and exact)
            E::scale(u[q0 + q], sc);
          }
        }
        if constexpr (sizeof(R) == 4) {
          CrossAcc<R> ca;
#pragma unroll
          for (int q = 0; q < (1 << KB); ++q) {
            ca.inner(v[q], u[q]);
            E::bfly_inner(v[q], t_post);
            E::bfly_inner(u[q], t_post);
          }
          sta += wt[7] * ca.take();
        }
        sta += adj_round<R, TB, KB, LO, r>(v, u, t_post, wt[4 + r], wt[9]);
      };
      if constexpr (RT == 0) {
        at_turn(b0, std::integral_constant<int, 0>{});
        __syncthreads();
        issue(s, tile + G);
      } else {
        __syncwarp();
        alt_store<R, TB, KB, 0>(sp, v, b0);
        alt_store<R, TB, KB, 0>(sl, u, b0);
        __syncthreads();
        const uint32_t b1 = PL::template base<1>(lane, warp);
        alt_load<R, TB, KB, 1, true>(sp, v, b1);
        alt_load<R, TB, KB, 1, true>(sl, u, b1);
        fin += adj_round<R, TB, KB, LO, 1>(v, u, t_pre, wt[1], wt[8]);
        if constexpr (RT == 1) {
          at_turn(b1, std::integral_constant<int, 1>{});
        } else {
          alt_store<R, TB, KB, 1>(sp, v, b1);
          alt_store<R, TB, KB, 1>(sl, u, b1);
          __syncwarp();
          const uint32_t b2 = PL::template base<2>(lane, warp);
          alt_load<R, TB, KB, 2, true>(sp, v, b2);
          alt_load<R, TB, KB, 2, true>(sl, u, b2);
          fin += adj_round<R, TB, KB, LO, 2>(v, u, t_pre, wt[2]);
          at_turn(b2, std::integral_constant<int, 2>{});
          alt_store<R, TB, KB, 2>(sp, v, b2);
          alt_store<R, TB, KB, 2>(sl, u, b2);
          __syncwarp();
          alt_load<R, TB, KB, 1, true>(sp, v, b1);
          alt_load<R, TB, KB, 1, true>(sl, u, b1);
          sta += adj_round<R, TB, KB, LO, 1>(v, u, t_post, wt[5], wt[9]);
        }
        alt_store<R, TB, KB, 1>(sp, v, b1);
        alt_store<R, TB, KB, 1>(sl, u, b1);
        __syncthreads();
        alt_load<R, TB, KB, 0, true>(sp, v, b0);
        alt_load<R, TB, KB, 0, true>(sl, u, b0);
        __syncthreads();
        issue(s, tile + G);
        sta += adj_round<R, TB, KB, LO, 0>(v, u, t_post, wt[4]);
      }
      const size_t g = 16ull * (tile_base | alt_index<CP, H0>(b0));
#pragma unroll
      for (int q = 0; q < (1 << KB); ++q) {
        E::st(D.vec[0] + g + 16ull * alt_index<CP, H0>((uint32_t)q << PL::reg_lo(0)), v[q]);
        E::st(D.vec[1] + g + 16ull * alt_index<CP, H0>((uint32_t)q << PL::reg_lo(0)), u[q]);
      }
      fetch_e<CP, H0>(tile + G);
    }
    put(pass, fin, sta);
  }

  // the plain pass of step j over the A set (three sets)
  __device__ __forceinline__ void plain(int j, int pass, int s_before) {
    using W = PlanA1Warp;
    const R t = D.tan[j];
    const int m = D.m0 + D.width[s_before];
    if (threadIdx.x < 3u) ctl().w[threadIdx.x] = round_weight(m + 4 * (int)threadIdx.x, D.lg[j]);
    __syncthreads();
    const volatile double(&wt)[16] = ctl().w;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t ba = pdep(lane, W::R1_LANE) | (warp << 9), bb = pdep(lane, W::R2_LANE) | (warp << 9),
                   bc = lane | (warp << 5);
    double sum = 0.0;
    unsigned char *sp = stage, *sl = lam();
    for (uint32_t tile = rank; tile < D.n_tiles; tile += G) {
      typename E::T v[16], u[16];
      CrossAcc<R> ca;
      wait();
      {
        const uint32_t sb = ba ^ ((ba >> 3) & 7u);
#pragma unroll
        for (int q = 0; q < 16; ++q) {
          const uint32_t o = pdep((uint32_t)q, W::R1_REG), at = 16u * (sb ^ o ^ ((o >> 3) & 7u));
          v[q] = E::ld(sp + at);
          u[q] = E::ld(sl + at);
        }
      }
      el_cross<R, W::R1_REG, W::R1_REG>(v, u, ca);
      sum += wt[0] * ca.take();
      el_bflys<R, W::R1_REG, W::R1_REG>(v, t);
      el_bflys<R, W::R1_REG, W::R1_REG>(u, t);
      el_store_swz<R, W::R1_REG>(sp, v, alt_fresh(ba));
      el_store_swz<R, W::R1_REG>(sl, u, alt_fresh(ba));
      __syncwarp();
      el_load<R, W::R2_REG, true>(sp, v, alt_fresh(bb));
      el_load<R, W::R2_REG, true>(sl, u, alt_fresh(bb));
      el_cross<R, W::R2_REG, W::R2_REG>(v, u, ca);
      sum += wt[1] * ca.take();
      el_bflys<R, W::R2_REG, W::R2_REG>(v, t);
      el_bflys<R, W::R2_REG, W::R2_REG>(u, t);
      el_store_swz<R, W::R2_REG>(sp, v, alt_fresh(bb));
      el_store_swz<R, W::R2_REG>(sl, u, alt_fresh(bb));
      __syncthreads();
      el_load<R, 0xF00u, true>(sp, v, bc);
      el_load<R, 0xF00u, true>(sl, u, bc);
      __syncthreads();
      issue(0, tile + G);
      el_cross<R, 0xF00u, 0xF00u>(v, u, ca);
      sum += wt[2] * ca.take();
      el_bflys<R, 0xF00u, 0xF00u>(v, t);
      el_bflys<R, 0xF00u, 0xF00u>(u, t);
      const size_t g = 16ull * (((size_t)tile << TB) | bc);
#pragma unroll
      for (int q = 0; q < 16; ++q) {
        E::st(D.vec[0] + g + 16ull * ((uint32_t)q << 8), v[q]);
        E::st(D.vec[1] + g + 16ull * ((uint32_t)q << 8), u[q]);
      }
    }
    put(pass, 0.0, sum);
  }

  __device__ __forceinline__ bool next_pass(int s) {
    if (__syncthreads_or(ctl().stop)) return false;  // every store of the CTA is issued
    if (threadIdx.x == 0) {
      red_release_add(B.ctr, 1u);
      epoch += G;
      if (!alt_wait(B, B.ctr, epoch)) ctl().stop = 1;
    }
    __syncwarp();  // (see AltCta::group_barrier)
    issue(s, rank);
    return true;
  }
  __device__ __forceinline__ void begin() {
    if (threadIdx.x == 0) {
      ctl().stop = 0;
      ctl().inflight = 0;
      mbar_init(bar(), 1);
      fence_barrier_init();
    }
    parity = epoch = 0u;
    auto* dst = reinterpret_cast<typename AltPhase<R>::entry*>(tab());
    for (int i = (int)threadIdx.x; i <= D.n_j; i += PL::kThreads) dst[i] = D.tab[i];
    __syncthreads();
  }
  __device__ __forceinline__ void leave() {
    if (threadIdx.x == 0 && ctl().stop && ctl().inflight) mbar_wait_bounded(bar(), parity, B.err);
  }
};

// W3 = 0: two sets, else three. Partial rows: two sets: pass j; three: 2 j (turning), 2 j + 1 (plain).
template <class R, int TB, int KB, int W2, int W3>
__global__ void __launch_bounds__(AltPlan<TB, KB>::kThreads, TB == 10 ? 4 : 1)
    adj_turn_kernel(const __grid_constant__ AdjRun<R> D, const __grid_constant__ AltBarrier B) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  AdjCta<R, TB, KB> C{D, B, blockIdx.x, gridDim.x, alt_stage(smem_raw)};
  C.begin();
  constexpr int C2 = TB - W2, C3 = TB - W3, H3 = TB + W2;
  if constexpr (W3 == 0) {
    if (D.j0 & 1) C.template fetch_e<C2, TB>(C.rank); else C.template fetch_e<TB, TB>(C.rank);
    C.issue(D.j0 & 1, C.rank);
    for (int j = D.j0;; ++j) {
      if (j & 1) {
        C.template turn<C2, TB>(1, j, j);
        if (j == D.j1) break;
        C.template fetch_e<TB, TB>(C.rank);
      } else {
        C.template turn<TB, TB>(0, j, j);
        if (j == D.j1) break;
        C.template fetch_e<C2, TB>(C.rank);
      }
      if (!C.next_pass((j + 1) & 1)) break;
    }
  } else {
    if (D.j0 & 1) C.template fetch_e<C3, H3>(C.rank); else C.template fetch_e<C2, TB>(C.rank);
    C.issue(1 + (D.j0 & 1), C.rank);
    for (int j = D.j0;; ++j) {
      if (j & 1)
        C.template turn<C3, H3>(2, j, 2 * j);
      else
        C.template turn<C2, TB>(1, j, 2 * j);
      if (j == D.j1 || !C.next_pass(0)) break;
      C.plain(j, 2 * j + 1, 1 + (j & 1));
      if (j & 1) C.template fetch_e<C2, TB>(C.rank); else C.template fetch_e<C3, H3>(C.rank);
      if (!C.next_pass(1 + ((j + 1) & 1))) break;
    }
  }
  C.leave();
}

#ifdef BK_ALT_REDUCE  // defined by the one source that launches it
// cross[j] = the terms of step j: those its starting pass summed (partial row row[j]), those
// of its plain pass (three sets, the next row) and those of the pass that finished it (the
// row after), CTAs in index order; one warp a step
__global__ void __launch_bounds__(128) adj_cross_kernel(const double* __restrict__ partials, int T, int G, int three,
                                                        const int* __restrict__ row, double* __restrict__ cross) {
  const int j = (int)(blockIdx.x * 4 + (threadIdx.x >> 5)), lane = (int)(threadIdx.x & 31);
  if (j >= T) return;
  const double* a = partials + 2 * (size_t)row[j] * G;
  const double* b = a + 2 * (size_t)(three ? 2 : 1) * G;
  double s = 0.0;
  for (int i = lane; i < G; i += 32) {
    s += a[2 * i + 1] + b[2 * i];
    if (three) s += a[2 * (size_t)G + 2 * i + 1];
  }
  s = warp_sum(s);
  if (lane == 0) cross[j] = s;
}
#endif

const void* adj_turn_kernel_f32(int tb, int w2, int w3);
const void* adj_turn_kernel_f64(int tb, int w2, int w3);
template <class R>
const void* adj_turn_table(int tb, int w2, int w3) {
  switch (tb * 256 + w2 * 16 + w3) {
#define BK_ADJ_CASE(key, TB, W2, W3) \
  case key: return reinterpret_cast<const void*>(adj_turn_kernel<R, TB, 4, W2, W3>)
    BK_ADJ_CASE(0xA30, 10, 3, 0);
    BK_ADJ_CASE(0xA40, 10, 4, 0);
    BK_ADJ_CASE(0xA50, 10, 5, 0);
    BK_ADJ_CASE(0xA60, 10, 6, 0);
    BK_ADJ_CASE(0xA70, 10, 7, 0);
    BK_ADJ_CASE(0xA80, 10, 8, 0);
    BK_ADJ_CASE(0xC70, 12, 7, 0);
    BK_ADJ_CASE(0xC80, 12, 8, 0);
    BK_ADJ_CASE(0xC90, 12, 9, 0);
    BK_ADJ_CASE(0xC55, 12, 5, 5);
    BK_ADJ_CASE(0xC65, 12, 6, 5);
    BK_ADJ_CASE(0xC66, 12, 6, 6);
    BK_ADJ_CASE(0xC76, 12, 7, 6);
    BK_ADJ_CASE(0xC77, 12, 7, 7);
    BK_ADJ_CASE(0xC87, 12, 8, 7);
    BK_ADJ_CASE(0xC88, 12, 8, 8);
    BK_ADJ_CASE(0xC98, 12, 9, 8);
    BK_ADJ_CASE(0xC99, 12, 9, 9);
#undef BK_ADJ_CASE
    default: return nullptr;
  }
}

}  // namespace bk
