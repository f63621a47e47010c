// Small statevectors (up to 12 qubits, complex128 — complex64 runs of these sizes
// compute in it too): every step of a run in one CTA, the state in registers.
//
// The element bits are split over the three rounds of a turning-pass tile
// (bk_alt.cuh). A step goes through the rounds once and the next one comes back:
//   [D, rounds 0 1 2][D, rounds 2 1 0][D, rounds 0 1 2] ...
// so the phase and the measurement always find the state in registers, in round 0's
// or round 2's layout, and a step costs two exchanges through shared memory, one of
// them inside a warp (rounds 1 and 2 share their warp bits): one CTA barrier a step.
// The phase coefficients of a thread's elements are the same in every step: both
// layouts' stay in registers, so D needs no energies and no table.
//
// Bound by FP64 arithmetic and the shared-memory pipe of the one SM at N = 12
// and by instruction latency at the smallest sizes. Measured on a B200 (a step without
// / with measurement): N = 12 1.8 / 2.5 us, N = 9 0.6 / 0.9 us; the former kernel, a
// shared-memory round trip and a CTA barrier per qubit, took 11.0 us at N = 12 and
// 2.6 us at N = 9 in complex64.
#pragma once
#include "bk_alt.cuh"

namespace bk {

// what step k needs: read one step ahead, so no step waits for it
struct alignas(16) SmallStep {
  double tan, scale;
  int slot;  // measurement row, or -1
  int pad;
};
struct SmallRun {
  double2* state;
  const uint16_t* E;
  const double2* tab;  // entry 0: no rotation, 1 + j: level c0 + 4 j
  const SmallStep* step;  // [steps + 1]
  double* partials;    // [rows][warps][3]
  double* results;     // [rows][4]
  int np;              // element bits (TB = 8: at most 8, the others dummies)
  int k0, k1;          // steps [k0, k1)
  int row0, rows;      // measurement rows of this launch
  int init;            // 1: start from the basis state s0, 0: from `state`
  int meas_first;      // measure psi_k0 (else an earlier launch has)
  int c0, e0;
  uint32_t s0;
};

template <int TB, int KB>
struct SmallCta {
  using PL = AltPlan<TB, KB>;
  using R = double;
  using V = El<R>::T;
  static constexpr int N = 1 << KB;

  // the rotations of round r's bits (TB = 8: those below np)
  template <int r>
  __device__ __forceinline__ static void rotate(V (&v)[N], R t, int np) {
    constexpr int lo = PL::reg_lo(r);
#pragma unroll
    for (int k = 0; k < PL::act_hi(r); ++k) {
      if (TB > 8 || lo + k < np) {
#pragma unroll
        for (int j = 0; j < N; ++j)
          if (!(j & (1 << k))) El<R>::bfly(v[j], v[j | (1 << k)], t);
      }
    }
  }
  // |psi|^2, P_< and <d_H> of the thread's elements, summed over the warp into its partial row
  __device__ __forceinline__ static void measure(const V (&v)[N], uint32_t pos, int lo, uint32_t below, uint32_t s0,
                                                 double* out) {
    double n[2] = {0, 0}, b[2] = {0, 0}, f[2] = {0, 0};
#pragma unroll
    for (int j = 0; j < N; ++j) {
      const uint32_t el = pos | ((uint32_t)j << lo);
      const int q = j & 1;
      const double w = fma(v[j].v.x, v[j].v.x, v[j].v.y * v[j].v.y);
      n[q] += w;
      b[q] += (below >> j) & 1u ? w : 0.0;
      f[q] = fma(w, alt_small(__popc(el ^ s0)), f[q]);
    }
    const double x = warp_sum(n[0] + n[1]), y = warp_sum(b[0] + b[1]), z = warp_sum(f[0] + f[1]);
    if ((threadIdx.x & 31u) == 0) {
      out[0] = x;
      out[1] = y;
      out[2] = z;
    }
  }
};

template <int TB, int KB>
__global__ void __launch_bounds__(AltPlan<TB, KB>::kThreads, 1) small_kernel(const __grid_constant__ SmallRun P) {
  using R = double;
  using C = SmallCta<TB, KB>;
  using PL = typename C::PL;
  constexpr int N = C::N, L0 = PL::reg_lo(0);
  extern __shared__ __align__(128) unsigned char tile[];
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint32_t b0 = PL::template base<0>(lane, warp), b1 = PL::template base<1>(lane, warp),
                 b2 = PL::template base<2>(lane, warp);
  const uint32_t size = TB > 8 ? 1u << TB : 1u << P.np;
  typename El<R>::T v[N];
  double2 p0[N], p2[N];  // (cos, sin) of the elements' phases in round 0's and round 2's layout
  uint32_t below0 = 0u, below2 = 0u;
#pragma unroll
  for (int j = 0; j < N; ++j) {
    const uint32_t el0 = b0 | ((uint32_t)j << L0), el2 = b2 | (uint32_t)j;
    const int ea = P.E[TB > 8 ? el0 : el0 & (size - 1u)], eb = P.E[TB > 8 ? el2 : el2 & (size - 1u)];
    p0[j] = P.tab[1 + ((ea - P.c0) >> 2)];
    p2[j] = P.tab[1 + ((eb - P.c0) >> 2)];
    below0 |= (ea < P.e0 ? 1u : 0u) << j;
    below2 |= (eb < P.e0 ? 1u : 0u) << j;
    v[j].v = make_double2(el0 == P.s0 ? 1.0 : 0.0, 0.0);
    if (!P.init && (TB > 8 || el0 < size)) v[j].v = P.state[el0];
  }
  SmallStep now = P.step[P.k0];
  if (!P.meas_first) now.slot = -1;
  auto row_of = [&](int slot) { return P.partials + 3 * ((size_t)(slot - P.row0) * PL::kWarps + warp); };
  uint32_t el_last = 0u;
  int lo_last = 0;
  for (int k = P.k0;; k += 2) {
    {  // down: rounds 0, 1, 2
      if (now.slot >= 0) C::measure(v, b0, L0, below0, P.s0, row_of(now.slot));
      el_last = b0;
      lo_last = L0;
      if (k == P.k1) break;
      const R t = now.tan, sc = now.scale;
      now = P.step[k + 1];
#pragma unroll
      for (int j = 0; j < N; ++j) {
        const double2 x = v[j].v;
        v[j].v = make_double2(fma(x.x, p0[j].x, -x.y * p0[j].y), fma(x.x, p0[j].y, x.y * p0[j].x));
      }
      if (sc != (R)1) {
#pragma unroll
        for (int j = 0; j < N; ++j) El<R>::scale(v[j], sc);
      }
      C::template rotate<0>(v, t, P.np);
      alt_store<R, TB, KB, 0>(tile, v, b0);
      __syncthreads();
      alt_load<R, TB, KB, 1, true>(tile, v, b1);
      C::template rotate<1>(v, t, P.np);
      alt_store<R, TB, KB, 1>(tile, v, b1);
      __syncwarp();  // rounds 1 and 2 share their warp bits
      alt_load<R, TB, KB, 2, true>(tile, v, b2);
      C::template rotate<2>(v, t, P.np);
    }
    {  // up: rounds 2, 1, 0
      if (now.slot >= 0) C::measure(v, b2, 0, below2, P.s0, row_of(now.slot));
      el_last = b2;
      lo_last = 0;
      if (k + 1 == P.k1) break;
      const R t = now.tan, sc = now.scale;
      now = P.step[k + 2];
#pragma unroll
      for (int j = 0; j < N; ++j) {
        const double2 x = v[j].v;
        v[j].v = make_double2(fma(x.x, p2[j].x, -x.y * p2[j].y), fma(x.x, p2[j].y, x.y * p2[j].x));
      }
      if (sc != (R)1) {
#pragma unroll
        for (int j = 0; j < N; ++j) El<R>::scale(v[j], sc);
      }
      C::template rotate<2>(v, t, P.np);
      alt_store<R, TB, KB, 2>(tile, v, b2);
      __syncwarp();
      alt_load<R, TB, KB, 1, true>(tile, v, b1);
      C::template rotate<1>(v, t, P.np);
      alt_store<R, TB, KB, 1>(tile, v, b1);
      __syncthreads();
      alt_load<R, TB, KB, 0, true>(tile, v, b0);
      C::template rotate<0>(v, t, P.np);
    }
  }
#pragma unroll
  for (int j = 0; j < N; ++j) {
    const uint32_t el = el_last | ((uint32_t)j << lo_last);
    if (TB > 8 || el < size) P.state[el] = v[j].v;
  }
  __syncthreads();  // the partial rows of every warp
  for (int row = (int)threadIdx.x; row < P.rows; row += PL::kThreads) {
    double s[3] = {0, 0, 0};
    const double* p = P.partials + 3 * (size_t)row * PL::kWarps;
    for (int w = 0; w < PL::kWarps; ++w)
#pragma unroll
      for (int q = 0; q < 3; ++q) s[q] += p[3 * w + q];
    double* out = P.results + 4 * (size_t)(P.row0 + row);
    out[0] = s[1];
    out[1] = s[2];
    out[2] = s[0];
  }
}

}  // namespace bk
