// Auxiliary kernels: E table, p_blind count, state init, the plain per-qubit path,
// state export and projective sampling.
#pragma once
#include "bk_device.cuh"

namespace bk {

// E(s) for all s as uint16 (reference keeps doubles: src/sampling/sampler.cuh:54-70).
// Each thread writes 8 consecutive states (one 16-byte store).
__global__ void energy_table_kernel(uint16_t* __restrict__ out, int n, uint32_t count) {
  const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t s0 = g * 8u;
  if (s0 >= count) return;
  if (count - s0 >= 8u) {
    uint16_t e[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) e[k] = (uint16_t)labs_energy(s0 + k, n);
    uint4 q;
    q.x = e[0] | ((uint32_t)e[1] << 16);
    q.y = e[2] | ((uint32_t)e[3] << 16);
    q.z = e[4] | ((uint32_t)e[5] << 16);
    q.w = e[6] | ((uint32_t)e[7] << 16);
    *reinterpret_cast<uint4*>(out + s0) = q;
  } else {
    for (uint32_t s = s0; s < count; ++s) out[s] = (uint16_t)labs_energy(s, n);
  }
}

// #{s : E(s) < e0} (src/sampling/sampler.cuh:198-227); integer atomics are order-independent.
__global__ void count_below_kernel(const uint16_t* __restrict__ E, uint32_t count, int e0,
                                   unsigned long long* out) {
  unsigned long long c = 0;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x)
    c += ((int)E[i] < e0) ? 1ull : 0ull;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
  if ((threadIdx.x & 31) == 0 && c) atomicAdd(out, c);
}

template <class A>
__global__ void set_basis_kernel(A* psi, uint32_t idx) {
  A one;
  one.x = 1;
  one.y = 0;
  psi[idx] = one;
}

// complex64 pair-planar storage: float4 k = (re[2k], re[2k+1], im[2k], im[2k+1])
struct Planar64 {};
__global__ void set_basis_planar_kernel(float* psi, uint32_t idx) { psi[4u * (idx >> 1) + (idx & 1u)] = 1.0f; }
__device__ __forceinline__ double norm2_at(const float2* psi, uint32_t i) { return norm2d(psi[i]); }
__device__ __forceinline__ double norm2_at(const double2* psi, uint32_t i) { return norm2d(psi[i]); }
__device__ __forceinline__ double norm2_at(const Planar64* psi, uint32_t i) {
  const float* f = reinterpret_cast<const float*>(psi) + 4u * (i >> 1) + (i & 1u);
  return (double)fmaf(f[0], f[0], f[2] * f[2]);
}
__device__ __forceinline__ double2 amp_at(const float2* psi, uint32_t i) {
  return make_double2(psi[i].x, psi[i].y);
}
__device__ __forceinline__ double2 amp_at(const double2* psi, uint32_t i) { return psi[i]; }
__device__ __forceinline__ double2 amp_at(const Planar64* psi, uint32_t i) {
  const float* f = reinterpret_cast<const float*>(psi) + 4u * (i >> 1) + (i & 1u);
  return make_double2(f[0], f[2]);
}

// ---------------------------------------------------------------------------
// Plain path: the reference's launch structure (src/sampling/sampler.cuh:604-618)
// — one diagonal-phase kernel per step with FP64 sincos (:73-91), then one
// 2x2 kernel per qubit with the matrix [[c, i s], [i s, c]] (:451-457).
// ---------------------------------------------------------------------------
template <class A>
__global__ void plain_phase_kernel(A* __restrict__ psi, const uint16_t* __restrict__ E, uint32_t count,
                                   double dt_over_n) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  const double th = -dt_over_n * (double)E[i];
  double sn, cs;
  sincos(th, &sn, &cs);
  const A a = psi[i];
  A r;
  r.x = (double)a.x * cs - (double)a.y * sn;
  r.y = (double)a.x * sn + (double)a.y * cs;
  psi[i] = r;
}

template <class A>
__global__ void plain_rx_kernel(A* __restrict__ psi, uint32_t half, int q, double c, double s) {
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= half) return;
  const uint32_t lo = k & ((1u << q) - 1u);
  const uint32_t a = ((k >> q) << (q + 1)) | lo;
  const uint32_t b = a | (1u << q);
  const A x = psi[a], y = psi[b];
  A xa, yb;
  // [a'; b'] = [[c, i s], [i s, c]] [a; b]
  xa.x = c * (double)x.x - s * (double)y.y;
  xa.y = c * (double)x.y + s * (double)y.x;
  yb.x = c * (double)y.x - s * (double)x.y;
  yb.y = c * (double)y.y + s * (double)x.x;
  psi[a] = xa;
  psi[b] = yb;
}

// Measurement over the whole state (plain path and any state the tiled A1 pass
// does not cover): fixed grid, FP64 per-block partials, ordered finalize.
template <class A>
__global__ void measure_kernel(const A* __restrict__ psi, const uint16_t* __restrict__ E, uint32_t count,
                               int e0, uint32_t s0, double* partials, unsigned int* ticket, double* results,
                               int slot) {
  MeasureAcc acc;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x)
    acc.add(norm2d(psi[i]), (int)E[i] < e0, __popc(i ^ s0));
  block_reduce_and_finalize(acc, partials, ticket, results, slot, (int)gridDim.x);
}

// Export as interleaved (re, im) doubles, optionally multiplied by a diagonal
// phase exp(-i angle_unit * E(s)) (Strang convention) and a real scale.
template <class A>
__global__ void export_kernel(const A* __restrict__ psi, const uint16_t* __restrict__ E, uint32_t count,
                              double angle_unit, double scale, double2* __restrict__ out) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  const double2 a = amp_at(psi, i);
  double2 r = make_double2(a.x * scale, a.y * scale);
  if (angle_unit != 0.0) {
    double sn, cs;
    sincos(-angle_unit * (double)E[i], &sn, &cs);
    r = make_double2(r.x * cs - r.y * sn, r.x * sn + r.y * cs);
  }
  out[i] = r;
}

// ---------------------------------------------------------------------------
// Projective sampling by inverse CDF (the reference calls the closed
// custatevecSampler*, src/sampling/sampler.cuh:464-466, 564-573): chunk sums of
// |psi|^2 in FP64, an exclusive scan over chunks, then per shot a binary search
// over chunks and a warp scan inside the chunk. Shot k returns the smallest s
// with u_k * total < cdf(s).
// ---------------------------------------------------------------------------
constexpr int kSampleChunkBits = 12;

template <class A>
__global__ void chunk_sums_kernel(const A* __restrict__ psi, uint32_t count, double* __restrict__ sums) {
  const uint32_t chunk = blockIdx.x;
  const uint32_t base = chunk << kSampleChunkBits;
  const uint32_t len = min(1u << kSampleChunkBits, count - base);
  double acc = 0.0;
  for (uint32_t i = threadIdx.x; i < len; i += blockDim.x) acc += norm2_at(psi, base + i);
  __shared__ double red[kThreads / 32];
  acc = warp_sum(acc);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0;
    for (int w = 0; w < (int)(blockDim.x / 32); ++w) s += red[w];
    sums[chunk] = s;
  }
}

// In-place exclusive scan of `m` chunk sums by one block; total written to sums[m].
__global__ void scan_chunks_kernel(double* sums, uint32_t m) {
  __shared__ double carry;
  __shared__ double wsum[32];
  if (threadIdx.x == 0) carry = 0.0;
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (uint32_t base = 0; base < m; base += blockDim.x) {
    const uint32_t i = base + threadIdx.x;
    const double x = (i < m) ? sums[i] : 0.0;
    double inc = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double y = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += y;
    }
    if (lane == 31) wsum[warp] = inc;
    __syncthreads();
    if (warp == 0) {
      double w = (lane < (int)(blockDim.x / 32)) ? wsum[lane] : 0.0;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const double y = __shfl_up_sync(0xffffffffu, w, o);
        if (lane >= o) w += y;
      }
      wsum[lane] = w;  // inclusive over warps
    }
    __syncthreads();
    const double before = carry + (warp > 0 ? wsum[warp - 1] : 0.0);
    if (i < m) sums[i] = before + inc - x;
    __syncthreads();
    if (threadIdx.x == blockDim.x - 1) carry = before + inc;
    __syncthreads();
  }
  if (threadIdx.x == 0) sums[m] = carry;
}

// One warp per shot.
template <class A>
__global__ void sample_kernel(const A* __restrict__ psi, uint32_t count, const double* __restrict__ prefix,
                              uint32_t m, const double* __restrict__ randnums, int64_t shots,
                              unsigned long long* __restrict__ out) {
  const int64_t shot = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (shot >= shots) return;
  const double total = prefix[m];
  const double target = randnums[shot] * total;
  // last chunk whose exclusive prefix is <= target
  uint32_t lo = 0, hi = m;  // answer in [lo, hi)
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (prefix[mid] <= target) lo = mid; else hi = mid;
  }
  const uint32_t base = lo << kSampleChunkBits;
  const uint32_t len = min(1u << kSampleChunkBits, count - base);
  // the chunk's 32 blocks of 128 states: coalesced sums, lane b keeps block b's (a lane
  // walking its own 128 states made a sampling point at n = 16 85 us instead of 70)
  double part = 0.0;
  for (uint32_t b = 0; b < 32u; ++b) {
    if (b * 128u >= len) break;
    double w = 0.0;
#pragma unroll
    for (uint32_t q = 0; q < 4u; ++q) {
      const uint32_t i = b * 128u + q * 32u + (uint32_t)lane;
      if (i < len) w += norm2_at(psi, base + i);
    }
    w = warp_sum(w);
    if ((uint32_t)lane == b) part = w;
  }
  double inc = part;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const double y = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += y;
  }
  // first block whose inclusive cumulative exceeds the target
  const unsigned blocks = __ballot_sync(0xffffffffu, target < prefix[lo] + inc && (uint32_t)lane * 128u < len);
  if (!blocks) {
    if (lane == 0) out[shot] = base + len - 1;  // rounding guard: clamp to the chunk's last state
    return;
  }
  const int blk = __ffs(blocks) - 1;
  const double start = prefix[lo] + __shfl_sync(0xffffffffu, inc - part, blk);
  // inside it: four consecutive states a lane
  const uint32_t b0 = (uint32_t)blk * 128u, b1 = min(len, b0 + 128u), mine0 = min(b1, b0 + 4u * (uint32_t)lane),
                 mine1 = min(b1, mine0 + 4u);
  double p[4], sum = 0.0;
#pragma unroll
  for (uint32_t q = 0; q < 4u; ++q) {
    p[q] = mine0 + q < mine1 ? norm2_at(psi, base + mine0 + q) : 0.0;
    sum += p[q];
  }
  inc = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const double y = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += y;
  }
  const unsigned lanes = __ballot_sync(0xffffffffu, target < start + inc && mine1 > mine0);
  if (!lanes) {
    if (lane == 0) out[shot] = base + b1 - 1;
    return;
  }
  if (lane == __ffs(lanes) - 1) {
    double c = start + inc - sum;
    uint32_t r = mine1 - 1;
#pragma unroll
    for (uint32_t q = 0; q < 4u; ++q) {
      c += p[q];
      if (target < c) {
        r = min(r, mine0 + q);
      }
    }
    out[shot] = base + r;
  }
}

}  // namespace bk

namespace bk {

// ---------------------------------------------------------------------------
// d_min (reference: src/labs_energy/labs_energy.hpp:175-207): is there a state
// with E < target on the Hamming sphere of radius d around s? Each thread
// unranks masks of weight d (combinatorial number system, colex order) in a
// grid-stride loop; the first hit raises *found and the others stop early.
// binom[c * 32 + k] = C(c, k) for c, k < 32.
// ---------------------------------------------------------------------------
__global__ void dmin_sphere_kernel(int n, uint32_t s, int target, int d, unsigned long long count,
                                   const unsigned long long* __restrict__ binom, int* found) {
  const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
  for (unsigned long long r = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; r < count; r += stride) {
    if (*reinterpret_cast<volatile int*>(found)) return;
    uint32_t mask = 0;
    unsigned long long rem = r;
    int c = n - 1;
    for (int k = d; k >= 1; --k) {
      while (binom[c * 32 + k] > rem) --c;
      mask |= 1u << c;
      rem -= binom[c * 32 + k];
      --c;
    }
    if (labs_energy(s ^ mask, n) < target) atomicExch(found, 1);
  }
}

// ---------------------------------------------------------------------------
// Batched single-flip steepest descent (reference: batch_steepest_descent_kernel,
// src/classical/classical.cuh:459-540; CPU form :625-712). One warp per start: lane l
// scores the flips p = l (and l + 32 from 33 spins on), the warp keeps the lowest
// energy and, among equal energies, the lowest p — the flip the sequential scan (first
// strictly better) takes. An iteration costs n evaluations and runs only while evals +
// n <= budget, as in the reference.
//
// A flip of spin p changes every C_k by d_k = -2 s_p t_k, t_k = s_{p+k} + s_{p-k} (a
// spin outside the chain counts 0), so the energy by
//   sum_k d_k (2 C_k + d_k) = -4 s_p V + 4 Q,  V = sum_k C_k t_k,  Q = sum_k t_k^2.
// V: with u_k, w_k the bits of the spins at p + k and p - k, t_k = (valid) - 2 (u_k +
// w_k), so V = prefix sums of C - 2 sum_k C_k (u_k + w_k), and C_k (|C_k| < n, a byte)
// against u_k + w_k (bytes) is four products an instruction (dp4a); the bytes stay in
// registers and a flip of spin q changes one of them per lane, the one at |p - q|.
// Q = n - 1 + 2 sum over the pairs inside the chain of s_{p+k} s_{p-k}: a popcount of
// the chain against its mirror image. About 90 instructions an iteration up to 32
// spins, where trying every flip with its n - 1 correlations took about 700
// (B200, 65536 starts: n = 28 58 us against 268, n = 63 256 us against 1869).
// ---------------------------------------------------------------------------
constexpr int kDescentWarps = 8;

__device__ __forceinline__ uint32_t bits_to_bytes(uint32_t b) { return (b * 0x00204081u) & 0x01010101u; }

// HALVES = 1: up to 32 spins, 2: up to 63
template <int HALVES>
struct DescentWord;
template <>
struct DescentWord<1> {
  using T = uint32_t;
  __device__ static T rev(T x) { return __brev(x); }
  __device__ static int popc(T x) { return __popc(x); }
};
template <>
struct DescentWord<2> {
  using T = unsigned long long;
  __device__ static T rev(T x) { return __brevll(x); }
  __device__ static int popc(T x) { return __popcll(x); }
};

template <int HALVES>
__global__ void __launch_bounds__(32 * kDescentWarps)
    descent_kernel(int n, const typename DescentWord<HALVES>::T* __restrict__ starts, long long count,
                   unsigned long long budget, typename DescentWord<HALVES>::T* __restrict__ final_states,
                   int* __restrict__ final_energies, uint32_t* __restrict__ evals_out) {
  using W = DescentWord<HALVES>;
  using T = typename W::T;
  constexpr int kBits = 32 * HALVES, kWords = 8 * HALVES;  // chain bits, words of four C bytes
  __shared__ __align__(16) signed char Cs[kDescentWarps][kBits];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const long long i = (long long)blockIdx.x * kDescentWarps + wib;
  if (i >= count) return;  // the whole warp leaves together
  signed char* C = Cs[wib];
  const T mask = (T)~(T)0 >> (kBits - n);
  T x = starts[i] & mask;
  int c[HALVES], e = 0;
#pragma unroll
  for (int h = 0; h < HALVES; ++h) {
    const int k = lane + 32 * h;
    c[h] = 0;
    if (k >= 1 && k < n) c[h] = (n - k) - 2 * W::popc((x ^ (x >> k)) & (mask >> k));
    C[k] = (signed char)c[h];
    e += c[h] * c[h];
  }
  e = __reduce_add_sync(0xffffffffu, e);
  // bytes u_k + w_k of each of the lane's spins
  uint32_t t[HALVES][kWords];
#pragma unroll
  for (int h = 0; h < HALVES; ++h) {
    const int p = lane + 32 * h;
    const T u = x >> p, w = W::rev(x) >> (kBits - 1 - p);
#pragma unroll
    for (int g = 0; g < kWords; ++g)
      t[h][g] = bits_to_bytes((uint32_t)(u >> (4 * g)) & 15u) + bits_to_bytes((uint32_t)(w >> (4 * g)) & 15u);
  }
  __syncwarp();
  unsigned long long evals = 1;
  while (evals + (unsigned long long)n <= budget) {
    // prefix sums of C: lane l holds sum_{k <= l} C_k (second half: k <= l + 32)
    int pre[HALVES];
#pragma unroll
    for (int h = 0; h < HALVES; ++h) {
      pre[h] = c[h];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, pre[h], o);
        if (lane >= o) pre[h] += y;
      }
      if (h == 1) pre[1] += __shfl_sync(0xffffffffu, pre[0], 31);
    }
    int dot[HALVES];
#pragma unroll
    for (int h = 0; h < HALVES; ++h) dot[h] = 0;
#pragma unroll
    for (int g = 0; g < kWords; g += 4) {
      const int4 q = *reinterpret_cast<const int4*>(C + 4 * g);  // the same address in every lane
#pragma unroll
      for (int h = 0; h < HALVES; ++h) {
        dot[h] = __dp4a(q.x, (int)t[h][g], dot[h]);
        dot[h] = __dp4a(q.y, (int)t[h][g + 1], dot[h]);
        dot[h] = __dp4a(q.z, (int)t[h][g + 2], dot[h]);
        dot[h] = __dp4a(q.w, (int)t[h][g + 3], dot[h]);
      }
    }
    int key = 0x7fffffff;  // energy change * 64 + p
    const T r = W::rev(x);
#pragma unroll
    for (int h = 0; h < HALVES; ++h) {
      const int p = lane + 32 * h;
      const int far = n - 1 - p;  // spins above p
      int up = __shfl_sync(0xffffffffu, pre[0], far & 31);
      if (HALVES == 2) {
        const int hi = __shfl_sync(0xffffffffu, pre[HALVES - 1], far & 31);
        if (far >= 32) up = hi;
      }
      if (p < n) {
        const int m = min(p, far);
        const T u = x >> p, w = r >> (kBits - 1 - p);
        const int unlike = W::popc((u ^ w) & (T)((((T)1 << m) - 1) << 1));
        const int V = up + pre[h] - 2 * dot[h];
        const int Q = n - 1 + 2 * (m - 2 * unlike);
        const int s = (u & 1) ? -1 : 1;
        key = min(key, 4 * (Q - s * V) * 64 + p);
      }
    }
    key = __reduce_min_sync(0xffffffffu, key);
    evals += (unsigned long long)n;
    if (key >= 0) break;  // no strictly better neighbour: a local minimum
    const int q = key & 63;
    e += key >> 6;
    const int sq = (int)((x >> q) & 1) ? -1 : 1;
    __syncwarp();
#pragma unroll
    for (int h = 0; h < HALVES; ++h) {
      const int k = lane + 32 * h;
      // the lane as the correlation C_k
      if (k >= 1 && k < n) {
        int d = 0;
        if (q + k < n) d += (int)((x >> (q + k)) & 1) ? -1 : 1;
        if (q - k >= 0) d += (int)((x >> (q - k)) & 1) ? -1 : 1;
        c[h] -= 2 * sq * d;
        C[k] = (signed char)c[h];
      }
      // the lane as spin p = k: the byte at |p - q| moves with spin q's new bit
      const int dist = k > q ? k - q : q - k;
      const uint32_t step = dist == 0 ? 0u : (sq > 0 ? 1u : 0xFFFFFFFFu) << (8 * (dist & 3));
#pragma unroll
      for (int g = 0; g < kWords; ++g) t[h][g] += (dist >> 2) == g ? step : 0u;
    }
    x ^= (T)1 << q;
    __syncwarp();
  }
  if (lane == 0) {
    final_states[i] = x;
    final_energies[i] = e;
    evals_out[i] = (uint32_t)evals;  // at most n flips' worth per energy level: far below 2^32
  }
}

// Per-shot energy and Hamming distance to the start state for drawn basis
// states (the reference evaluates both on the host for every shot,
// src/sampling/sampler.cuh:575-596): one thread per shot, exact integers.
__global__ void shot_stats_kernel(const unsigned long long* __restrict__ states, long long count, int n,
                                  unsigned long long s0, int* __restrict__ energies, int* __restrict__ flips) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  const unsigned long long b = states[i];
  energies[i] = labs_energy((uint32_t)b, n);
  flips[i] = __popcll(b ^ s0);
}

}  // namespace bk
