// Turning-pass engine (sm_100a): one pass over the statevector per Trotter step.
//
// A step is psi <- M D psi with M a product of commuting single-qubit rotations,
// so the qubits of a step may be rotated in any order. With the element bits
// split into two sets X and Y (each a tile of the statevector can hold), the
// steps run as
//   [D_0 X][Y D_1 Y][X D_2 X] ... [. finish]
// where a bracket is ONE pass over the state: the pass finishes step k - 1 on its
// set, measures psi_k, applies D_k and starts step k on the same set. Every step
// costs one pass, where a pass per set costs two. With three sets (large states)
// a plain pass over the third set A sits between two turning passes:
//   [D_0 S][A][T D_1 T][A][S D_2 S][A] ...
// two passes a step instead of three.
//
// Tiles. 2^TB 16-byte elements (bk_persist.cuh): the A set is element bits
// [0, TB), an S set [h0, h0 + w) with the tile's other cp = TB - w bits contiguous
// low ones. A thread keeps 2^KB elements in registers; round 0 holds the top KB
// tile bits in registers, round 1 the next KB, round 2 the lowest (those left).
// A turning pass climbs down the rounds that its set needs, turns (measurement,
// D, amplitude bit 0 of complex64) in the last of them and climbs back up, so
// w <= KB needs no shared-memory round trip, w <= 2 KB two, more four. The last
// round is round 0 again: lanes run over the low tile bits and every global
// store is a run of min(512, 16 * 2^cp) bytes.
//
// What bounds it (B200): up to 2^23 elements shared memory and its latency (N = 23
// complex64: shared-memory pipe 52%, issue 26% of peak at 16 warps an SM; a step of
// N = 19 is 5.4 us against 27 us for the persistent task engine, N = 22 23 against
// 37); beyond, DRAM: N = 28 complex64 1.54 ms a step = 5.6 TB/s over its two passes
// (2.09 ms with a pass per set and the strided passes fused through L2).
//
// All passes of a run are one cooperative launch: a CTA takes tiles
// rank, rank + G, ... of each pass and a counter barrier over the G CTAs
// separates the passes (bounded polls, a common abort word). The next tile's TMA
// load is issued as soon as the current tile's last shared-memory read is done.
#pragma once
#include "bk_s23.cuh"

namespace bk {

// Full per-energy phase table: every LABS energy is c0 + 4 j. Entry 0 rotates by
// nothing, entry 1 + j by level j; a pass without D reads entry 0 through a stride
// of 0 (a branch around the unrolled phase costs the register allocation more).
template <class R>
struct AltPhase;
struct AltTab {
  const unsigned char* base;  // where E = 0 would be
  uint32_t per_e;             // bytes per unit of E (an entry per 4 units), or 0
};
template <>
struct AltPhase<float> {
  using entry = float2;  // {-tan(r/4), sin(r/2)}: two half-angle shear rotations
  __device__ static void apply(El<float>::T& v, uint32_t e2, const AltTab& t) {
    const float2 H0 = *reinterpret_cast<const float2*>(t.base + (e2 & 0xFFFFu) * t.per_e);
    const float2 H1 = *reinterpret_cast<const float2*>(t.base + (e2 >> 16) * t.per_e);
    const float2 A = make_float2(H0.x, H1.x), B = make_float2(H0.y, H1.y);
    PhaseV<float>::shear2(v.re, v.im, A, B);
    PhaseV<float>::shear2(v.re, v.im, A, B);
  }
};
template <>
struct AltPhase<double> {
  using entry = double2;  // {cos r, sin r}
  __device__ static void apply(El<double>::T& v, uint32_t e, const AltTab& t) {
    const double2 cs = *reinterpret_cast<const double2*>(t.base + e * t.per_e);
    v.v = make_double2(fma(v.v.x, cs.x, -v.v.y * cs.y), fma(v.v.x, cs.y, v.v.y * cs.x));
  }
};

// the table at `tab` (shared memory), or its entry 0 for every E
template <class R>
__device__ __forceinline__ AltTab alt_tab(const unsigned char* tab, bool on, uint32_t c0) {
  constexpr uint32_t kEntry = sizeof(typename AltPhase<R>::entry), kPerE = kEntry / 4u;
  return on ? AltTab{tab + kEntry - c0 * kPerE, kPerE} : AltTab{tab, 0u};
}

// TMA coordinates of a set's tiles: the dimensions of the tile id's two parts.
struct AltSet {
  int mid_dim, hi_dim, mid_bits, pad;
};

// A run's geometry and tables (kernel parameter), the same for every statevector of a batch launch.
template <class R>
struct AltRunDesc {
  const uint16_t* E;
  const typename AltPhase<R>::entry* tab;
  const int* slot;     // [steps + 1] measurement row, or -1
  double* partials;    // [rows][units][3]: norm, P_<, <d_H> of a unit's elements
  AltSet set[3];       // the A set, the S sets
  uint32_t n_tiles;
  uint32_t units;      // units of a measured row: a warp's share of a tile, with three sets a CTA's tiles
  int n_j, c0;         // levels of the phase table (after its entry 0), lowest level
  int k0, k1;          // steps [k0, k1)
  int row0;            // first measurement row of `partials`
  int meas_first;      // measure psi_k0 (else an earlier segment has)
};
// One statevector (kernel parameter; device memory for a batch).
template <class R>
struct alignas(64) AltInst {
  CUtensorMap map[3];  // tiles of the A set and of the S sets
  unsigned char* state;
  const R* tan;        // [steps]
  const R* scale;      // [steps]
  double* results;     // batch: [rows][4]
  int e0;
  uint32_t s0;
};
// The statevectors of a batch launch: group g of G CTAs takes instances g, g + n_groups, ...
template <class R>
struct AltBatch {
  const AltInst<R>* inst;
  int n_inst, n_rows;  // n_rows: of this launch, from row D.row0 on
  uint32_t G;
  size_t part_stride;  // doubles of one partial-sum buffer ([n_rows][units][3]); every group has two
};

// Barrier over the G CTAs of a run; `ctr` counts arrivals over all passes.
struct AltBarrier {
  unsigned int* ctr;   // batch: one per group, 32 words apart
  int* err;
  int* abort;
  uint32_t poll_limit;
};

template <int TB, int KB>
struct AltPlan {
  static constexpr int kThreads = 1 << (TB - KB);
  static constexpr int kWarps = kThreads / 32;
  static constexpr int kPer = 1 << KB;
  static_assert(TB - KB >= 5 && 3 * KB >= TB && TB - KB <= 9, "three rounds cover the tile");
  // lowest register bit and number of new tile bits of each round
  static constexpr int reg_lo(int r) { return r == 0 ? TB - KB : r == 1 ? TB - 2 * KB : 0; }
  static constexpr int act_hi(int r) { return r < 2 ? KB : TB - 2 * KB; }
  // tile position of a thread's register element 0. Round 0: lanes over tile bits
  // 0-4. Round 1: the bits below its registers first, then those from TB - KB up
  // (with two low bits the third lane takes bit 8, so that the three lowest lanes
  // fold onto different residues of the swizzle); rounds 1 and 2 share their warp
  // bits (the top ones), so data moves inside a warp between them.
  template <int r>
  __device__ static uint32_t base(uint32_t lane, uint32_t warp) {
    if constexpr (r == 0) return lane | (warp << 5);
    constexpr int top = TB - (TB - KB - 5);  // warp bits [top, TB) of rounds 1 and 2
    if constexpr (r == 2) return (lane << KB) | (warp << top);
    constexpr int lo = TB - 2 * KB;          // tile bits below round 1's registers
    if constexpr (lo == 2 && TB == 10) {
      return (lane & 3u) | ((lane & 4u) << 6) | ((lane & 24u) << 3) | (warp << top);
    }
    return (lane & ((1u << lo) - 1u)) | ((lane >> lo) << (TB - KB)) | (warp << top);
  }
};

// element index of tile position p relative to the tile's base: bits at or above CP move to H0
template <int CP, int H0>
__device__ __forceinline__ constexpr uint32_t alt_index(uint32_t p) {
  return (p & ((1u << CP) - 1u)) | ((p >> CP) << H0);
}

// A value the compiler may not relate to earlier uses: the swizzled addresses of
// a round are cheap to form again and too many to keep between the rounds.
__device__ __forceinline__ uint32_t alt_fresh(uint32_t x) {
  asm volatile("" : "+r"(x));
  return x;
}

template <class R, int TB, int KB, int r, bool SWZ>
__device__ __forceinline__ void alt_load(const unsigned char* s, typename El<R>::T (&v)[1 << KB], uint32_t base) {
  constexpr int lo = AltPlan<TB, KB>::reg_lo(r);
  const uint32_t sb = alt_fresh(SWZ ? swz<double>(base) : base);
#pragma unroll
  for (int j = 0; j < (1 << KB); ++j)
    v[j] = El<R>::ld(s + 16u * (sb ^ (SWZ ? swz<double>((uint32_t)j << lo) : (uint32_t)j << lo)));
}
template <class R, int TB, int KB, int r>
__device__ __forceinline__ void alt_store(unsigned char* s, const typename El<R>::T (&v)[1 << KB], uint32_t base) {
  constexpr int lo = AltPlan<TB, KB>::reg_lo(r);
  const uint32_t sb = alt_fresh(swz<double>(base));
#pragma unroll
  for (int j = 0; j < (1 << KB); ++j) El<R>::st(s + 16u * (sb ^ swz<double>((uint32_t)j << lo)), v[j]);
}
// A set one bit wider than two rounds hold: its lowest bit, tile bit CP, is lane bit CP in
// round 1 (whose lanes run over the bits below its registers), so it is rotated across
// lanes instead of in a round of its own (two more trips through shared memory).
__host__ __device__ constexpr bool alt_lane_bit(int TB, int KB, int CP) { return TB - CP == 2 * KB + 1 && CP > 0; }

// the rotations of round r's new bits that belong to the set (tile bits >= cp)
template <class R, int TB, int KB, int CP, int r>
__device__ __forceinline__ void alt_rotate(typename El<R>::T (&v)[1 << KB], R t) {
  constexpr int lo = AltPlan<TB, KB>::reg_lo(r);
#pragma unroll
  for (int k = 0; k < AltPlan<TB, KB>::act_hi(r); ++k) {
    if (lo + k >= CP) {
#pragma unroll
      for (int j = 0; j < (1 << KB); ++j)
        if (!(j & (1 << k))) El<R>::bfly(v[j], v[j | (1 << k)], t);
    }
  }
  if constexpr (r == 1 && alt_lane_bit(TB, KB, CP)) {
#pragma unroll
    for (int j = 0; j < (1 << KB); ++j) {
      const typename El<R>::T q = El<R>::shfl_xor(v[j], 1 << CP);
      El<R>::bfly_partner(v[j], q, t);
    }
  }
}
// E of the thread's elements in round r's layout, brought into shared memory by
// asynchronous copies while the tile is on its way (every thread reads back only
// what it copied: no barrier). Round 2 holds consecutive elements (16-byte copies);
// the others one 4-byte word per element (complex128: the word around its uint16).
__device__ __forceinline__ void cp_async4(uint32_t dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

template <class R, int TB, int KB, int CP, int H0, int r>
struct AltE {
  static constexpr int kThreads = AltPlan<TB, KB>::kThreads;
  static constexpr int lo = AltPlan<TB, KB>::reg_lo(r);
  static constexpr bool kRun = r == 2 && CP >= KB;             // 2^KB consecutive elements
  static constexpr int kPieces = (1 << KB) * (int)sizeof(uint16_t) * El<R>::kAmps / 16;  // 16-byte pieces of a run
  __device__ static void fetch(const uint16_t* __restrict__ E, uint32_t tile_base, uint32_t base, uint32_t es) {
    const uint32_t g0 = tile_base | alt_index<CP, H0>(base);
    const uint32_t tid = threadIdx.x;
    if constexpr (kRun) {
      const unsigned char* p = reinterpret_cast<const unsigned char*>(E + (size_t)g0 * El<R>::kAmps);
#pragma unroll
      for (int q = 0; q < kPieces; ++q) cp_async16(es + 16u * (uint32_t)(q * kThreads + tid), p + 16 * q);
    } else {
      const uint32_t* p = reinterpret_cast<const uint32_t*>(E) + (sizeof(R) == 4 ? g0 : g0 >> 1);
#pragma unroll
      for (int j = 0; j < (1 << KB); ++j)
        cp_async4(es + 4u * (uint32_t)(j * kThreads + tid), p + (alt_index<CP, H0>((uint32_t)j << lo) >> (sizeof(R) == 4 ? 0 : 1)));
    }
  }
  // E of element j of the thread
  __device__ static uint32_t get1(const unsigned char* es, uint32_t base, uint32_t j) {
    const uint32_t tid = threadIdx.x;
    if constexpr (kRun) {
      constexpr uint32_t per = 16 / (sizeof(uint16_t) * El<R>::kAmps);  // elements of a piece
      const unsigned char* p = es + 16u * ((j / per) * kThreads + tid);
      if constexpr (sizeof(R) == 4)
        return reinterpret_cast<const uint32_t*>(p)[j % per];
      else
        return reinterpret_cast<const uint16_t*>(p)[j % per];
    } else {
      const uint32_t w = *reinterpret_cast<const uint32_t*>(es + 4u * (j * kThreads + tid));
      return sizeof(R) == 4 ? w : (((base + (j << lo)) & 1u) ? w >> 16 : w & 0xFFFFu);
    }
  }
  // E of elements j0 .. j0 + 7 of the thread (base: tile position of its element 0)
  __device__ static void get8(const unsigned char* es, uint32_t base, int j0, uint32_t (&ev)[8]) {
    const uint32_t tid = threadIdx.x;
    if constexpr (kRun) {
#pragma unroll
      for (int q = 0; q < (sizeof(R) == 4 ? 2 : 1); ++q) {
        const uint4 a = *reinterpret_cast<const uint4*>(es + 16u * (uint32_t)((j0 / (sizeof(R) == 4 ? 4 : 8) + q) * kThreads + tid));
        const uint32_t w[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          if constexpr (sizeof(R) == 4) {
            ev[4 * q + i] = w[i];
          } else {
            ev[2 * i] = w[i] & 0xFFFFu;
            ev[2 * i + 1] = w[i] >> 16;
          }
        }
      }
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const uint32_t w = *reinterpret_cast<const uint32_t*>(es + 4u * (uint32_t)((j0 + i) * kThreads + tid));
        if constexpr (sizeof(R) == 4) {
          ev[i] = w;
        } else {
          const uint32_t odd = (base + (((uint32_t)(j0 + i) << lo))) & 1u;  // which uint16 of the word
          ev[i] = odd ? w >> 16 : w & 0xFFFFu;
        }
      }
    }
  }
};

// what a turning pass does at its turn
template <class R>
struct AltTurn {
  R t_pre, t_post, scale;
  uint32_t c0;
  bool post, meas;
};

// |psi|^2 of an element's amplitudes: their sum, the share with E < e0 and the sum
// weighted by the Hamming distance to s0 (a small integer becomes a double by an
// exponent and one subtraction: the conversion unit is a quarter of the FP64 rate)
__device__ __forceinline__ double alt_small(uint32_t k) { return __hiloint2double(0x43300000, (int)k) - 4503599627370496.0; }
__device__ __forceinline__ void alt_weights(const El<float>::T& v, uint32_t e2, uint32_t el, int e0, uint32_t s0,
                                            double& n, double& b, double& f) {
  const double w0 = (double)fmaf(v.re.x, v.re.x, v.im.x * v.im.x), w1 = (double)fmaf(v.re.y, v.re.y, v.im.y * v.im.y);
  const uint32_t d = (el << 1) ^ s0;
  n = w0 + w1;
  b = ((int)(e2 & 0xFFFFu) < e0 ? w0 : 0.0) + ((int)(e2 >> 16) < e0 ? w1 : 0.0);
  f = fma(w0, alt_small(__popc(d)), w1 * alt_small(__popc(d ^ 1u)));
}
__device__ __forceinline__ void alt_weights(const El<double>::T& v, uint32_t e, uint32_t el, int e0, uint32_t s0,
                                            double& n, double& b, double& f) {
  n = fma(v.v.x, v.v.x, v.v.y * v.v.y);
  b = (int)e < e0 ? n : 0.0;
  f = n * alt_small(__popc(el ^ s0));
}

// where the threshold and the trap are (read by the passes that measure), and where a
// warp's sums go: put(norm, P_<, <d_H>) by its lane 0
template <class Put>
struct AltMeas {
  const int* e0;
  const uint32_t* s0;
  Put put;
};

// Measurement of the thread's elements at the turn: rolled, from the thread's own
// slots of the tile and of the staged E (no barrier), so that it costs the passes
// that measure nothing neither registers nor instruction cache. Unrolled on the
// register copies it pushed the 2^12-element kernels into spills, which go to L2:
// next to the tile the L1 has little room.
template <class R, int TB, int KB, int CP, int H0, int r, class Put>
__device__ __forceinline__ void alt_measure(const typename El<R>::T (&v)[1 << KB], unsigned char* tile,
                                            const unsigned char* es, int e0, uint32_t s0, uint32_t tile_base,
                                            uint32_t base, const Put& put) {
  constexpr int lo = AltPlan<TB, KB>::reg_lo(r);
  alt_store<R, TB, KB, r>(tile, v, base);
  const uint32_t sb = swz<double>(base), g0 = tile_base | alt_index<CP, H0>(base);
  double norm = 0.0, below = 0.0, flips = 0.0;
#pragma unroll 1
  for (uint32_t j0 = 0; j0 < (1u << KB); j0 += 4u) {
    // four elements at once: short sums over independent terms instead of one chain
    double n4[4], b4[4], f4[4];
#pragma unroll
    for (uint32_t i = 0; i < 4u; ++i) {
      const uint32_t j = j0 + i;
      const typename El<R>::T x = El<R>::ld(tile + 16u * (sb ^ swz<double>(j << lo)));
      const uint32_t e = AltE<R, TB, KB, CP, H0, r>::get1(es, base, j);
      alt_weights(x, e, g0 + alt_index<CP, H0>(j << lo), e0, s0, n4[i], b4[i], f4[i]);
    }
    norm += (n4[0] + n4[1]) + (n4[2] + n4[3]);
    below += (b4[0] + b4[1]) + (b4[2] + b4[3]);
    flips += (f4[0] + f4[1]) + (f4[2] + f4[3]);
  }
  const double a = warp_sum(norm), b = warp_sum(below), c = warp_sum(flips);
  if ((threadIdx.x & 31u) == 0) put(a, b, c);
}

template <class R, int TB, int KB, int CP, int H0, int r, class Put>
__device__ __forceinline__ void alt_turn(typename El<R>::T (&v)[1 << KB], unsigned char* tile, const unsigned char* es,
                                         const AltTurn<R>& T, uint32_t tile_base, uint32_t base,
                                         const unsigned char* tab, const AltMeas<Put>& M) {
  cp_async_wait();
  if (T.meas) {
    alt_measure<R, TB, KB, CP, H0, r>(v, tile, es, *M.e0, *M.s0, tile_base, base, M.put);
    alt_load<R, TB, KB, r, true>(tile, v, base);  // the measurement needs the registers
  }
  const AltTab P = alt_tab<R>(tab, T.post, T.c0);
#pragma unroll
  for (int j0 = 0; j0 < (1 << KB); j0 += 8) {
    uint32_t ev[8];
    AltE<R, TB, KB, CP, H0, r>::get8(es, base, j0, ev);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      AltPhase<R>::apply(v[j0 + i], ev[i], P);
      El<R>::bfly_inner(v[j0 + i], T.t_post);
    }
  }
  if (T.scale != (R)1) {
#pragma unroll
    for (int j = 0; j < (1 << KB); ++j) El<R>::scale(v[j], T.scale);
  }
  alt_rotate<R, TB, KB, CP == TB ? 0 : CP, r>(v, T.t_post);
}

// the round a pass turns in (CP = TB: the A set)
__host__ __device__ constexpr int alt_turn_round(int TB, int KB, int CP) {
  return CP == TB ? 2 : alt_lane_bit(TB, KB, CP) ? 1 : (TB - CP + KB - 1) / KB - 1;
}

// A turning pass on one staged tile (CP = TB: a tile of the A set). `wait()` returns
// when the tile has landed, `stage_free()` runs in every thread after a barrier
// behind the last shared-memory read.
// 2^10-element tiles are read straight into round 0's registers: a CTA has one of them a
// pass (or little more), so there is nothing to load ahead, and the copy through shared
// memory with its barrier is latency on top of the exchange's.
constexpr bool alt_direct(int TB) { return TB == 10; }
template <class R>
__device__ __forceinline__ typename El<R>::T alt_ldcg(const unsigned char* p) {
  const float4 q = __ldcg(reinterpret_cast<const float4*>(p));  // other SMs write it: never from L1
  return El<R>::ld(&q);
}

template <class R, int TB, int KB, int CP, int H0, class Put, class W, class F>
__device__ __forceinline__ void alt_tile_turn(unsigned char* tile, unsigned char* state, const AltTurn<R>& T,
                                              uint32_t tile_base, const unsigned char* tab, unsigned char* es,
                                              const AltMeas<Put>& M, W&& wait, F&& stage_free) {
  using PL = AltPlan<TB, KB>;
  constexpr int RT = alt_turn_round(TB, KB, CP);
  constexpr int LO = CP == TB ? 0 : CP;  // lowest tile bit of the set
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint32_t b0 = PL::template base<0>(lane, warp);
  typename El<R>::T v[1 << KB];
  if constexpr (alt_direct(TB)) {
    const unsigned char* g = state + 16ull * (tile_base | alt_index<CP, H0>(b0));
#pragma unroll
    for (int j = 0; j < (1 << KB); ++j)
      v[j] = alt_ldcg<R>(g + 16ull * alt_index<CP, H0>((uint32_t)j << PL::reg_lo(0)));
  } else {
    wait();
    alt_load<R, TB, KB, 0, false>(tile, v, b0);
  }
  if constexpr (RT == 0) {
    alt_rotate<R, TB, KB, LO, 0>(v, T.t_pre);
    if (T.meas) __syncwarp();  // the measurement's swizzled slots were other lanes' linear ones
    alt_turn<R, TB, KB, CP, H0, 0>(v, tile, es, T, tile_base, b0, tab, M);
    __syncthreads();
    stage_free();
  } else {
    alt_rotate<R, TB, KB, LO, 0>(v, T.t_pre);
    __syncwarp();  // the linear tile's reads against swizzled stores: same warp
    alt_store<R, TB, KB, 0>(tile, v, b0);
    __syncthreads();
    const uint32_t b1 = PL::template base<1>(lane, warp);
    alt_load<R, TB, KB, 1, true>(tile, v, b1);
    alt_rotate<R, TB, KB, LO, 1>(v, T.t_pre);
    if constexpr (RT == 1) {
      alt_turn<R, TB, KB, CP, H0, 1>(v, tile, es, T, tile_base, b1, tab, M);
    } else {
      alt_store<R, TB, KB, 1>(tile, v, b1);
      __syncwarp();  // rounds 1 and 2 share their warp bits
      const uint32_t b2 = PL::template base<2>(lane, warp);
      alt_load<R, TB, KB, 2, true>(tile, v, b2);
      alt_rotate<R, TB, KB, LO, 2>(v, T.t_pre);
      alt_turn<R, TB, KB, CP, H0, 2>(v, tile, es, T, tile_base, b2, tab, M);
      alt_store<R, TB, KB, 2>(tile, v, b2);
      __syncwarp();
      alt_load<R, TB, KB, 1, true>(tile, v, b1);
      alt_rotate<R, TB, KB, LO, 1>(v, T.t_post);
    }
    alt_store<R, TB, KB, 1>(tile, v, b1);
    __syncthreads();
    alt_load<R, TB, KB, 0, true>(tile, v, b0);
    __syncthreads();
    stage_free();
    alt_rotate<R, TB, KB, LO, 0>(v, T.t_post);
  }
  unsigned char* g = state + 16ull * (tile_base | alt_index<CP, H0>(b0));
#pragma unroll
  for (int j = 0; j < (1 << KB); ++j)
    El<R>::st(g + 16ull * alt_index<CP, H0>((uint32_t)j << PL::reg_lo(0)), v[j]);
}

__device__ __forceinline__ void alt_issue(const AltSet& S, const CUtensorMap* map, uint32_t tile, uint32_t bytes,
                                          unsigned char* stage, uint32_t fb) {
  const int mid = (int)(tile & ((1u << S.mid_bits) - 1u)), hi = (int)(tile >> S.mid_bits);
  const int md = S.mid_dim, hd = S.hi_dim;
  fence_proxy_async_shared();  // the CTA's generic accesses of the stage precede the copy's writes
  mbar_arrive_expect_tx(fb, bytes);
  tma_load_5d(smem_addr(stage), map, tile_coord(0, md, mid, hd, hi), tile_coord(1, md, mid, hd, hi),
              tile_coord(2, md, mid, hd, hi), tile_coord(3, md, mid, hd, hi), tile_coord(4, md, mid, hd, hi), fb);
}
// first element of a tile: the id's low bits are element bits [CP, H0), the others those above the set
template <int TB, int CP, int H0>
__device__ __forceinline__ uint32_t alt_tile_base(uint32_t tile) {
  if constexpr (CP == TB) return tile << TB;
  constexpr int mb = H0 - CP;
  return ((tile & ((1u << mb) - 1u)) << CP) | ((tile >> mb) << (H0 + TB - CP));
}

// A plain pass on one staged tile of the A set (2^12 elements, loaded through the
// 128-byte TMA swizzle so that the first round reads without bank conflicts; the
// rounds of the warp-local A1, then the top four bits): three rounds, the last
// one's lanes over the low bits.
template <class R, class W, class F>
__device__ __forceinline__ void alt_tile_plain(unsigned char* tile, unsigned char* state, R t, uint32_t tile_base,
                                               W&& wait, F&& stage_free) {
  using PL = PlanA1Warp;
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint32_t ba = pdep(lane, PL::R1_LANE) | (warp << 9);
  typename El<R>::T v[16];
  wait();
  {
    const uint32_t sb = ba ^ ((ba >> 3) & 7u);
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const uint32_t o = pdep((uint32_t)j, PL::R1_REG);
      v[j] = El<R>::ld(tile + 16u * (sb ^ o ^ ((o >> 3) & 7u)));
    }
  }
  el_bflys<R, PL::R1_REG, PL::R1_REG>(v, t);
  el_store_swz<R, PL::R1_REG>(tile, v, alt_fresh(ba));  // a thread's 128-byte groups are its own: no hazard
  __syncwarp();
  const uint32_t bb = pdep(lane, PL::R2_LANE) | (warp << 9);
  el_load<R, PL::R2_REG, true>(tile, v, alt_fresh(bb));
  el_bflys<R, PL::R2_REG, PL::R2_REG>(v, t);
  el_store_swz<R, PL::R2_REG>(tile, v, alt_fresh(bb));
  __syncthreads();
  const uint32_t bc = lane | (warp << 5);
  el_load<R, 0xF00u, true>(tile, v, bc);
  __syncthreads();
  stage_free();
  el_bflys<R, 0xF00u, 0xF00u>(v, t);
  unsigned char* g = state + 16ull * (tile_base | bc);
#pragma unroll
  for (int j = 0; j < 16; ++j) El<R>::st(g + 16ull * ((uint32_t)j << 8), v[j]);
}

// thread 0: wait until `ctr` reaches `target`; false on timeout or abort
__device__ __forceinline__ bool alt_wait(const AltBarrier& B, const unsigned int* ctr, uint32_t target) {
  uint32_t polls = 0;
  while ((int32_t)(ld_acquire(ctr) - target) < 0) {
    if (++polls > B.poll_limit) {
      atomicCAS(B.err, 0, DEV_TIMEOUT);
      atomicExch(B.abort, 1);
      return false;
    }
    if ((polls & 63u) == 0u && aborted(B.abort)) return false;
  }
  fence_proxy_async_global();  // the TMA reads what the barrier released
  return true;
}

// dynamic shared memory: the tile, a word of E per element, the CTA's control
// block, the phase table
struct AltCtl {
  uint64_t full_bar;
  int stop;      // the run has failed: every thread leaves at the end of the pass
  int inflight;  // thread 0: a tile's copy is on its way
  double acc[16][3];  // per warp: norm, P_<, <d_H> of the pass (three sets); batch: of a row's units
  // batch: the statevector the group works on
  const CUtensorMap* map;
  unsigned char* state;
  const void *tan, *scale;
  double* partials;
  int e0;
  uint32_t s0;
};
template <int TB>
struct AltSmem {
  static constexpr int kEOff = 16 << TB, kCtlOff = kEOff + (4 << TB), kTabOff = kCtlOff + 640;
  static_assert(sizeof(AltCtl) <= 640, "the control block's room");
  // + room to align the tile to 1024 bytes (swizzled loads)
  static int bytes(int n_j, int entry) { return kTabOff + (((n_j + 1) * entry + 127) & ~127) + 1024; }
};

// One CTA of a run's group. kBatch: the statevector's fields come from the control
// block (the group changes them), else from the kernel parameter.
template <class R, int TB, int KB, bool kBatch>
struct AltCta {
  using PL = AltPlan<TB, KB>;
  using SM = AltSmem<TB>;
  static constexpr uint32_t kBytes = 16u << TB;
  const AltRunDesc<R>& D;
  const AltInst<R>& I;
  const AltBarrier& B;
  unsigned int* ctr;   // the group's arrivals
  uint32_t rank, G;
  unsigned char* stage;
  uint32_t parity, epoch;

  __device__ __forceinline__ volatile AltCtl& ctl() const { return *reinterpret_cast<volatile AltCtl*>(stage + SM::kCtlOff); }
  __device__ __forceinline__ uint32_t bar() const { return smem_addr(stage) + SM::kCtlOff; }
  __device__ __forceinline__ unsigned char* es() const { return stage + SM::kEOff; }
  __device__ __forceinline__ unsigned char* tab() const { return stage + SM::kTabOff; }

  __device__ __forceinline__ unsigned char* state() const { return kBatch ? ctl().state : I.state; }
  __device__ __forceinline__ const R* tans() const { return kBatch ? static_cast<const R*>(ctl().tan) : I.tan; }
  __device__ __forceinline__ const R* scales() const { return kBatch ? static_cast<const R*>(ctl().scale) : I.scale; }
  __device__ __forceinline__ const CUtensorMap* maps() const { return kBatch ? ctl().map : I.map; }
  template <class Put>
  __device__ __forceinline__ AltMeas<Put> meas(const Put& put) const {
    if constexpr (kBatch)
      return AltMeas<Put>{const_cast<const int*>(&ctl().e0), const_cast<const uint32_t*>(&ctl().s0), put};
    else
      return AltMeas<Put>{&I.e0, &I.s0, put};
  }

  __device__ __forceinline__ void issue(int map, uint32_t tile) {
    if constexpr (alt_direct(TB)) return;
    if (threadIdx.x == 0 && tile < D.n_tiles && !ctl().stop) {
      alt_issue(D.set[map], maps() + map, tile, kBytes, stage, bar());
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
  // E of a tile of set (CP, H0) for this thread's elements at the turn
  template <int CP, int H0>
  __device__ __forceinline__ void fetch_e(uint32_t tile) {
    if (tile >= D.n_tiles) return;
    constexpr int RT = alt_turn_round(TB, KB, CP);
    AltE<R, TB, KB, CP, H0, RT>::fetch(D.E, alt_tile_base<TB, CP, H0>(tile),
                                       PL::template base<RT>(threadIdx.x & 31u, threadIdx.x >> 5), smem_addr(es()));
  }
  // The turning pass of step k on the tiles of set `s` (E of the first one already fetched).
  // kTiles: a measured row keeps the sums of every warp of every tile, so they are added up
  // in the same order whatever the number of CTAs, and a statevector of a batch measures what
  // its own run does, bit for bit. Three sets (never in a group of a batch) keep the sums of
  // a CTA: 24 bytes a warp and tile are 6 MB a row at N = 28.
  template <int CP, int H0, bool kTiles>
  __device__ __forceinline__ void turn(int s, int k) {
    AltTurn<R> T;
    const bool pre = k > D.k0;
    T.post = k < D.k1;
    T.t_pre = pre ? tans()[k - 1] : (R)0;  // a tangent of 0 rotates nothing
    T.t_post = T.post ? tans()[k] : (R)0;
    T.scale = T.post ? scales()[k] : (R)1;
    T.c0 = (uint32_t)D.c0;
    const int slot = (pre || D.meas_first) ? D.slot[k] : -1;
    T.meas = slot >= 0;
    auto unit = [&](uint32_t u) {
      return (kBatch ? ctl().partials : D.partials) + 3 * ((size_t)(slot - D.row0) * D.units + u);
    };
    if (!kTiles && T.meas && (threadIdx.x & 31u) == 0) {
      volatile double(&a)[3] = ctl().acc[threadIdx.x >> 5];
      a[0] = a[1] = a[2] = 0.0;
    }
    for (uint32_t tile = rank; tile < D.n_tiles; tile += G) {
      auto put = [&](double a, double b, double c) {
        const uint32_t warp = threadIdx.x >> 5;
        if constexpr (kTiles) {
          double* o = unit(tile * PL::kWarps + warp);
          o[0] = a;
          o[1] = b;
          o[2] = c;
        } else {
          volatile double(&acc)[3] = ctl().acc[warp];
          acc[0] = acc[0] + a;
          acc[1] = acc[1] + b;
          acc[2] = acc[2] + c;
        }
      };
      alt_tile_turn<R, TB, KB, CP, H0>(stage, state(), T, alt_tile_base<TB, CP, H0>(tile), tab(), es(), meas(put),
                                       [&]() { wait(); }, [&]() { issue(s, tile + G); });
      fetch_e<CP, H0>(tile + G);  // after the stores, when the registers are free
    }
    if (!kTiles && T.meas) {
      __syncthreads();
      if (threadIdx.x < 3u) {
        double x = 0;
        for (int w = 0; w < PL::kWarps; ++w) x += ctl().acc[w][threadIdx.x];
        unit(rank)[threadIdx.x] = x;
      }
    }
  }
  __device__ __forceinline__ void plain(int s, int k) {
    const R t = tans()[k];
    for (uint32_t tile = rank; tile < D.n_tiles; tile += G)
      alt_tile_plain<R>(stage, state(), t, alt_tile_base<TB, TB, TB>(tile), [&]() { wait(); }, [&]() { issue(s, tile + G); });
  }
  // the end of a pass: every CTA's stores are in memory
  __device__ __forceinline__ bool group_barrier() {
    if (__syncthreads_or(ctl().stop)) return false;  // every store of the CTA is issued
    if (threadIdx.x == 0) {
      red_release_add(ctr, 1u);  // releases every thread's stores (ordered before it by the CTA barrier)
      epoch += G;
      if (!alt_wait(B, ctr, epoch)) ctl().stop = 1;
    }
    // lane 0's warp waits for it here: its other lanes must not spin on the tile's
    // barrier while lane 0 polls (a warp in a suspended try_wait polls nothing)
    __syncwarp();
    return true;
  }
  // ... then the next pass's first tile
  __device__ __forceinline__ bool next_pass(int map) {
    if (!group_barrier()) return false;
    if constexpr (alt_direct(TB)) {
      if (__syncthreads_or(ctl().stop)) return false;  // thread 0 has seen every CTA's stores
    } else {
      issue(map, rank);
    }
    return true;
  }
  __device__ __forceinline__ void stage_table() {
    auto* dst = reinterpret_cast<typename AltPhase<R>::entry*>(tab());
    for (int i = (int)threadIdx.x; i <= D.n_j; i += PL::kThreads) dst[i] = D.tab[i];
    __syncthreads();
  }
  __device__ __forceinline__ void begin() {
    if (threadIdx.x == 0) {
      ctl().stop = 0;
      ctl().inflight = 0;
      mbar_init(bar(), 1);
      fence_barrier_init();
    }
    parity = epoch = 0u;
    __syncthreads();
  }
  // a copy still on its way after a failure lands before its CTA leaves
  __device__ __forceinline__ void leave() {
    if (threadIdx.x == 0 && ctl().stop && ctl().inflight) mbar_wait_bounded(bar(), parity, B.err);
  }
};

// Two sets: A (the tile's bits) and the W bits above it. False when the run has failed.
template <class R, int TB, int KB, int W, bool kBatch>
__device__ __forceinline__ bool alt_run2(AltCta<R, TB, KB, kBatch>& C) {
  const AltRunDesc<R>& D = C.D;
  if (D.k0 & 1) C.template fetch_e<TB - W, TB>(C.rank); else C.template fetch_e<TB, TB>(C.rank);
  C.issue(D.k0 & 1, C.rank);
  for (int k = D.k0;; ++k) {
    if (k & 1) {
      C.template turn<TB - W, TB, true>(1, k);
      if (k == D.k1) return true;
      C.template fetch_e<TB, TB>(C.rank);
    } else {
      C.template turn<TB, TB, true>(0, k);
      if (k == D.k1) return true;
      C.template fetch_e<TB - W, TB>(C.rank);
    }
    if (!C.next_pass((k + 1) & 1)) return false;
  }
}

// Three sets: turning passes on the W2 bits above the A set and the W3 bits above
// those in turn, plain passes over the A set between them.
template <class R, int W2, int W3, bool kBatch>
__device__ __forceinline__ bool alt_run3(AltCta<R, 12, 4, kBatch>& C) {
  constexpr int TB = 12, C2 = TB - W2, C3 = TB - W3, H3 = TB + W2;
  const AltRunDesc<R>& D = C.D;
  if (D.k0 & 1) C.template fetch_e<C3, H3>(C.rank); else C.template fetch_e<C2, TB>(C.rank);
  C.issue(1 + (D.k0 & 1), C.rank);
  for (int k = D.k0;; ++k) {
    if (k & 1)
      C.template turn<C3, H3, false>(2, k);
    else
      C.template turn<C2, TB, false>(1, k);
    if (k == D.k1) return true;
    if (!C.next_pass(0)) return false;
    C.plain(0, k);
    if (k & 1) C.template fetch_e<C2, TB>(C.rank); else C.template fetch_e<C3, H3>(C.rank);
    if (!C.next_pass(1 + ((k + 1) & 1))) return false;
  }
}

// The sums of a measured row's units, by a CTA of as many threads as the passes' and in the
// same order wherever it runs: in thread 0.
template <int TB>
constexpr int kAltRowThreads = TB == 10 ? AltPlan<10, 4>::kThreads : AltPlan<12, 4>::kThreads;
template <int kRow>
__device__ __forceinline__ void alt_row_sum(const double* part, uint32_t units, volatile double (*red)[3], double (&s)[3]) {
  const uint32_t t = threadIdx.x;
  s[0] = s[1] = s[2] = 0.0;
#pragma unroll 4
  for (uint32_t u = t; u < units; u += kRow)
#pragma unroll
    for (int q = 0; q < 3; ++q) s[q] += __ldcg(&part[3 * (size_t)u + q]);
#pragma unroll
  for (int q = 0; q < 3; ++q) s[q] = warp_sum(s[q]);
  __syncthreads();  // the last row's sums have been read
  if ((t & 31u) == 0)
#pragma unroll
    for (int q = 0; q < 3; ++q) red[t >> 5][q] = s[q];
  __syncthreads();
  if (t == 0)
    for (int w = 1; w < kRow / 32; ++w)
#pragma unroll
      for (int q = 0; q < 3; ++q) s[q] += red[w][q];
}

__device__ __forceinline__ unsigned char* alt_stage(unsigned char* raw) {
  return raw + ((1024u - (smem_addr(raw) & 1023u)) & 1023u);
}

// W3 = 0: two sets (A and W2), else three
template <class R, int TB, int KB, int W2, int W3>
__global__ void __launch_bounds__(AltPlan<TB, KB>::kThreads, TB == 10 ? 6 : TB == 12 ? 2 : 1)
    alt_kernel(const __grid_constant__ AltRunDesc<R> D, const __grid_constant__ AltInst<R> I,
               const __grid_constant__ AltBarrier B) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  AltCta<R, TB, KB, false> C{D, I, B, B.ctr, blockIdx.x, gridDim.x, alt_stage(smem_raw)};
  C.begin();
  C.stage_table();
  if constexpr (W3 == 0)
    alt_run2<R, TB, KB, W2>(C);
  else
    alt_run3<R, W2, W3>(C);
  C.leave();
}

// Many statevectors of one size: groups of Q.G CTAs work through them on their own,
// each with its own barrier, so a small statevector's barriers and waits overlap
// those of the other groups. Results are reduced by the group (units in index
// order) after the statevector's last pass, from one of two partial-sum buffers:
// the next use of a buffer lies behind the barriers of the statevector between.
template <class R, int TB, int KB, int W2, int W3>
__global__ void __launch_bounds__(AltPlan<TB, KB>::kThreads, TB == 10 ? 6 : TB == 12 ? 2 : 1)
    alt_batch_kernel(const __grid_constant__ AltRunDesc<R> D, const __grid_constant__ AltBatch<R> Q,
                     const __grid_constant__ AltBarrier B) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  const uint32_t group = blockIdx.x / Q.G, n_groups = gridDim.x / Q.G;
  AltCta<R, TB, KB, true> C{D, *Q.inst, B, B.ctr + 32u * group, blockIdx.x % Q.G, Q.G, alt_stage(smem_raw)};
  C.begin();
  C.stage_table();
  uint32_t turn = 0;
  bool ok = true;
  for (int i = (int)group; ok && i < Q.n_inst; i += (int)n_groups, ++turn) {
    const AltInst<R>& I = Q.inst[i];
    double* part = D.partials + (2 * (size_t)group + (turn & 1u)) * Q.part_stride;
    if (threadIdx.x == 0) {
      volatile AltCtl& c = C.ctl();
      c.map = I.map;
      c.state = I.state;
      c.tan = I.tan;
      c.scale = I.scale;
      c.partials = part;
      c.e0 = I.e0;
      c.s0 = I.s0;
    }
    __syncthreads();
    if constexpr (W3 == 0)
      ok = alt_run2<R, TB, KB, W2>(C);
    else
      ok = alt_run3<R, W2, W3>(C);
    if (!ok || !(ok = C.group_barrier())) break;
    if (__syncthreads_or(C.ctl().stop)) break;  // also: thread 0 has seen every CTA's partial sums
    static_assert(kAltRowThreads<TB == 13 ? 12 : TB> == AltPlan<TB, KB>::kThreads, "the CTA sums a row");
    for (int row = (int)C.rank; row < Q.n_rows; row += (int)Q.G) {
      double s[3];
      alt_row_sum<AltPlan<TB, KB>::kThreads>(part + 3 * (size_t)row * D.units, D.units, C.ctl().acc, s);
      if (threadIdx.x == 0) {
        double* out = I.results + 4 * (size_t)(D.row0 + row);
        out[0] = s[1];
        out[1] = s[2];
        out[2] = s[0];
      }
    }
    __syncthreads();
  }
  C.leave();
}

#ifdef BK_ALT_REDUCE  // defined by the one source that launches it
// results[row0 + row] = sum over a row's units in a fixed order (a CTA a row)
template <int kRow>
__global__ void __launch_bounds__(kRow)
    alt_reduce_kernel(const double* __restrict__ partials, uint32_t units, double* __restrict__ results) {
  __shared__ volatile double red[16][3];
  const int row = (int)blockIdx.x;
  double s[3];
  alt_row_sum<kRow>(partials + 3 * (size_t)row * units, units, red, s);
  if (threadIdx.x == 0) {
    results[4 * (size_t)row + 0] = s[1];
    results[4 * (size_t)row + 1] = s[2];
    results[4 * (size_t)row + 2] = s[0];
  }
}

#endif

// The kernel of a geometry (tile bits, set widths), or nullptr: instantiated in
// bk_alt_f32.cu and bk_alt_f64.cu.
const void* alt_kernel_f32(int tb, int w2, int w3, bool batch);
const void* alt_kernel_f64(int tb, int w2, int w3, bool batch);

template <class R, int TB, int KB, int W2, int W3>
const void* alt_pick(bool batch) {
  // larger statevectors fill the GPU one at a time, complex64 members up to 18 qubits
  // (W2 < 8 of the 2^10-element tiles) compute in complex128
  if constexpr (W3 == 0 && !(sizeof(R) == 4 && TB == 10 && W2 < 8))
    if (batch) return reinterpret_cast<const void*>(alt_batch_kernel<R, TB, KB, W2, W3>);
  return batch ? nullptr : reinterpret_cast<const void*>(alt_kernel<R, TB, KB, W2, W3>);
}
template <class R>
const void* alt_kernel_table(int tb, int w2, int w3, bool batch) {
  switch (tb * 256 + w2 * 16 + w3) {
    case 0xA30: return alt_pick<R, 10, 4, 3, 0>(batch);
    case 0xA40: return alt_pick<R, 10, 4, 4, 0>(batch);
    case 0xA50: return alt_pick<R, 10, 4, 5, 0>(batch);
    case 0xA60: return alt_pick<R, 10, 4, 6, 0>(batch);
    case 0xA70: return alt_pick<R, 10, 4, 7, 0>(batch);
    case 0xA80: return alt_pick<R, 10, 4, 8, 0>(batch);
    case 0xC70: return alt_pick<R, 12, 4, 7, 0>(batch);
    case 0xC80: return alt_pick<R, 12, 4, 8, 0>(batch);
    case 0xC90: return alt_pick<R, 12, 4, 9, 0>(batch);
    case 0xD90: return alt_pick<R, 13, 5, 9, 0>(batch);
    case 0xDA0: return alt_pick<R, 13, 5, 10, 0>(batch);
    case 0xC66: return alt_pick<R, 12, 4, 6, 6>(batch);
    case 0xC76: return alt_pick<R, 12, 4, 7, 6>(batch);
    case 0xC77: return alt_pick<R, 12, 4, 7, 7>(batch);
    case 0xC87: return alt_pick<R, 12, 4, 8, 7>(batch);
    case 0xC88: return alt_pick<R, 12, 4, 8, 8>(batch);
    case 0xC98: return alt_pick<R, 12, 4, 9, 8>(batch);
    case 0xC99: return alt_pick<R, 12, 4, 9, 9>(batch);
    default: return nullptr;
  }
}

}  // namespace bk
