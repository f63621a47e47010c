// Full-space Hamiltonian matvec and Lanczos building blocks (sm_100a).
//
// The reference's full-space Krylov solver (src/subspace/diagonalizer.cuh:377-416,
// driver :418-560) multiplies by H = diag(scale E(s)) - g sum_j X_j with one
// thread per basis state gathering its N neighbours i ^ 2^j from global memory
// (fullspace_matvec_kernel_d, :60-77). On a B200 the 126 MB L2 already serves
// that form's neighbours up to ~2^23 states away, and the DRAM cost is the far
// neighbours. Here one product is:
//   up to 22 bits a block pass (fs_block_kernel): 8192-state blocks, the block of x
//     staged in shared memory by a bulk copy for the 13 low-bit neighbours, the others
//     as coalesced sweeps of the partner blocks (L2 hits), the diagonal from the cached
//     uint16 E table;
//   beyond, tile passes in one launch (fs_turn_kernel).
//
// Lanczos steps (the driver's cuBLAS calls, :437-482) are fused element-wise
// kernels with per-block partial sums reduced in a fixed order (deterministic).
#pragma once
#include "bk_device.cuh"
#include "bk_s23.cuh"

namespace bk {

constexpr int kFsTileBits = 13;  // 8192 doubles per tile
constexpr int kFsThreads = 256;
constexpr int kLzBlocks = 296;   // partial-sum blocks of the Lanczos reductions (2 per SM on a B200)

// One neighbour-sum pass over a tile smaller than 8192 doubles (n < 13: the
// whole vector in one CTA). Tile position p -> state index: bits [0, cp) stay,
// bits [cp, tb) go to [h0, h0 + tb - cp); the tile id splits into mb "mid" bits
// (index bits [cp, h0)) and the bits above h0 + tb - cp. first: pass 0 (writes
// the diagonal term); act_lo: lowest tile bit whose neighbours this pass sums.
__global__ void __launch_bounds__(kFsThreads) fs_pass_kernel(const double* __restrict__ x, double* __restrict__ y,
                                                             const uint16_t* __restrict__ E, double scale, double g,
                                                             int tb, int cp, int h0, int mb, int first, int act_lo) {
  extern __shared__ __align__(16) double ft[];
  const uint32_t tile = blockIdx.x;
  const int w = tb - cp;
  const uint64_t mid = tile & ((1u << mb) - 1u), hi = tile >> mb;
  const uint64_t base = (mid << cp) | (hi << (h0 + w));
  const uint32_t size = 1u << tb, lo_mask = (1u << cp) - 1u;
  for (uint32_t p = threadIdx.x; p < size; p += kFsThreads)
    ft[p] = x[base | (p & lo_mask) | ((uint64_t)(p >> cp) << h0)];
  __syncthreads();
  for (uint32_t p = threadIdx.x; p < size; p += kFsThreads) {
    double s = 0.0;
    for (int b = act_lo; b < tb; ++b) s += ft[p ^ (1u << b)];
    const uint64_t gi = base | (p & lo_mask) | ((uint64_t)(p >> cp) << h0);
    y[gi] = first ? scale * (double)E[gi] * ft[p] - g * s : y[gi] - g * s;
  }
}


constexpr int kFsPer = (1 << kFsTileBits) / kFsThreads;  // 32 tile positions per thread
// Up to 22 bits: CTA = one 8192-state block (index bits 0-12). The block of x arrives
// in shared memory by one 64 KB bulk copy; the 13 low-bit neighbours are read there.
// Each bit j from 13 on pairs the block with the block 2^(j-13) away, read as one
// coalesced sweep (32 loads in flight per thread) into register accumulators: the
// partner is in L2 (x is 32 MB at most).
__global__ void __launch_bounds__(kFsThreads, 2) fs_block_kernel(const double* __restrict__ x, double* __restrict__ y,
                                                                 const uint16_t* __restrict__ E, double scale, double g,
                                                                 int n_gather, int* err) {
  extern __shared__ __align__(128) double ft[];
  __shared__ __align__(8) uint64_t bar;
  const uint32_t tid = threadIdx.x;
  const uint64_t base = (uint64_t)blockIdx.x << kFsTileBits;
  const uint32_t fb = smem_addr(&bar);
  if (tid == 0) {
    mbar_init(fb, 1);
    fence_barrier_init();
    mbar_arrive_expect_tx(fb, 8u << kFsTileBits);
    bulk_load(smem_addr(ft), x + base, 8u << kFsTileBits, fb);
  }
  // no thread may poll the barrier before thread 0 has initialised it (an SM's
  // shared memory can still hold a completed barrier of an earlier CTA)
  __syncthreads();
  double acc[kFsPer];
#pragma unroll
  for (int k = 0; k < kFsPer; ++k) acc[k] = 0.0;
  // high bits first (global, mostly L2), while the block's own copy is in flight
  for (int j = kFsTileBits; j < n_gather; ++j) {
    const double* nb = x + (base ^ (1ull << j));
#pragma unroll
    for (int k = 0; k < kFsPer; ++k) acc[k] += __ldg(nb + tid + kFsThreads * k);
  }
  const bool ok = mbar_wait_bounded(fb, 0, err);
  if (__syncthreads_or(!ok)) return;
#pragma unroll
  for (int k = 0; k < kFsPer; ++k) {
    const uint32_t p = tid + kFsThreads * (uint32_t)k;
    double s = 0.0;
#pragma unroll
    for (int b = 0; b < kFsTileBits; ++b) s += ft[p ^ (1u << b)];
    const double v = scale * (double)E[base + p] * ft[p] - g * (s + acc[k]);
    __stcs(y + base + p, v);
  }
}

// ---------------------------------------------------------------------------
// Product in tile passes, one cooperative launch (n >= 23). The index bits are split
// into A = [0, 13), S1 = [13, 13 + w1) and S2 = the w2 bits above;
// a tile is 8192 doubles of x, an S tile 2^w rows of 2^(13 - w) contiguous ones:
//   1. S2 over the whole vector:  y  = -g sum_S2
//   2. slab by slab (the 2^(13 + w1) states of one value of the S2 bits):
//      A:  y += scale E x - g sum_A;   S1: y -= g sum_S1
// S1 of a slab is queued `lag` slabs behind its A tiles, so x and y of the slab are
// still in L2: DRAM sees x twice, y twice written and once read and E once, 42 bytes a
// state (43.6 in a profile at N = 27). Sweeping the ten bits above A through L2 instead, 80 bytes a
// state of L2 reads, took 1.82 ms at N = 27 with the far bits' pass; this takes 1.27 ms,
// bound by the chain of one tile (x, y, sums from shared memory, stores), which the two
// CTAs of an SM hide from each other in part. A tile's x is loaded (TMA) once the tile
// before it is summed; a thread keeps the 32 doubles of the top five tile bits in
// registers, so those neighbours need no shared-memory read, and reads the others from
// the tile. Tasks are dealt to the CTAs in order; a slab's counter is awaited only by
// S1 tiles, whose CTA owes nothing while it waits. Every wait is bounded.
// ---------------------------------------------------------------------------
constexpr int kFtThreads = 256;
constexpr int kFtPer = (1 << kFsTileBits) / kFtThreads;  // 32
constexpr int kFtChunk = 4;                              // states of a thread summed at once
constexpr int kFtAhead = 3;                              // chunks of y in registers: one in use, two on their way
constexpr int kFtSmem = (8 << kFsTileBits) + 128;        // the tile + alignment slack

struct FtParams {
  CUtensorMap map1, map2;  // x tiles of S1, S2
  const double* x;
  double* y;
  const uint16_t* E;
  double scale, g;
  int w1, w2;
  int mid1, hi1, mid2, hi2;  // tensor-map dimensions of an S tile id's parts
  uint32_t tiles;            // 2^(n - 13)
  uint32_t slabs, lag;
  unsigned int* done;        // [slabs] finished A tiles
  unsigned int* arrived;     // CTAs past phase 1
  int* err;
  int* abort;
  uint32_t poll_limit;
};

// thread 0: bounded wait for a counter
__device__ __forceinline__ bool ft_wait(const FtParams& P, const unsigned int* ctr, uint32_t target) {
  uint32_t polls = 0;
  while (ld_acquire(ctr) < target) {
    if (++polls > P.poll_limit) {
      atomicCAS(P.err, 0, DEV_TIMEOUT);
      atomicExch(P.abort, 1);
      return false;
    }
    if ((polls & 63u) == 0u && *reinterpret_cast<const volatile int*>(P.abort) != 0) return false;
  }
  return true;
}

enum FtKind : uint32_t { FT_A = 0, FT_S1 = 1, FT_S2 = 2, FT_END = 3 };
struct FtTask {
  uint32_t kind, tile, slab;
};
// task g of the launch: the S2 tiles, then per slab its A tiles and, `lag` slabs later, its S1 tiles
__device__ __forceinline__ FtTask ft_task(const FtParams& P, uint32_t g) {
  const uint32_t n2 = P.w2 > 0 ? P.tiles : 0u, per = P.tiles / P.slabs;
  if (g < n2) return FtTask{FT_S2, g, 0u};
  g -= n2;
  if (g >= 2u * P.tiles) return FtTask{FT_END, 0u, 0u};
  // blocks of `per` tasks: A(0) .. A(lag - 1), then A(h + lag), S1(h) alternating, then the last S1
  const uint32_t b = g / per, i = g - b * per;
  uint32_t slab;
  bool first;
  if (b < P.lag) {
    first = true;
    slab = b;
  } else if (b < P.lag + 2u * (P.slabs - P.lag)) {
    first = ((b - P.lag) & 1u) == 0u;
    slab = (b - P.lag) / 2u + (first ? P.lag : 0u);
  } else {
    first = false;
    slab = b - P.slabs;
  }
  return FtTask{first ? FT_A : FT_S1, slab * per + i, slab};
}

// sum of a register double's neighbours over tile bits 8-12
__device__ __forceinline__ double ft_register_sum(const double (&x)[kFtPer], int j) {
  return (x[j ^ 1] + x[j ^ 2]) + (x[j ^ 4] + x[j ^ 8]) + x[j ^ 16];
}

__global__ void __launch_bounds__(kFtThreads, 2) fs_turn_kernel(const __grid_constant__ FtParams P) {
  extern __shared__ __align__(128) unsigned char ft_raw[];
  __shared__ __align__(8) uint64_t bar;
  __shared__ int stop_word;
  volatile int* stop = &stop_word;
  unsigned char* stage = ft_raw + ((128u - (smem_addr(ft_raw) & 127u)) & 127u);
  const double* ft = reinterpret_cast<const double*>(stage);
  const uint32_t tid = threadIdx.x, fb = smem_addr(&bar);
  constexpr uint32_t kBytes = 8u << kFsTileBits;
  if (tid == 0) {
    *stop = 0;
    mbar_init(fb, 1);
    fence_barrier_init();
  }
  __syncthreads();
  const uint64_t keep = policy_evict_last();  // x and y of a slab, between its A and its S1 tiles
  auto issue = [&](const FtTask& t) {
    if (tid != 0 || t.kind == FT_END || *stop) return;
    const uint32_t dst = smem_addr(stage);
    fence_proxy_async_shared();
    mbar_arrive_expect_tx(fb, kBytes);
    if (t.kind == FT_A) {
      bulk_load_hint(dst, P.x + ((size_t)t.tile << kFsTileBits), kBytes, fb, policy_evict_last());  // S1 reads it again
    } else {
      const bool s1 = t.kind == FT_S1;
      const int mb = s1 ? P.w1 : P.w1 + P.w2;  // index bits between the rows' contiguous part and the set
      const int md = s1 ? P.mid1 : P.mid2, hd = s1 ? P.hi1 : P.hi2;
      const int mid = (int)(t.tile & ((1u << mb) - 1u)), hi = (int)(t.tile >> mb);
      tma_load_5d_hint(dst, s1 ? &P.map1 : &P.map2, tile_coord(0, md, mid, hd, hi), tile_coord(1, md, mid, hd, hi),
                       tile_coord(2, md, mid, hd, hi), tile_coord(3, md, mid, hd, hi), tile_coord(4, md, mid, hd, hi),
                       fb, policy_evict_first());
    }
  };
  const bool two = P.w2 > 0;
  bool joined = !two;  // phase 1 is behind every CTA
  FtTask t = ft_task(P, blockIdx.x);
  issue(t);
  uint32_t it = 0;
  for (; t.kind != FT_END; ++it) {
    const FtTask nt = ft_task(P, blockIdx.x + (it + 1u) * gridDim.x);
    if (t.kind != FT_S2 && (!joined || t.kind == FT_S1)) {
      // y of phase 1 from every CTA, or of the slab's A tiles
      if (tid == 0) {
        bool ok = true;
        if (!joined) {
          red_release_add(P.arrived, 1u);
          ok = ft_wait(P, P.arrived, gridDim.x);
        }
        if (ok && t.kind == FT_S1) ok = ft_wait(P, P.done + t.slab, P.tiles / P.slabs);
        if (!ok) *stop = 1;
      }
      joined = true;
      if (__syncthreads_or(*stop)) break;
    }
    // where the thread's doubles live: tile position p = tid + 256 j
    const int w = t.kind == FT_A ? 0 : t.kind == FT_S1 ? P.w1 : P.w2;
    size_t base, step;  // first state, distance of the states of neighbouring j
    if (t.kind == FT_A) {
      base = ((size_t)t.tile << kFsTileBits) + tid;
      step = kFtThreads;
    } else {
      const int cp = kFsTileBits - w, h0 = t.kind == FT_S1 ? kFsTileBits : kFsTileBits + P.w1, mb = h0 - cp;
      const size_t mid = t.tile & ((1u << mb) - 1u), hi = t.tile >> mb;
      base = (mid << cp) | (hi << (h0 + w)) | (tid & ((1u << cp) - 1u)) | ((size_t)(tid >> cp) << h0);
      step = (size_t)(kFtThreads >> cp) << h0;
    }
    double* y = P.y + base;
    double yv[kFtAhead][kFtChunk];
    constexpr int kChunks = kFtPer / kFtChunk;
    if (t.kind == FT_A) {
      const uint16_t* E = P.E + base;
      uint32_t ev[kFtAhead][kFtChunk];
      auto fetch = [&](int c) {
#pragma unroll
        for (int i = 0; i < kFtChunk; ++i) {
          const size_t o = (size_t)(c * kFtChunk + i) * step;
          ev[c % kFtAhead][i] = __ldg(E + o);
          yv[c % kFtAhead][i] = two ? __ldcs(y + o) : 0.0;
        }
      };
      fetch(0);
      fetch(1);
      if (!mbar_wait_bounded(fb, it & 1u, P.err)) *stop = 1;
      double x[kFtPer];
#pragma unroll
      for (int j = 0; j < kFtPer; ++j) x[j] = ft[tid + kFtThreads * j];
#pragma unroll
      for (int c = 0; c < kChunks; ++c) {
        if (c + 2 < kChunks) fetch(c + 2);
#pragma unroll
        for (int i = 0; i < kFtChunk; ++i) {
          const int j = c * kFtChunk + i;
          const double* q = ft + kFtThreads * j;
          double a = ft_register_sum(x, j);
#pragma unroll
          for (int b = 0; b < 8; ++b) a += q[tid ^ (1u << b)];
          st_global_hint(y + (size_t)j * step,
                         yv[c % kFtAhead][i] + (P.scale * (double)ev[c % kFtAhead][i] * x[j] - P.g * a), keep);
        }
      }
    } else {
      const bool add = t.kind == FT_S1;
      auto fetch = [&](int c) {
#pragma unroll
        for (int i = 0; i < kFtChunk; ++i)
          yv[c % kFtAhead][i] = add ? __ldcg(y + (size_t)(c * kFtChunk + i) * step) : 0.0;
      };
      fetch(0);
      fetch(1);
      if (!mbar_wait_bounded(fb, it & 1u, P.err)) *stop = 1;
      double x[kFtPer];
#pragma unroll
      for (int j = 0; j < kFtPer; ++j) x[j] = ft[tid + kFtThreads * j];
#pragma unroll
      for (int c = 0; c < kChunks; ++c) {
        if (c + 2 < kChunks) fetch(c + 2);
        double s[kFtChunk];
#pragma unroll
        for (int i = 0; i < kFtChunk; ++i) s[i] = ft_register_sum(x, c * kFtChunk + i);  // w >= 5: the set's bits
        for (int b = kFsTileBits - w; b < 8; ++b) {
#pragma unroll
          for (int i = 0; i < kFtChunk; ++i) s[i] += ft[kFtThreads * (c * kFtChunk + i) + (tid ^ (1u << b))];
        }
#pragma unroll
        for (int i = 0; i < kFtChunk; ++i)
          __stcs(y + (size_t)(c * kFtChunk + i) * step, yv[c % kFtAhead][i] - P.g * s[i]);
      }
    }
    __syncthreads();
    issue(nt);
    // (the barrier above is behind every store of the task)
    if (tid == 0 && t.kind == FT_A) red_release_add(P.done + t.slab, 1u);
    t = nt;
    if (__syncthreads_or(*stop)) break;
  }
  // a failed run: the copy of task `it` (phase it) may still be on its way, and lands before
  // the CTA leaves; none was issued behind it, stop was set first
  if (tid == 0 && *stop) mbar_wait_bounded(fb, it & 1u, P.err);
}

// The reference's form (diagonalizer.cuh:60-77): one thread per state, its n
// neighbours gathered from global memory in bit order (the BK_PLAIN comparison).
__global__ void __launch_bounds__(256) fs_plain_kernel(const double* __restrict__ x, double* __restrict__ y,
                                                       const uint16_t* __restrict__ E, double scale, double g, int n,
                                                       uint64_t N) {
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  double yi = (double)E[i] * scale * x[i];
  for (int j = 0; j < n; ++j) yi -= g * x[i ^ (1ull << j)];
  y[i] = yi;
}

__device__ __forceinline__ double block_sum(double v, double* red) {
  v = warp_sum(v);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) red[warp] = v;
  __syncthreads();
  double s = 0.0;
  if (threadIdx.x == 0)
    for (int i = 0; i < (int)(blockDim.x >> 5); ++i) s += red[i];
  return s;  // valid in thread 0
}

// w -= beta[jb] * vprev (jb >= 0); partials[block] = sum of v * w over the block's states
__global__ void __launch_bounds__(256) lz_orth_dot_kernel(double* __restrict__ w, const double* __restrict__ vprev,
                                                          const double* __restrict__ v, const double* __restrict__ beta,
                                                          int jb, uint64_t N, double* __restrict__ partials) {
  __shared__ double red[8];
  const double b = jb >= 0 ? beta[jb] : 0.0;
  double acc = 0.0;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < N; i += (uint64_t)gridDim.x * blockDim.x) {
    double wi = w[i];
    if (jb >= 0) wi -= b * vprev[i];
    w[i] = wi;
    acc += v[i] * wi;
  }
  const double s = block_sum(acc, red);
  if (threadIdx.x == 0) partials[blockIdx.x] = s;
}

// w -= alpha[ja] * v; partials[block] = sum of w^2
// w and v may be the same vector (the start vector's norm): no __restrict__ on them
__global__ void __launch_bounds__(256) lz_axpy_nrm_kernel(double* w, const double* v,
                                                          const double* __restrict__ alpha, int ja, uint64_t N,
                                                          double* __restrict__ partials) {
  __shared__ double red[8];
  const double a = ja >= 0 ? alpha[ja] : 0.0;
  double acc = 0.0;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < N; i += (uint64_t)gridDim.x * blockDim.x) {
    const double wi = w[i] - a * v[i];
    if (ja >= 0) w[i] = wi;
    acc += wi * wi;
  }
  const double s = block_sum(acc, red);
  if (threadIdx.x == 0) partials[blockIdx.x] = s;
}

// out[slot] = sum of partials[0..count) in a fixed order (sqrt of it when take_sqrt)
__global__ void lz_reduce_kernel(const double* __restrict__ partials, int count, double* __restrict__ out, int slot,
                                 int take_sqrt) {
  __shared__ double red[8];
  double acc = 0.0;
  for (int i = threadIdx.x; i < count; i += blockDim.x) acc += partials[i];
  const double s = block_sum(acc, red);
  if (threadIdx.x == 0) out[slot] = take_sqrt ? sqrt(s) : s;
}

// dst = src * (1 / norm[slot]); dst may equal src (in-place normalisation), so
// neither is __restrict__
__global__ void __launch_bounds__(256) lz_scale_kernel(double* dst, const double* src,
                                                       const double* __restrict__ norm, int slot, uint64_t N) {
  const double inv = 1.0 / norm[slot];
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < N; i += (uint64_t)gridDim.x * blockDim.x)
    dst[i] = src[i] * inv;
}

// x = sum_j V[j] * coef[j] (a Ritz vector from the Krylov basis)
__global__ void __launch_bounds__(256) lz_combine_kernel(const double* __restrict__ V, const double* __restrict__ coef,
                                                         int m, uint64_t N, double* __restrict__ x) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < N; i += (uint64_t)gridDim.x * blockDim.x) {
    double s = 0.0;
    for (int j = 0; j < m; ++j) s += V[(uint64_t)j * N + i] * coef[j];
    x[i] = s;
  }
}

}  // namespace bk
