// radix.cuh — stable LSD radix sorts: the one-sweep sort of the allocating paths (ingest.cu,
// exec_pagerank.cu) and the histogram / scan / scatter passes of the allocation-free batch
// path (noalloc.cu), whose fixed scratch has no room for look-back state.
#pragma once
#include <stdint.h>
#include <cuda_runtime.h>

namespace cytom {

// Allocation-free passes: 256 threads per tile, IPT keys per thread. Small tiles (IPT 4)
// give every SM many independent warps, which the latency-bound ranking and scatter need.
constexpr int RS_T = 256, RS_WARPS = RS_T / 32;
constexpr int RS_IPT_SMALL = 4;

// Per-tile digit counts of one 8-bit pass, digit-major: hist[digit * nb + tile].
// Stable scatter of one pass given the exclusive scan of the histogram.
template <int IPT>
__global__ void radix_upsweep_kernel(const uint64_t* __restrict__ keys, uint64_t n, int shift,
                                     uint32_t* __restrict__ hist, uint32_t nb) {
  __shared__ uint32_t cnt[256];
  cnt[threadIdx.x] = 0;
  __syncthreads();
  uint64_t base = (uint64_t)blockIdx.x * (RS_T * IPT);
  uint32_t d_reg[IPT];
#pragma unroll
  for (int k = 0; k < IPT; ++k) {
    uint64_t i = base + (uint64_t)k * RS_T + threadIdx.x;
    d_reg[k] = (i < n) ? (uint32_t)((keys[i] >> shift) & 0xFF) : 256u;
  }
  // warp-aggregated counts (skewed digits would serialise per-key shared atomics)
  const unsigned lane = threadIdx.x & 31;
#pragma unroll
  for (int k = 0; k < IPT; ++k) {
    const unsigned peers = __match_any_sync(0xFFFFFFFFu, d_reg[k]);
    if (d_reg[k] < 256u && (__ffs(peers) - 1) == (int)lane) atomicAdd(&cnt[d_reg[k]], (uint32_t)__popc(peers));
  }
  __syncthreads();
  hist[(uint64_t)threadIdx.x * nb + blockIdx.x] = cnt[threadIdx.x];
}

template <int IPT>
__global__ void radix_downsweep_kernel(const uint64_t* __restrict__ keys, const uint32_t* __restrict__ vals,
                                       uint64_t n, int shift, const uint32_t* __restrict__ offs, uint32_t nb,
                                       uint64_t* __restrict__ keys_out, uint32_t* __restrict__ vals_out) {
  __shared__ uint32_t wcnt[RS_WARPS][256];
  __shared__ uint32_t base_d[256];
  const unsigned lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const unsigned lt = (1u << lane) - 1u;
  for (int d = threadIdx.x; d < RS_WARPS * 256; d += RS_T) (&wcnt[0][0])[d] = 0;
  base_d[threadIdx.x] = offs[(uint64_t)threadIdx.x * nb + blockIdx.x];
  __syncthreads();
  const uint64_t wbase = (uint64_t)blockIdx.x * (RS_T * IPT) + (uint64_t)wid * (32 * IPT);
  // every key and value is loaded before any is used
  uint64_t k_reg[IPT];
  uint32_t v_reg[IPT];
  uint32_t d_reg[IPT];
#pragma unroll
  for (int k = 0; k < IPT; ++k) {
    uint64_t i = wbase + (uint64_t)k * 32 + lane;
    k_reg[k] = (i < n) ? keys[i] : 0ULL;
    v_reg[k] = (vals && i < n) ? vals[i] : 0u;
    d_reg[k] = (i < n) ? (uint32_t)((k_reg[k] >> shift) & 0xFF) : 256u;
  }
  // phase 1: each key's rank among the warp's keys of its digit, in input order
  uint32_t r_reg[IPT];
#pragma unroll
  for (int k = 0; k < IPT; ++k) {
    const uint32_t d = d_reg[k];
    const unsigned peers = __match_any_sync(0xFFFFFFFFu, d);
    const int leader = __ffs(peers) - 1;
    uint32_t old = 0;
    if ((int)lane == leader && d < 256u) {
      old = wcnt[wid][d];
      wcnt[wid][d] = old + __popc(peers);
    }
    r_reg[k] = __shfl_sync(0xFFFFFFFFu, old, leader) + __popc(peers & lt);
    __syncwarp();
  }
  __syncthreads();
  // phase 2: exclusive prefix across warps per digit
  {
    uint32_t run = 0;
    const int d = threadIdx.x;
#pragma unroll
    for (int w = 0; w < RS_WARPS; ++w) {
      uint32_t t = wcnt[w][d];
      wcnt[w][d] = run;
      run += t;
    }
  }
  __syncthreads();
  // phase 3: scatter (stable: block offset + warp offset + rank)
#pragma unroll
  for (int k = 0; k < IPT; ++k) {
    const uint32_t d = d_reg[k];
    if (d < 256u) {
      const uint32_t pos = base_d[d] + wcnt[wid][d] + r_reg[k];
      keys_out[pos] = k_reg[k];
      if (vals) vals_out[pos] = v_reg[k];
    }
  }
}

// ---- one-sweep sort ------------------------------------------------------------------
// Digits of up to 9 bits, as equal as the key's bits allow (os_plan: a 44-bit edge key takes
// 5 passes, not 6). One kernel counts every pass's digits; each pass is then one kernel that
// reads its keys once: a block takes the next tile, ranks its keys per digit, publishes the
// tile's digit counts, orders the keys in shared memory, adds up the counts of the tiles
// before it (decoupled look-back, OS_LB status rows in flight per step) and writes the
// tile's runs coalesced. Tiles are taken in order from a ticket, so a tile only ever looks
// at tiles whose blocks are already running. A status row that stays empty for OS_POLLS
// polls (fewer where a test says so) is not waited for any longer: the thread counts that
// tile's keys itself.
// Bound by instruction issue (the ballots of the ranking: issue slots 47 %, ALU pipe 60 %)
// and its latency, DRAM 28 %. 12.5 M 44-bit keys with weights: 1,368 us (six passes of
// count, three scan kernels, scatter) -> 629 us; without weights 511 us; 1 M with weights
// 170 -> 114 us. Tiles of 16 keys a thread and two blocks per SM measured best: 12 keys 623
// / 562 / 130 us (12.5 M with, without weights, 1 M with), 8 keys and three blocks 644 / 575 /
// 121, 16 keys and one block 694 / 580 / 109. __match_any_sync in place of the ballots:
// 737 / 657 / 127.
constexpr int OS_T = 512, OS_WARPS = OS_T / 32;
constexpr int OS_BITS = 9, OS_BINS = 1 << OS_BITS;
static_assert(OS_BINS == OS_T, "one thread per digit");
constexpr int OS_IPT_SMALL = 4, OS_IPT_LARGE = 16;
constexpr int OS_LB = 8;
constexpr uint32_t OS_POLLS = 1u << 18;
constexpr int OS_MAX_PASSES = 8;   // 64 bits
constexpr int OS_COPIES = 4;       // copies of the digit counters (by lane): fewer same-address conflicts
// a single block sorts up to this many keys in shared memory, every pass in one launch
constexpr int OS_BLOCK_T = 1024, OS_BLOCK_WARPS = OS_BLOCK_T / 32;
constexpr int OS_BLOCK_IPT_SMALL = 2, OS_BLOCK_IPT_LARGE = 8;

struct OsPlan {
  int passes;
  int shift[OS_MAX_PASSES];
  uint32_t mask[OS_MAX_PASSES];
};
inline OsPlan os_plan(int bits) {
  OsPlan p{};
  p.passes = (bits + OS_BITS - 1) / OS_BITS;
  int at = 0;
  for (int k = 0; k < p.passes; ++k) {
    const int w = (bits - at + (p.passes - k) - 1) / (p.passes - k);
    p.shift[k] = at;
    p.mask[k] = (1u << w) - 1u;
    at += w;
  }
  return p;
}

// Lanes of the warp whose digit equals this lane's (every lane takes part).
__device__ __forceinline__ unsigned os_peers(uint32_t d) {
  unsigned m = 0xFFFFFFFFu;
#pragma unroll
  for (int b = 0; b < OS_BITS; ++b) {
    const bool bit = (d >> b) & 1u;
    const unsigned bal = __ballot_sync(0xFFFFFFFFu, bit);
    m &= bit ? bal : ~bal;
  }
  return m;
}

// Rank of each of the thread's keys among its warp's keys of the same digit, in input order
// (item by item, lanes in order); wc = the warp's digit counters, zero on entry, the warp's
// digit counts on return.
template <int IPT>
__device__ __forceinline__ void os_rank(const uint64_t (&key)[IPT], int shift, uint32_t mask, uint16_t* wc,
                                        uint16_t (&rank)[IPT]) {
  const unsigned lane = threadIdx.x & 31, lt = (1u << lane) - 1u;
#pragma unroll
  for (int k = 0; k < IPT; ++k) {
    const uint32_t d = (uint32_t)(key[k] >> shift) & mask;
    const unsigned peers = os_peers(d);
    const unsigned before = wc[d];
    __syncwarp();
    if ((peers & lt) == 0) wc[d] = (uint16_t)(before + __popc(peers));
    __syncwarp();
    rank[k] = (uint16_t)(before + __popc(peers & lt));
  }
}

// Exclusive prefix over the block's threads (T threads, wsum: one word per warp).
template <int T>
__device__ __forceinline__ uint32_t os_block_prefix(uint32_t v, uint32_t* wsum) {
  const unsigned lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  uint32_t inc = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, inc, o);
    if (lane >= (unsigned)o) inc += y;
  }
  if (lane == 31) wsum[wid] = inc;
  __syncthreads();
  uint32_t off = 0;
#pragma unroll
  for (int w = 0; w < T / 32; ++w) off += w < (int)wid ? wsum[w] : 0u;
  return off + inc - v;
}

// Every pass's digit counts in one read of the keys; the last block turns them into
// exclusive offsets. Also clears the status rows of the first pass.
__global__ void __launch_bounds__(OS_T) radix_hist_kernel(const uint64_t* __restrict__ keys, uint64_t n, OsPlan plan,
                                                          uint32_t* __restrict__ hist, uint32_t* __restrict__ done,
                                                          uint4* __restrict__ status, uint64_t status_vec);

// Status word of (tile, digit): the count in the low bits, the top two bits tell what it
// counts. 32-bit words hold counts below 2^30, so sorts of 2^30 keys and more use 64-bit ones.
template <class ST>
__device__ __forceinline__ ST os_flag(int f) {
  return (ST)f << (sizeof(ST) * 8 - 2);  // 1: this tile's count; 2: all tiles up to it
}
template <class ST>
__device__ __forceinline__ ST os_value(ST w) {
  return w & (((ST)1 << (sizeof(ST) * 8 - 2)) - 1);
}

template <int IPT>
__host__ __device__ constexpr size_t os_smem() {
  return (size_t)OS_T * IPT * 8 > (size_t)OS_WARPS * OS_BINS * 2 ? (size_t)OS_T * IPT * 8
                                                                 : (size_t)OS_WARPS * OS_BINS * 2;
}

template <int IPT, bool VALS, class ST>
__global__ void __launch_bounds__(OS_T, 2) radix_onesweep_kernel(
    const uint64_t* __restrict__ keys, const uint32_t* __restrict__ vals, uint64_t n, int shift, uint32_t mask,
    const uint32_t* __restrict__ doff, uint32_t* __restrict__ ticket, ST* status, ST* __restrict__ status_next,
    uint64_t* __restrict__ keys_out, uint32_t* __restrict__ vals_out, uint32_t max_polls) {
  extern __shared__ __align__(16) uint8_t os_raw[];
  __shared__ uint32_t s_tile, s_wsum[OS_WARPS];
  __shared__ uint32_t s_off[OS_BINS];  // digit's first place in the tile, then output place - tile place
  uint16_t* wcnt = reinterpret_cast<uint16_t*>(os_raw);  // [warp][digit], until the keys are placed
  uint64_t* skeys = reinterpret_cast<uint64_t*>(os_raw);
  uint32_t* svals = reinterpret_cast<uint32_t*>(os_raw);
  const unsigned lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  constexpr uint32_t TILE = OS_T * IPT;
  if (threadIdx.x == 0) s_tile = atomicAdd(ticket, 1u);
  for (uint32_t i = threadIdx.x; i < OS_WARPS * OS_BINS / 8; i += OS_T)
    reinterpret_cast<uint4*>(wcnt)[i] = make_uint4(0, 0, 0, 0);
  __syncthreads();
  const uint32_t tile = s_tile;
  const uint64_t base = (uint64_t)tile * TILE;
  const uint64_t wbase = base + (uint64_t)wid * (32 * IPT);
  const uint32_t cnt = n - base < (uint64_t)TILE ? (uint32_t)(n - base) : TILE;
  // the key's bits are all ones past the end: such places rank behind every key of the tile
  uint64_t key[IPT];
#pragma unroll
  for (int k = 0; k < IPT; ++k) {
    const uint64_t i = wbase + (uint64_t)k * 32 + lane;
    key[k] = i < n ? __ldcs(keys + i) : ~0ULL;
  }
  uint16_t rank[IPT];
  os_rank<IPT>(key, shift, mask, wcnt + wid * OS_BINS, rank);
  __syncthreads();
  // thread d: digit d's count in the tile, and each warp's first place among them
  uint32_t total = 0;
#pragma unroll
  for (int w = 0; w < OS_WARPS; ++w) {
    const uint32_t c = wcnt[w * OS_BINS + threadIdx.x];
    wcnt[w * OS_BINS + threadIdx.x] = (uint16_t)total;
    total += c;
  }
  volatile ST* row = status + (uint64_t)tile * OS_BINS + threadIdx.x;
  *row = os_flag<ST>(tile == 0 ? 2 : 1) | (ST)total;
  status_next[(uint64_t)tile * OS_BINS + threadIdx.x] = 0;
  const uint32_t first = os_block_prefix<OS_T>(total, s_wsum);
  s_off[threadIdx.x] = first;
  __syncthreads();
#pragma unroll
  for (int k = 0; k < IPT; ++k) {
    const uint32_t d = (uint32_t)(key[k] >> shift) & mask;
    rank[k] = (uint16_t)(rank[k] + s_off[d] + wcnt[wid * OS_BINS + d]);
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < IPT; ++k) skeys[rank[k]] = key[k];
  // look-back: digit threadIdx.x's keys in the tiles before this one
  ST before = 0;
  if (tile != 0) {
    int64_t t = (int64_t)tile - 1;
    uint32_t polls = 0;
    bool open = true;
    while (open) {
      ST w[OS_LB];
#pragma unroll
      for (int b = 0; b < OS_LB; ++b)
        w[b] = t - b >= 0 ? *(const volatile ST*)(status + (uint64_t)(t - b) * OS_BINS + threadIdx.x) : (ST)0;
#pragma unroll
      for (int b = 0; b < OS_LB; ++b) {
        if (!open) continue;
        const int f = (int)(w[b] >> (sizeof(ST) * 8 - 2));
        if (f == 0) {
          // not published yet: read again from here (and, past the limit, count it here)
          if (++polls > max_polls && t >= 0) {
            const uint64_t tb = (uint64_t)t * TILE;
            for (uint32_t i = 0; i < TILE; ++i)
              before += ((uint32_t)(keys[tb + i] >> shift) & mask) == threadIdx.x ? 1 : 0;
            if (--t < 0) open = false;
          }
          break;
        }
        before += os_value<ST>(w[b]);
        if (f == 2 || --t < 0) open = false;
      }
    }
    *row = os_flag<ST>(2) | (before + (ST)total);
  }
  s_off[threadIdx.x] = doff[threadIdx.x] + (uint32_t)before - first;
  __syncthreads();
  uint32_t dst[IPT];
#pragma unroll
  for (int k = 0; k < IPT; ++k) {
    const uint32_t i = (uint32_t)k * OS_T + threadIdx.x;
    if (i < cnt) {
      const uint64_t q = skeys[i];
      dst[k] = s_off[(uint32_t)(q >> shift) & mask] + i;
      keys_out[dst[k]] = q;
    }
  }
  if constexpr (VALS) {
    uint32_t v[IPT];
#pragma unroll
    for (int k = 0; k < IPT; ++k) {
      const uint64_t i = wbase + (uint64_t)k * 32 + lane;
      v[k] = i < n ? __ldcs(vals + i) : 0u;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < IPT; ++k) svals[rank[k]] = v[k];
    __syncthreads();
#pragma unroll
    for (int k = 0; k < IPT; ++k) {
      const uint32_t i = (uint32_t)k * OS_T + threadIdx.x;
      if (i < cnt) vals_out[dst[k]] = svals[i];
    }
  }
}

// Every pass of a small sort in one block: keys (and values) stay in shared memory.
template <int IPT>
__host__ __device__ constexpr size_t os_block_smem() {
  return (size_t)OS_BLOCK_T * IPT * 12 + (size_t)OS_BLOCK_WARPS * OS_BINS * 2;
}
template <int IPT, bool VALS>
__global__ void __launch_bounds__(OS_BLOCK_T, 1) radix_block_kernel(const uint64_t* __restrict__ keys,
                                                                    const uint32_t* __restrict__ vals, uint32_t n,
                                                                    OsPlan plan, uint64_t* __restrict__ keys_out,
                                                                    uint32_t* __restrict__ vals_out) {
  extern __shared__ __align__(16) uint8_t os_raw[];
  __shared__ uint32_t s_wsum[OS_BLOCK_WARPS], s_off[OS_BINS];
  constexpr uint32_t N = OS_BLOCK_T * IPT;
  uint64_t* skeys = reinterpret_cast<uint64_t*>(os_raw);
  uint32_t* svals = reinterpret_cast<uint32_t*>(os_raw + (size_t)N * 8);
  uint16_t* wcnt = reinterpret_cast<uint16_t*>(os_raw + (size_t)N * 12);
  const unsigned lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const uint32_t wbase = wid * (32 * IPT);
  uint64_t key[IPT];
  uint32_t val[IPT];
#pragma unroll
  for (int k = 0; k < IPT; ++k) {
    const uint32_t i = wbase + (uint32_t)k * 32 + lane;
    key[k] = i < n ? keys[i] : ~0ULL;
    val[k] = (VALS && i < n) ? vals[i] : 0u;
  }
  for (int p = 0; p < plan.passes; ++p) {
    const int shift = plan.shift[p];
    const uint32_t mask = plan.mask[p];
    for (uint32_t i = threadIdx.x; i < OS_BLOCK_WARPS * OS_BINS / 8; i += OS_BLOCK_T)
      reinterpret_cast<uint4*>(wcnt)[i] = make_uint4(0, 0, 0, 0);
    __syncthreads();
    uint16_t rank[IPT];
    os_rank<IPT>(key, shift, mask, wcnt + wid * OS_BINS, rank);
    __syncthreads();
    uint32_t total = 0;
    if (threadIdx.x < OS_BINS) {
#pragma unroll 8
      for (int w = 0; w < OS_BLOCK_WARPS; ++w) {
        const uint32_t c = wcnt[w * OS_BINS + threadIdx.x];
        wcnt[w * OS_BINS + threadIdx.x] = (uint16_t)total;
        total += c;
      }
    }
    const uint32_t first = os_block_prefix<OS_BLOCK_T>(total, s_wsum);
    if (threadIdx.x < OS_BINS) s_off[threadIdx.x] = first;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < IPT; ++k) {
      const uint32_t d = (uint32_t)(key[k] >> shift) & mask;
      const uint32_t at = rank[k] + s_off[d] + wcnt[wid * OS_BINS + d];
      skeys[at] = key[k];
      if (VALS) svals[at] = val[k];
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < IPT; ++k) {
      const uint32_t i = wbase + (uint32_t)k * 32 + lane;
      key[k] = skeys[i];
      if (VALS) val[k] = svals[i];
    }
  }
#pragma unroll
  for (int k = 0; k < IPT; ++k) {
    const uint32_t i = wbase + (uint32_t)k * 32 + lane;
    if (i < n) {
      keys_out[i] = key[k];
      if (VALS) vals_out[i] = val[k];
    }
  }
}

}  // namespace cytom
