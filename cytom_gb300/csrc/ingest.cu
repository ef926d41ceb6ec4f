// ingest.cu — edge sources, streaming insert and compaction of the tile store.
//
// Replaces, for one GPU:
//   RMATContext::getEdge / rMatIterative   (src/include/edge-inserter/rmat-context.h:39-73)
//   Jobs GridGraph reader                  (src/include/core/jobs.h:53-64, 111-118)
//   MetaTileManager::insertEdge + TileManager::insertEdge
//                                          (meta-tile-manager.h:112-125, tile-manager.h:136-163)
//   TileManager::compactStorage / fillCSR  (tile-manager.h:192-291, 518-565)
//
// Compaction is a global merge: the append region is radix-sorted by the
// composite key (x, y, src_local, tgt_local), deduplicated within itself and
// against the compacted store (binary search in the tile's segment), and the
// survivors are merged into a new buffer by output-position ranking. Every
// compacted tile is then exactly the reference's sorted, deduplicated CSR.
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <vector>

#include "engine.h"
#include "radix.cuh"

namespace cytom {

// --------------------------------------------------------------------------
// Hash (Ligra 64-bit, src/include/util/util.h:188-196)
// --------------------------------------------------------------------------
__host__ __device__ __forceinline__ uint64_t hash64(uint64_t a) {
  a = (a + 0x7ed55d166bef7a1dULL) + (a << 12);
  a = (a ^ 0xc761c23c510fa2ddULL) ^ (a >> 9);
  a = (a + 0x165667b183a9c0e1ULL) + (a << 59);
  a = (a + 0xd3a2646cab3487e3ULL) ^ (a << 49);
  a = (a + 0xfd7046c5ef9ab54cULL) + (a << 3);
  a = (a ^ 0xb55a4f090dd4a67bULL) ^ (a >> 32);
  return a;
}

// --------------------------------------------------------------------------
// RMAT
// --------------------------------------------------------------------------
// util::hashDouble(i) = (double)hash(i) / (double)UINT64_MAX, and (double)UINT64_MAX
// is exactly 2^64, so `hashDouble(i) < t` <=> `(double)hash(i) < t * 2^64`. Because
// the u64 -> double rounding is monotone, that is `hash(i) < H` for the least H
// whose double value reaches t * 2^64. The kernel compares integers against H;
// the host derives H once from the double thresholds a, a+b, a+b+c.
struct RmatThr {
  unsigned long long h[3];
  int all[3];  // 1 when every hash is below the threshold
};

static void rmat_threshold(double t, unsigned long long* h, int* all) {
  const double two64 = 18446744073709551616.0;
  double A = t * two64;
  *all = 0;
  if (!(A > 0.0)) {  // also NaN
    *h = 0;
    return;
  }
  if (A > (double)UINT64_MAX) {  // (double)UINT64_MAX == 2^64
    *all = 1;
    *h = 0;
    return;
  }
  // A < 2^64 here or A == 2^64 (handled above); search H in a window around A.
  unsigned long long guess = (A >= two64)                     ? UINT64_MAX
                             : (A >= 9223372036854775808.0) ? (unsigned long long)(A)
                                                            : (unsigned long long)std::ceil(A);
  unsigned long long lo = guess > 8192 ? guess - 8192 : 0;
  unsigned long long hi = guess < UINT64_MAX - 8192 ? guess + 8192 : UINT64_MAX;
  // predicate p(h) = ((double)h >= A) is monotone; find the least h with p(h).
  if ((double)hi < A) {  // all values in range below A: every hash < A
    *all = 1;
    *h = 0;
    return;
  }
  while (lo < hi) {
    unsigned long long mid = lo + (hi - lo) / 2;
    if ((double)mid >= A) hi = mid;
    else lo = mid + 1;
  }
  *h = lo;
}

// hash64 with its shift-and-add steps as multiplications (a + (a << 12) = 4097 a, a + (a << 3)
// = 9 a): one wide multiply-add and one 32-bit one each, on the pipe that the rest of the
// hash leaves idle.
__device__ __forceinline__ uint64_t hash64_mad(uint64_t a) {
  a = a * 4097ULL + 0x7ed55d166bef7a1dULL;
  a = (a ^ 0xc761c23c510fa2ddULL) ^ (a >> 9);
  a = (a + 0x165667b183a9c0e1ULL) + (a << 59);
  a = (a + 0xd3a2646cab3487e3ULL) ^ (a << 49);
  a = a * 9ULL + 0xfd7046c5ef9ab54cULL;
  a = (a ^ 0xb55a4f090dd4a67bULL) ^ (a >> 32);
  return a;
}

// One edge per thread and step; `scale` hashes per edge: bound by integer instructions. The
// thresholds ascend (rmat_generate sees to that), so the quadrant of hash h is the number of
// thresholds at or below it: the source bit is h >= h1, the target bit the parity of the three
// comparisons (12.5 M edges of scale 22 with weights: 645 -> 448 us). ALL: some threshold lies above every hash (RmatThr::all).
template <bool ALL>
__global__ void rmat_kernel(RmatThr thr, uint32_t scale, uint64_t hseed, uint64_t first,
                            uint64_t count, uint32_t* __restrict__ src, uint32_t* __restrict__ tgt,
                            uint32_t* __restrict__ w, uint64_t wseed_h, uint32_t wmin,
                            uint64_t wspan) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  const uint64_t t0 = thr.h[0], t1 = thr.h[1], t2 = thr.h[2];
  const uint32_t m0 = ALL && thr.all[0] ? 0u : 1u, m1 = ALL && thr.all[1] ? 0u : 1u, m2 = ALL && thr.all[2] ? 0u : 1u;
  for (uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; k < count; k += stride) {
    uint64_t index = first + k;
    uint64_t r = hash64(2ULL * index * hseed);
    uint64_t st = hash64((2ULL * index + 1ULL) * hseed);
    // bit j (value 2^j) uses hash(rs + (scale-1-j)*st): the most significant bit
    // uses hash(rs), as rMatIterative walks back from the finest level.
    uint32_t es = 0, et = 0;
#pragma unroll 2
    for (uint32_t j = 0; j < scale; ++j) {
      const uint64_t h = hash64_mad(r);
      r += st;
      const uint32_t c0 = h >= t0 ? m0 : 0u, c1 = h >= t1 ? m1 : 0u, c2 = h >= t2 ? m2 : 0u;
      es = es * 2u + c1;
      et = et * 2u + (c0 ^ c1 ^ c2);
    }
    src[k] = es;
    tgt[k] = et;
    if (w) {
      uint64_t key = wseed_h ^ (((uint64_t)es << 32) | (uint64_t)et);
      w[k] = wmin + (uint32_t)(hash64(key) % wspan);
    }
  }
}

static int grid_for(Ctx* c, uint64_t work, int threads, int per_sm = 8) {
  uint64_t blocks = (work + threads - 1) / threads;
  uint64_t cap = (uint64_t)c->num_sms * per_sm;
  if (blocks > cap) blocks = cap;
  if (blocks == 0) blocks = 1;
  return (int)blocks;
}

int rmat_generate(Ctx* c, const cytom_rmat_params* p, uint64_t first, uint64_t count,
                  uint32_t* src, uint32_t* tgt, uint32_t* w) {
  if (count == 0) return CYTOM_OK;
  RmatThr thr;
  double a_ = p->a, ab_ = p->a + p->b, abc_ = p->a + p->b + p->c;
  rmat_threshold(a_, &thr.h[0], &thr.all[0]);
  rmat_threshold(ab_, &thr.h[1], &thr.all[1]);
  rmat_threshold(abc_, &thr.h[2], &thr.all[2]);
  // the walk takes the first threshold above the hash, so a later one below it never counts
  for (int k = 1; k < 3; ++k) {
    if (thr.all[k - 1]) thr.all[k] = 1;
    else if (!thr.all[k]) thr.h[k] = std::max(thr.h[k], thr.h[k - 1]);
  }
  const bool all = thr.all[0] || thr.all[1] || thr.all[2];
  uint64_t hseed = hash64(p->seed);
  uint64_t wspan = (uint64_t)p->wmax - (uint64_t)p->wmin + 1ULL;
  int slot = prof_begin(c, KC_RMAT);
  auto fn = all ? rmat_kernel<true> : rmat_kernel<false>;
  fn<<<grid_for(c, count, 256, 16), 256, 0, c->stream>>>(
      thr, p->scale, hseed, first, count, src, tgt, (p->wmax > 0) ? w : nullptr,
      hash64(p->weight_seed), p->wmin, wspan);
  c->launches++;
  prof_end(c, slot, (double)count * ((p->wmax > 0) ? 12.0 : 8.0));
  return cuda_err(c, cudaGetLastError(), "rmat_kernel");
}

// --------------------------------------------------------------------------
// GridGraph decode
// --------------------------------------------------------------------------
__global__ void gridgraph_decode_kernel(const int2* __restrict__ rec, uint64_t m, uint64_t n,
                                        uint32_t* __restrict__ src, uint32_t* __restrict__ tgt,
                                        unsigned int* bad) {
  uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  unsigned int nb = 0;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m; i += stride) {
    int2 r = rec[i];
    bool ok = r.x >= 0 && r.y >= 0 && (uint64_t)r.x < n && (uint64_t)r.y < n;
    nb += ok ? 0 : 1;
    src[i] = ok ? (uint32_t)r.x : 0u;
    tgt[i] = ok ? (uint32_t)r.y : 0u;
  }
  if (nb) atomicAdd(bad, nb);
}

int gridgraph_decode(Ctx* c, const void* dbytes, uint64_t m, uint32_t* src, uint32_t* tgt) {
  if (m == 0) return CYTOM_OK;
  cudaError_t e = cudaMemsetAsync(c->d_flag, 0, sizeof(unsigned int), c->stream);
  if (e != cudaSuccess) return cuda_err(c, e, "memset");
  int slot = prof_begin(c, KC_INSERT);
  gridgraph_decode_kernel<<<grid_for(c, m, 256), 256, 0, c->stream>>>(
      (const int2*)dbytes, m, c->n, src, tgt, c->d_flag);
  c->launches++;
  prof_end(c, slot, (double)m * 16.0);
  e = cudaMemcpyAsync(c->h_pinned, c->d_flag, sizeof(unsigned int), cudaMemcpyDeviceToHost,
                      c->stream);
  if (e != cudaSuccess) return cuda_err(c, e, "memcpy");
  e = cudaStreamSynchronize(c->stream);
  if (e != cudaSuccess) return cuda_err(c, e, "gridgraph_decode");
  unsigned int bad = *(unsigned int*)c->h_pinned;
  if (bad) return set_err(c, CYTOM_ERR_RANGE, "gridgraph record with a negative id or an id >= vertex count");
  return CYTOM_OK;
}

// --------------------------------------------------------------------------
// Insert
// --------------------------------------------------------------------------
// Composite key: [x : lT][y : lT][src_local : lvpt][tgt_local : lvpt].
__device__ __forceinline__ uint64_t make_key(uint32_t s, uint32_t t, uint32_t lvpt, uint32_t lT) {
  uint64_t m = (1ULL << lvpt) - 1ULL;
  uint64_t x = (uint64_t)s >> lvpt, y = (uint64_t)t >> lvpt;
  uint64_t tile = (x << lT) | y;
  return (tile << (2 * lvpt)) | (((uint64_t)s & m) << lvpt) | ((uint64_t)t & m);
}

// Appends one batch to the append region and counts its degrees, checking every endpoint: an
// edge with an endpoint out of range is left out and counted in *bad. The host then rejects
// the whole batch (append_undo_kernel takes its degrees back; the keys lie past the region's
// end). One pass over the batch instead of a checking pass before; the degree atomics are
// one per endpoint: aggregating a warp's equal vertices first (two __match_any_sync an edge)
// took longer than the atomics it saved. Bound by the atomics (16.8 M edges, ids without
// order: 320 -> 262 us; 20,011 edges 14.2 -> 8.7).
//
// HUBS: a block counts the first APPEND_HUBS vertices in shared memory and adds them up at its
// end. Atomics on one sector go one after another, and in graphs numbered by degree or by a
// generator the first take several per cent of the endpoints (12.5 M RMAT-22 edges 366 us
// without, 326 with one such vertex, 253 with 64 or 512, 255 with 2,048, 236 with 4,096, which
// leaves fewer blocks per SM). Where ids say nothing about degrees it costs the clearing and the
// adding up. With / without, in us:
//   vertices  edges   RMAT ids       RMAT, ids shuffled   uniform
//   2^12      2^17    12.0 / 20.8    12.1 / 11.7          9.9 / 8.3
//   2^16      2^17    9.9 / 12.3     8.5 / 8.0            8.3 / 7.0
//   2^16      2^18    12.2 / 20.8    11.2 / 10.2          9.9 / 8.3
//   2^22      2^17    8.4 / 9.4      8.0 / 7.3            8.4 / 7.1
//   2^22      2^18    11.0 / 14.4    10.7 / 9.8           9.5 / 8.7
//   2^22      2^20    24.4 / 31.3    20.7 / 20.6          17.2 / 16.2
//   2^22      2^24    298 / 378      212 / 212            198 / 195
// (2^16 edges: 8.1 / 13.7 on 2^12 vertices, 8.1 / 8.9 on 2^16, 7.8 / 8.4 on 2^20 with RMAT ids,
// 7.5 / 6.2, 7.0 / 6.1 and 6.5 / 6.1 uniform.)
constexpr uint32_t APPEND_HUBS = 2048;
constexpr uint64_t kAppendHubsMin = 1ULL << 17;  // edges: from here on the gain is well above the cost

template <bool HUBS>
__global__ void append_kernel(const uint32_t* __restrict__ src, const uint32_t* __restrict__ tgt,
                              const uint32_t* __restrict__ w, uint64_t count, uint64_t n,
                              uint64_t* __restrict__ keys, uint32_t* __restrict__ kw,
                              uint32_t* __restrict__ out_deg, uint32_t* __restrict__ in_deg,
                              uint32_t lvpt, uint32_t lT, unsigned int* __restrict__ bad) {
  __shared__ uint32_t s_out[HUBS ? APPEND_HUBS : 1], s_in[HUBS ? APPEND_HUBS : 1];
  if (HUBS) {
    for (uint32_t i = threadIdx.x; i < APPEND_HUBS; i += blockDim.x) s_out[i] = s_in[i] = 0;
    __syncthreads();
  }
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  unsigned nb = 0;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += stride) {
    const uint32_t s = src[i], t = tgt[i];
    if (s >= n || t >= n) {
      ++nb;
      continue;
    }
    keys[i] = make_key(s, t, lvpt, lT);
    if (w) kw[i] = w[i];
    if (HUBS && s < APPEND_HUBS) atomicAdd(&s_out[s], 1u);
    else atomicAdd(&out_deg[s], 1u);
    if (HUBS && t < APPEND_HUBS) atomicAdd(&s_in[t], 1u);
    else atomicAdd(&in_deg[t], 1u);
  }
  if (nb) atomicAdd(bad, nb);
  if (HUBS) {
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < APPEND_HUBS && i < n; i += blockDim.x) {
      if (s_out[i]) atomicAdd(&out_deg[i], s_out[i]);
      if (s_in[i]) atomicAdd(&in_deg[i], s_in[i]);
    }
  }
}

// Takes back the degrees of a rejected batch.
__global__ void append_undo_kernel(const uint32_t* __restrict__ src, const uint32_t* __restrict__ tgt, uint64_t count,
                                   uint64_t n, uint32_t* __restrict__ out_deg, uint32_t* __restrict__ in_deg) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += stride) {
    const uint32_t s = src[i], t = tgt[i];
    if (s >= n || t >= n) continue;
    atomicSub(&out_deg[s], 1u);
    atomicSub(&in_deg[t], 1u);
  }
}

// ---- dynamic compaction (TileManager::insertEdge, tile-manager.h:117, 150-161) ----
// Appended edges per tile (one atomic per tile and warp).
__global__ void dyn_count_kernel(const uint64_t* __restrict__ keys, uint64_t count, uint32_t lvpt,
                                 uint32_t* __restrict__ pending) {
  uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += stride) {
    const uint32_t t = (uint32_t)(keys[i] >> (2 * lvpt));
    const unsigned m = __match_any_sync(__activemask(), t);
    if ((threadIdx.x & 31u) == (unsigned)(__ffs(m) - 1)) atomicAdd(&pending[t], (unsigned)__popc(m));
  }
}
// A tile whose edges (stored + appended) reached its threshold raises the flag; the
// threshold doubles past the count, as one doubling per crossing would leave it.
__global__ void dyn_check_kernel(const unsigned long long* __restrict__ tile_ptr, const uint32_t* __restrict__ pending,
                                 uint64_t ntiles, unsigned long long* __restrict__ next, unsigned* __restrict__ flag) {
  uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; t < ntiles; t += stride) {
    const unsigned long long total = (tile_ptr[t + 1] - tile_ptr[t]) + pending[t];
    unsigned long long nx = next[t];
    if (total >= nx) {
      while (nx <= total) nx *= 2;
      next[t] = nx;
      atomicOr(flag, 1u);
    }
  }
}
__global__ void dyn_init_kernel(unsigned long long* __restrict__ next, uint64_t ntiles) {
  uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; t < ntiles; t += stride) next[t] = 4096;
}

// The counters, made before the first insert with dynamic compaction on changes anything.
static int dynamic_counters(Ctx* c) {
  if (c->dyn_pending) return CYTOM_OK;
  const uint64_t nt = c->ntiles;
  uint32_t* pending = nullptr;
  if (cy_malloc(&pending, nt * 4) != cudaSuccess || cy_malloc(&c->dyn_next, nt * 8) != cudaSuccess) {
    cudaGetLastError();
    cudaFree(pending);
    c->dyn_next = nullptr;
    return set_err(c, CYTOM_ERR_OOM, "dynamic compaction counters");
  }
  c->dyn_pending = pending;
  cudaMemsetAsync(c->dyn_pending, 0, nt * 4, c->stream);
  dyn_init_kernel<<<grid_for(c, nt, 256), 256, 0, c->stream>>>(c->dyn_next, nt);
  c->launches++;
  if (c->A) {  // edges appended before the counters existed
    dyn_count_kernel<<<grid_for(c, c->A, 256), 256, 0, c->stream>>>(c->app_keys, c->A, c->lvpt, c->dyn_pending);
    c->launches++;
  }
  return cuda_err(c, cudaGetLastError(), "dynamic compaction counters");
}

// After an insert with dynamic compaction on: counts the batch's edges per tile and
// compacts the store when some tile reached its threshold.
static int dynamic_compaction(Ctx* c, uint64_t first, uint64_t count) {
  const uint64_t nt = c->ntiles;
  dyn_count_kernel<<<grid_for(c, count, 256), 256, 0, c->stream>>>(c->app_keys + first, count, c->lvpt,
                                                                    c->dyn_pending);
  cudaMemsetAsync(c->d_flag, 0, sizeof(unsigned int), c->stream);
  dyn_check_kernel<<<grid_for(c, nt, 256), 256, 0, c->stream>>>(c->tile_ptr, c->dyn_pending, nt, c->dyn_next,
                                                                c->d_flag);
  c->launches += 2;
  cudaError_t e = cudaMemcpyAsync(c->h_pinned, c->d_flag, sizeof(unsigned int), cudaMemcpyDeviceToHost, c->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
  if (e != cudaSuccess) return cuda_err(c, e, "dynamic compaction check");
  if (!*(unsigned int*)c->h_pinned) return CYTOM_OK;
  c->dyn_compactions++;
  return compact(c);
}

int insert_device(Ctx* c, const uint32_t* src, const uint32_t* tgt, const uint32_t* w,
                  uint64_t count) {
  if (count == 0) return CYTOM_OK;
  if (c->wtype != CYTOM_UNWEIGHTED && w == nullptr)
    return set_err(c, CYTOM_ERR_INVAL, "weighted store needs a weight per edge");
  cudaError_t e = cudaMemsetAsync(c->d_flag, 0, sizeof(unsigned int), c->stream);
  if (e != cudaSuccess) return cuda_err(c, e, "memset");
  int rc = ensure_app_capacity(c, c->A + count);
  if (!rc && c->cfg.use_dynamic_compaction) rc = dynamic_counters(c);
  if (rc) return rc;
  const uint32_t* wuse = (c->wtype != CYTOM_UNWEIGHTED) ? w : nullptr;
  int slot = prof_begin(c, KC_INSERT);
  auto* append = count >= kAppendHubsMin ? append_kernel<true> : append_kernel<false>;
  append<<<grid_for(c, count, 256), 256, 0, c->stream>>>(
      src, tgt, wuse, count, c->n, c->app_keys + c->A, wuse ? c->app_w + c->A : nullptr, c->out_deg,
      c->in_deg, c->lvpt, c->lT, c->d_flag);
  c->launches++;
  prof_end(c, slot, (double)count * (wuse ? 28.0 : 24.0));
  e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_err(c, e, "append_kernel");
  // one wait: the batch's copies (host path) and the append
  e = cudaMemcpyAsync(c->h_pinned, c->d_flag, sizeof(unsigned int), cudaMemcpyDeviceToHost, c->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
  if (e != cudaSuccess) return cuda_err(c, e, "insert");
  if (*(unsigned int*)c->h_pinned) {
    append_undo_kernel<<<grid_for(c, count, 256), 256, 0, c->stream>>>(src, tgt, count, c->n, c->out_deg, c->in_deg);
    c->launches++;
    e = cudaStreamSynchronize(c->stream);  // the caller's buffers are borrowed for this call only
    if (e != cudaSuccess) return cuda_err(c, e, "insert");
    return set_err(c, CYTOM_ERR_RANGE, "edge endpoint >= vertex count; batch rejected");
  }
  // the jobs are seeded by these edges when the compaction installs them
  c->A += count;
  if (c->cfg.use_dynamic_compaction) return dynamic_compaction(c, c->A - count, count);
  return CYTOM_OK;
}

// --------------------------------------------------------------------------
// Device-wide exclusive scan (u32), three phases with recursion on block sums.
// --------------------------------------------------------------------------
constexpr int SCAN_T = 256, SCAN_IPT = 16, SCAN_TILE = SCAN_T * SCAN_IPT;

__device__ __forceinline__ uint32_t warp_incl_scan(uint32_t v) {
  const unsigned lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    uint32_t y = __shfl_up_sync(0xFFFFFFFFu, v, o);
    if (lane >= (unsigned)o) v += y;
  }
  return v;
}

// Returns the exclusive block prefix of `v`; *total receives the block sum.
__device__ __forceinline__ uint32_t block_excl_scan(uint32_t v, uint32_t* total) {
  __shared__ uint32_t wsum[SCAN_T / 32];
  __shared__ uint32_t tot_s;
  const unsigned lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  uint32_t inc = warp_incl_scan(v);
  if (lane == 31) wsum[wid] = inc;
  __syncthreads();
  if (wid == 0) {
    uint32_t s = (lane < SCAN_T / 32) ? wsum[lane] : 0u;
    uint32_t si = warp_incl_scan(s);
    if (lane < SCAN_T / 32) wsum[lane] = si - s;
    if (lane == SCAN_T / 32 - 1) tot_s = si;
  }
  __syncthreads();
  uint32_t r = wsum[wid] + inc - v;
  *total = tot_s;
  __syncthreads();
  return r;
}

__global__ void scan_reduce_kernel(const uint32_t* __restrict__ in, uint64_t n,
                                   uint32_t* __restrict__ sums) {
  uint64_t base = (uint64_t)blockIdx.x * SCAN_TILE + (uint64_t)threadIdx.x * SCAN_IPT;
  uint32_t s = 0;
#pragma unroll
  for (int k = 0; k < SCAN_IPT; ++k) {
    uint64_t i = base + k;
    s += (i < n) ? in[i] : 0u;
  }
  uint32_t t;
  block_excl_scan(s, &t);
  if (threadIdx.x == 0) sums[blockIdx.x] = t;
}

__global__ void scan_down_kernel(const uint32_t* __restrict__ in, uint32_t* __restrict__ out,
                                 uint64_t n, const uint32_t* __restrict__ offs,
                                 uint32_t* total_out) {
  uint64_t base = (uint64_t)blockIdx.x * SCAN_TILE + (uint64_t)threadIdx.x * SCAN_IPT;
  uint32_t v[SCAN_IPT];
  uint32_t s = 0;
#pragma unroll
  for (int k = 0; k < SCAN_IPT; ++k) {
    uint64_t i = base + k;
    v[k] = (i < n) ? in[i] : 0u;
    s += v[k];
  }
  uint32_t t;
  const uint32_t boff = offs ? offs[blockIdx.x] : 0u;
  uint32_t p = block_excl_scan(s, &t) + boff;
#pragma unroll
  for (int k = 0; k < SCAN_IPT; ++k) {
    uint64_t i = base + k;
    if (i < n) out[i] = p;
    p += v[k];
  }
  if (total_out && blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) *total_out = boff + t;
}

// Words of scratch a scan of n values needs for its per-tile sums and their offsets,
// every recursion level together.
static uint64_t scan_scratch_words(uint64_t n) {
  const uint64_t nb = (n + SCAN_TILE - 1) / SCAN_TILE;
  return nb <= 1 ? 0 : 2 * nb + scan_scratch_words(nb);
}

// The scan on scratch the caller provides (scan_scratch_words(n) words): launches only.
static int scan_into(Ctx* c, const uint32_t* in, uint32_t* out, uint64_t n, uint32_t* total_dev,
                     uint32_t* scratch) {
  if (n == 0) return CYTOM_OK;
  const uint64_t nb = (n + SCAN_TILE - 1) / SCAN_TILE;
  if (nb == 1) {
    scan_down_kernel<<<1, SCAN_T, 0, c->stream>>>(in, out, n, nullptr, total_dev);
    c->launches++;
    return cuda_err(c, cudaGetLastError(), "scan_down");
  }
  uint32_t* sums = scratch;
  uint32_t* soffs = scratch + nb;
  scan_reduce_kernel<<<(unsigned)nb, SCAN_T, 0, c->stream>>>(in, n, sums);
  c->launches++;
  int rc = scan_into(c, sums, soffs, nb, nullptr, scratch + 2 * nb);
  if (rc) return rc;
  scan_down_kernel<<<(unsigned)nb, SCAN_T, 0, c->stream>>>(in, out, n, soffs, total_dev);
  c->launches++;
  return cuda_err(c, cudaGetLastError(), "scan");
}

int exclusive_scan_u32(Ctx* c, const uint32_t* in, uint32_t* out, uint64_t n, uint32_t* total_dev) {
  const uint64_t words = scan_scratch_words(n);
  if (words == 0) return scan_into(c, in, out, n, total_dev, nullptr);
  uint32_t* scratch = nullptr;
  if (cy_malloc_async((void**)&scratch, words * 4, c->stream) != cudaSuccess)
    return set_err(c, CYTOM_ERR_OOM, "scan temp");
  const int rc = scan_into(c, in, out, n, total_dev, scratch);
  cudaFreeAsync(scratch, c->stream);
  return rc;
}

// --------------------------------------------------------------------------
// LSD radix sort of (u64 key, u32 value) pairs, stable (radix.cuh).
// --------------------------------------------------------------------------
__global__ void __launch_bounds__(OS_T) radix_hist_kernel(const uint64_t* __restrict__ keys, uint64_t n, OsPlan plan,
                                                          uint32_t* __restrict__ hist, uint32_t* __restrict__ done,
                                                          uint4* __restrict__ status, uint64_t status_vec) {
  extern __shared__ uint32_t s_hist[];  // [pass][digit][copy]
  __shared__ uint32_t s_wsum[OS_WARPS];
  __shared__ bool s_last;
  const int words = plan.passes * OS_BINS * OS_COPIES;
  for (int i = threadIdx.x; i < words; i += OS_T) s_hist[i] = 0;
  const uint64_t gid = (uint64_t)blockIdx.x * OS_T + threadIdx.x, stride = (uint64_t)gridDim.x * OS_T;
  for (uint64_t i = gid; i < status_vec; i += stride) status[i] = make_uint4(0, 0, 0, 0);
  __syncthreads();
  const unsigned copy = threadIdx.x & (OS_COPIES - 1);
  constexpr int U = 4;  // keys in flight per thread
  for (uint64_t b = gid; b < n; b += U * stride) {
    uint64_t k[U];
#pragma unroll
    for (int u = 0; u < U; ++u) k[u] = b + u * stride < n ? keys[b + u * stride] : 0ULL;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (b + u * stride >= n) continue;
#pragma unroll
      for (int p = 0; p < OS_MAX_PASSES; ++p)
        if (p < plan.passes)
          atomicAdd(&s_hist[((uint32_t)p * OS_BINS + ((uint32_t)(k[u] >> plan.shift[p]) & plan.mask[p])) * OS_COPIES + copy],
                  1u);
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < plan.passes * OS_BINS; i += OS_T) {
    uint32_t v = 0;
#pragma unroll
    for (int k = 0; k < OS_COPIES; ++k) v += s_hist[i * OS_COPIES + k];
    if (v) atomicAdd(hist + i, v);
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(done, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  for (int p = 0; p < plan.passes; ++p) {
    const uint32_t v = __ldcg(hist + p * OS_BINS + threadIdx.x);
    hist[p * OS_BINS + threadIdx.x] = os_block_prefix<OS_T>(v, s_wsum);
    __syncthreads();
  }
}

// Sorts of up to 8,192 keys run in one block (one launch); up to 2^19 keys in tiles of
// 2,048, which spread them over the SMs (60,000 keys: 55 us, in 4,096-key tiles 64); above in
// tiles of 8,192, whose runs of a digit average 16 keys (128 bytes) and whose status rows are
// few (1 M keys: 114 us, in tiles of 2,048 141 us).
constexpr uint64_t kOsSmallMax = 1ULL << 19;

template <int IPT, bool VALS, class ST>
static void onesweep_launch(Ctx* c, unsigned tiles, const uint64_t* kin, const uint32_t* vin, uint64_t n, int shift,
                            uint32_t mask, const uint32_t* doff, uint32_t* ticket, void* st, void* st_next,
                            uint64_t* kout, uint32_t* vout) {
  const uint32_t polls = c->inj_idle_limit ? c->inj_idle_limit : OS_POLLS;
  auto fn = radix_onesweep_kernel<IPT, VALS, ST>;
  if (os_smem<IPT>() > 40 * 1024)  // with the static part past the 48 KB default
    cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)os_smem<IPT>());
  fn<<<tiles, OS_T, os_smem<IPT>(), c->stream>>>(kin, vin, n, shift, mask, doff, ticket, (ST*)st, (ST*)st_next, kout,
                                             vout, polls);
}

template <int IPT, bool VALS>
static void block_sort_launch(Ctx* c, const uint64_t* keys, const uint32_t* vals, uint64_t n, const OsPlan& plan,
                              uint64_t* kout, uint32_t* vout) {
  auto fn = radix_block_kernel<IPT, VALS>;
  cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)os_block_smem<IPT>());
  fn<<<1, OS_BLOCK_T, os_block_smem<IPT>(), c->stream>>>(keys, vals, (uint32_t)n, plan, kout, vout);
}

int radix_sort_pairs(Ctx* c, uint64_t* keys, uint64_t* keys_alt, uint32_t* vals, uint32_t* vals_alt,
                     uint64_t n, int bits, bool* result_in_alt) {
  *result_in_alt = false;
  if (n <= 1 || bits <= 0) return CYTOM_OK;
  const OsPlan plan = os_plan(bits);
  const double bytes = (double)n * (vals ? 12.0 : 8.0);
  if (n <= (uint64_t)OS_BLOCK_T * OS_BLOCK_IPT_LARGE) {
    int slot = prof_begin(c, KC_SORT);
    if (n <= (uint64_t)OS_BLOCK_T * OS_BLOCK_IPT_SMALL) {
      if (vals) block_sort_launch<OS_BLOCK_IPT_SMALL, true>(c, keys, vals, n, plan, keys_alt, vals_alt);
      else block_sort_launch<OS_BLOCK_IPT_SMALL, false>(c, keys, vals, n, plan, keys_alt, vals_alt);
    } else {
      if (vals) block_sort_launch<OS_BLOCK_IPT_LARGE, true>(c, keys, vals, n, plan, keys_alt, vals_alt);
      else block_sort_launch<OS_BLOCK_IPT_LARGE, false>(c, keys, vals, n, plan, keys_alt, vals_alt);
    }
    c->launches++;
    prof_end(c, slot, bytes * 2.0);
    *result_in_alt = true;
    return cuda_err(c, cudaGetLastError(), "radix");
  }
  const bool small = n <= kOsSmallMax, wide = n >= (1ULL << 30);
  const uint64_t tile = (uint64_t)OS_T * (small ? OS_IPT_SMALL : OS_IPT_LARGE);
  const uint64_t tiles = (n + tile - 1) / tile;
  // digit counts and tickets (cleared), then two sets of status rows: a pass clears the rows
  // of the next one
  const size_t head = ((size_t)plan.passes * OS_BINS + 16 + 3) / 4 * 16;
  const size_t rows = (size_t)tiles * OS_BINS * (wide ? 8 : 4);
  char* tmp = nullptr;
  if (cy_malloc_async((void**)&tmp, head + 2 * rows, c->stream) != cudaSuccess)
    return set_err(c, CYTOM_ERR_OOM, "radix histogram");
  uint32_t* hist = (uint32_t*)tmp;
  uint32_t* tickets = hist + (size_t)plan.passes * OS_BINS;  // one per pass, then the counting kernel's block count
  char* st[2] = {tmp + head, tmp + head + rows};
  int slot = prof_begin(c, KC_SORT);
  cudaError_t e = cudaMemsetAsync(tmp, 0, head, c->stream);
  const size_t hsm = (size_t)plan.passes * OS_BINS * OS_COPIES * 4;
  if (e == cudaSuccess && hsm > 40 * 1024)
    e = cudaFuncSetAttribute(radix_hist_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)hsm);
  if (e == cudaSuccess) {
    radix_hist_kernel<<<grid_for(c, (n + 7) / 8, OS_T, 3), OS_T, hsm, c->stream>>>(
        keys, n, plan, hist, tickets + OS_MAX_PASSES, (uint4*)st[0], rows / 16);
    c->launches++;
    e = cudaGetLastError();
  }
  prof_end(c, slot, bytes);
  uint64_t *kin = keys, *kout = keys_alt;
  uint32_t *vin = vals, *vout = vals_alt;
  for (int p = 0; p < plan.passes && e == cudaSuccess; ++p) {
    slot = prof_begin(c, KC_SORT);
    const uint32_t* doff = hist + (size_t)p * OS_BINS;
    void *sa = st[p & 1], *sb = st[(p & 1) ^ 1];
#define CYTOM_OS(IPT, V, ST) \
  onesweep_launch<IPT, V, ST>(c, (unsigned)tiles, kin, vin, n, plan.shift[p], plan.mask[p], doff, tickets + p, sa, sb, kout, vout)
    if (small) {
      if (vals) CYTOM_OS(OS_IPT_SMALL, true, uint32_t);
      else CYTOM_OS(OS_IPT_SMALL, false, uint32_t);
    } else if (!wide) {
      if (vals) CYTOM_OS(OS_IPT_LARGE, true, uint32_t);
      else CYTOM_OS(OS_IPT_LARGE, false, uint32_t);
    } else {
      if (vals) CYTOM_OS(OS_IPT_LARGE, true, unsigned long long);
      else CYTOM_OS(OS_IPT_LARGE, false, unsigned long long);
    }
#undef CYTOM_OS
    c->launches++;
    prof_end(c, slot, bytes * 2.0);
    e = cudaGetLastError();
    std::swap(kin, kout);
    std::swap(vin, vout);
  }
  cudaFreeAsync(tmp, c->stream);
  *result_in_alt = (plan.passes & 1) != 0;
  return cuda_err(c, e, "radix");
}

// --------------------------------------------------------------------------
// Compaction
// --------------------------------------------------------------------------
// For each sorted appended key: first of its run? present in the compacted tile?
// keep[i] = 1 for a new distinct edge; lb[i] = its insertion index in the old store;
// wsel[i] = the least weight of its run. A weight that undercuts the stored copy of
// an existing edge lowers that copy in place. Bound by the search's instructions: offsets in
// the tile are 32-bit, and a snapshot with a source directory is searched from there (12.5 M
// keys against 12.5 to 37.5 M stored edges 253 us, 232 by the offsets, 154 by both).
constexpr unsigned long long kNoFix = ~0ULL, kFixFlag = 1ULL << 62;

__global__ void dedupe_lookup_kernel(const uint64_t* __restrict__ K, const uint32_t* __restrict__ W,
                                     uint64_t A, const uint32_t* __restrict__ edges,
                                     const uint32_t* __restrict__ wts,
                                     const unsigned long long* __restrict__ tile_ptr,
                                     const uint32_t* __restrict__ dir, uint32_t nbw,
                                     uint32_t lvpt, uint32_t* __restrict__ keep,
                                     unsigned long long* __restrict__ lb,
                                     uint32_t* __restrict__ wsel) {
  uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  const uint64_t m = (1ULL << lvpt) - 1ULL;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < A; i += stride) {
    uint64_t key = K[i];
    if (i > 0 && K[i - 1] == key) {
      keep[i] = 0;
      lb[i] = kNoFix;
      continue;
    }
    uint32_t wmin = 0;
    if (W) {
      wmin = W[i];
      for (uint64_t j = i + 1; j < A && K[j] == key; ++j) wmin = min(wmin, W[j]);
    }
    uint64_t tile = key >> (2 * lvpt);
    uint32_t local = (uint32_t)((((key >> lvpt) & m) << 16) | (key & m));
    uint64_t lo = tile_ptr[tile], hi = tile_ptr[tile + 1];
    // fillCSR starts its duplicate filter at (UINT16_MAX, UINT16_MAX)
    // (tile-manager.h:519-541): when that edge is the first in its tile's sorted
    // list -- an otherwise empty tile -- the reference drops it.
    if (local == 0xFFFFFFFFu && lo == hi && (i == 0 || (K[i - 1] >> (2 * lvpt)) != tile)) {
      keep[i] = 0;
      lb[i] = kNoFix;
      continue;
    }
    const uint32_t* te = edges + lo;
    const bool full = hi - lo > 0xFFFFFFFFULL;  // all 2^32 pairs of the tile
    uint32_t at = 0, left = full ? 0xFFFFFFFFu : (uint32_t)(hi - lo);
    if (dir && !full) {  // the edges of the source's block alone
      const uint32_t* d = dir + tile * (nbw + 1) + (local >> 21);
      at = d[0];
      left = d[1] - at;
    }
    const uint32_t end = at + left;
    while (left) {
      const uint32_t half = left >> 1;
      if (te[at + half] < local) {
        at += half + 1;
        left -= half + 1;
      } else {
        left = half;
      }
    }
    const uint64_t pos = lo + at;
    const bool found = (at < end || full) && te[at] == local;
    if (found) {
      // a lower weight for a stored edge is applied to the merged copy (fixup_weights_kernel):
      // the store itself may still be read by runs of the previous batch
      keep[i] = 0;
      lb[i] = (W && wmin < wts[pos]) ? (kFixFlag | pos) : kNoFix;
      wsel[i] = wmin;
    } else {
      keep[i] = 1;
      lb[i] = pos;
      wsel[i] = wmin;
    }
  }
}

// Also sets the column-mask bit (StoreDesc::cmask) of every appended key's source and
// tile column, once per run of keys with the same (tile, source); duplicates and dropped
// corner edges only add bits that are allowed to be spare.
__global__ void pack_kept_kernel(const uint64_t* __restrict__ K, uint64_t A,
                                 const uint32_t* __restrict__ keep, const uint32_t* __restrict__ P,
                                 const unsigned long long* __restrict__ lb,
                                 const uint32_t* __restrict__ wsel, uint32_t lvpt,
                                 unsigned long long* __restrict__ q, uint32_t* __restrict__ nloc,
                                 uint32_t* __restrict__ nw, uint32_t* __restrict__ ntile,
                                 unsigned long long* __restrict__ cmask, uint32_t lT, uint32_t cshift) {
  uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  const uint64_t m = (1ULL << lvpt) - 1ULL;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < A; i += stride) {
    if (cmask) {
      const uint64_t ts = K[i] >> lvpt;  // (tile, local source)
      if (i == 0 || (K[i - 1] >> lvpt) != ts) {
        const uint64_t tile = ts >> lvpt;
        const uint64_t u = ((tile >> lT) << lvpt) | (ts & m);
        atomicOr(cmask + u, 1ULL << ((tile & ((1ULL << lT) - 1ULL)) >> cshift));
      }
    }
    if (!keep[i]) continue;
    uint64_t key = K[i];
    uint32_t p = P[i];
    q[p] = lb[i] + p;
    nloc[p] = (uint32_t)((((key >> lvpt) & m) << 16) | (key & m));
    if (nw) nw[p] = wsel[i];
    ntile[p] = (uint32_t)(key >> (2 * lvpt));
  }
}

// Weight of a stored edge lowered by the batch, on the merged copy: the old edge at pos
// moved by the kept new edges inserted at or before pos (q[p] - p <= pos).
__global__ void fixup_weights_kernel(const unsigned long long* __restrict__ lb, const uint32_t* __restrict__ wsel,
                                     uint64_t A, const unsigned long long* __restrict__ q,
                                     const uint32_t* __restrict__ Kdev, uint32_t* __restrict__ ow) {
  const uint64_t K = *Kdev;
  uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < A; i += stride) {
    const unsigned long long v = lb[i];
    if (v == kNoFix || !(v & kFixFlag)) continue;
    const uint64_t pos = v & ~kFixFlag;
    uint64_t lo = 0, hi = K;
    while (lo < hi) {
      const uint64_t mid = (lo + hi) >> 1;
      if (q[mid] - mid <= pos) lo = mid + 1;
      else hi = mid;
    }
    atomicMin(ow + pos + lo, wsel[i]);
  }
}

__device__ __forceinline__ uint64_t lower_bound_tile(const uint32_t* a, uint64_t n, uint32_t v) {
  uint64_t lo = 0, hi = n;
  while (lo < hi) {
    uint64_t mid = lo + ((hi - lo) >> 1);
    if (a[mid] < v) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

__global__ void new_tile_ptr_kernel(const unsigned long long* __restrict__ tile_ptr,
                                    uint64_t ntiles, const uint32_t* __restrict__ ntile,
                                    const uint32_t* __restrict__ Kdev,
                                    unsigned long long* __restrict__ out) {
  uint64_t K = *Kdev;
  uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; t <= ntiles; t += stride) {
    uint64_t add = (t == ntiles) ? K : lower_bound_tile(ntile, K, (uint32_t)t);
    out[t] = tile_ptr[t] + add;
  }
}

// Output position o of the merged store holds kept batch element b when q[b] == o,
// otherwise old store element o - (number of q below o). One warp produces 32
// consecutive outputs per step, 1024 per span. merge_spans_kernel gives every span its
// first new element (sb) and the tile of its first output (ts) by binary searches that
// all run at once. A warp marks its span's new elements in a 1024-bit map, one word per
// step: lane k holds step k's word and, by a warp scan, the new elements before it, so the
// sources of every step are known without further memory round trips and the loads of MG
// steps issue together, however many elements are new. Stores are coalesced 128-byte warp
// writes. (Spans with more than 64 new elements used to load their candidates step by step:
// 12.5 M new edges into 37.5 M, look-up included, 902 -> 703 us; 1 M into 42 M 254 -> 244.)
//
// The store is streamed with evict-first loads and stores, leaving L2 to the jobs that
// run on the installed snapshot meanwhile (the pipelined stream).
// The same pass writes the chunk table of the new store and, when the context keeps a
// source directory, its per-edge entries (the work of dir_edges_kernel): each output
// knows its tile (searched from the span's first tile on) and the edge before it. A step
// inside one tile keeps the tile in uniform registers. Where sources lie thinly an edge
// starts up to vpt / 32 directory entries: a warp writes long runs together, and tiles of few
// edges are left to dir_tiles_kernel, or a handful of warps at the corners of the graph hold
// up the whole merge (SMs active 22 % of its time at 13 M edges of an RMAT-22 stream).
// The instructions of a step bound it (104 before, 38 without and 60 with a directory), then
// DRAM: the 64 merges of that stream 14.2 -> 9.3 ms, four merges of 12.5 M new edges
// 853 -> 597 us; without a directory 37.5 M outputs take 115 us (5.2 TB/s).
constexpr int MERGE_STEPS = 32;  // 1024 outputs per warp span
constexpr uint64_t MERGE_SPAN = 32ULL * MERGE_STEPS;
constexpr int MG = 8;            // steps whose loads are issued together
constexpr int MG_MINB = 4;       // 5 blocks per SM: 9.9 ms for the stream's merges, 6: 13.3

__global__ void merge_spans_kernel(const unsigned long long* __restrict__ q, const uint32_t* __restrict__ Kdev,
                                   uint64_t E, const unsigned long long* __restrict__ tp, uint64_t ntiles,
                                   uint64_t nsp, uint32_t* __restrict__ sb, uint32_t* __restrict__ ts,
                                   uint32_t* __restrict__ chunk_tile) {
  const uint64_t K = *Kdev;
  const uint64_t total = E + K;
  uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  const uint64_t gid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (gid == 0) chunk_tile[(total + kChunk - 1) / kChunk] = (uint32_t)(ntiles - 1);
  for (uint64_t sp = gid; sp <= nsp; sp += stride) {
    const uint64_t target = sp * MERGE_SPAN;
    uint64_t lo = 0, hi = K;
    while (lo < hi) {
      uint64_t mid = lo + ((hi - lo) >> 1);
      if (q[mid] < target) lo = mid + 1;
      else hi = mid;
    }
    sb[sp] = (uint32_t)lo;
    // the last tile t with tp[t] <= target
    lo = 0;
    hi = ntiles - 1;
    while (lo < hi) {
      const uint64_t mid = (lo + hi + 1) >> 1;
      if (tp[mid] <= target) lo = mid;
      else hi = mid - 1;
    }
    ts[sp] = (uint32_t)lo;
  }
}

// Directory entries that start at one edge per lane: blocks b0..b1 (none if b0 > b1) of the
// directory slice at `dt` hold `off`. Called by whole warps: a lane writes a short run by
// itself, a long one is written by the warp together.
constexpr int DIR_RUN = 32;
// Tiles of fewer edges are written by dir_tiles_kernel, a warp each, in place of the kernels
// that go over the edges.
constexpr uint32_t DIR_SMALL = 256;  // 1: the stream's merges 11.6 ms, not 9.3; 1024: its dir_tiles 1.8, not 0.8

__device__ __forceinline__ void dir_runs(uint32_t* __restrict__ dir, uint64_t dt, int b0, int b1, uint32_t off) {
  unsigned lng = __ballot_sync(0xFFFFFFFFu, b1 - b0 >= DIR_RUN);
  if (b1 - b0 < DIR_RUN)
    for (int bb = b0; bb <= b1; ++bb) dir[dt + bb] = off;
  while (lng) {
    const int j = __ffs(lng) - 1;
    lng &= lng - 1;
    const uint64_t d = __shfl_sync(0xFFFFFFFFu, dt, j);
    const int e = __shfl_sync(0xFFFFFFFFu, b1, j);
    const uint32_t v = __shfl_sync(0xFFFFFFFFu, off, j);
    for (int bb = __shfl_sync(0xFFFFFFFFu, b0, j) + (int)(threadIdx.x & 31); bb <= e; bb += 32) dir[d + bb] = v;
  }
}

// Per output (offsets relative to the span start): its tile, found forward from the
// warp's tile state (tile t; toff turns a span offset into an offset within the tile;
// tend = the span offset where the tile ends; tlast = the tile of the next span's first
// output), the chunk-table entry at every 128th output, and the directory entries of the
// 32-source blocks that start at this edge. The tile state of lane 31 carries over to the
// next step.
__device__ __forceinline__ void merge_index_step(uint32_t o, uint32_t nout, uint32_t ev, uint32_t pv, uint32_t& t,
                                                 uint32_t& toff, uint32_t& tend, uint32_t tlast, uint64_t wbase,
                                                 const unsigned long long* __restrict__ tp,
                                                 uint32_t* __restrict__ ctb, uint32_t* __restrict__ dir,
                                                 uint32_t nbw) {
  uint32_t lt = t, loff = toff, lend = tend;
  int b0 = 0, b1 = -1;
  uint32_t off = 0;
  if (o < nout) {
    if (o >= lend) {  // the last tile of (lt, tlast] that starts at or before this output
      uint32_t lo = lt + 1, hi = tlast;
      while (lo < hi) {
        const uint32_t mid = (lo + hi + 1) >> 1;
        if (tp[mid] <= wbase + o) lo = mid;
        else hi = mid - 1;
      }
      lt = lo;
      loff = (uint32_t)(wbase - tp[lt]);
      const unsigned long long nx = tp[lt + 1] - wbase;
      lend = nx > 0xFFFFFFFFULL ? 0xFFFFFFFFu : (uint32_t)nx;
    }
    if ((o & (kChunk - 1)) == 0) ctb[o / kChunk] = lt;
    if (dir && (lend == 0xFFFFFFFFu || lend + loff >= DIR_SMALL)) {
      off = o + loff;
      b1 = (int)(ev >> 21);
      b0 = off == 0 ? 0 : (int)(pv >> 21) + 1;
    }
  }
  if (dir) dir_runs(dir, (uint64_t)lt * (nbw + 1), b0, b1, off);
  t = __shfl_sync(0xFFFFFFFFu, lt, 31);
  toff = __shfl_sync(0xFFFFFFFFu, loff, 31);
  tend = __shfl_sync(0xFFFFFFFFu, lend, 31);
}

template <bool W, bool DIR>
__global__ void __launch_bounds__(256, MG_MINB) merge_gather_kernel(
    const uint32_t* __restrict__ edges, const uint32_t* __restrict__ wts, uint64_t E,
    const unsigned long long* __restrict__ q, const uint32_t* __restrict__ nloc, const uint32_t* __restrict__ nw,
    const uint32_t* __restrict__ Kdev, const uint32_t* __restrict__ sb, const uint32_t* __restrict__ ts, uint64_t nsp,
    const unsigned long long* __restrict__ tp, uint32_t* __restrict__ chunk_tile, uint32_t* __restrict__ dir,
    uint32_t nbw, uint32_t* __restrict__ oe, uint32_t* __restrict__ ow) {
  __shared__ uint2 s_map[256 / 32][MERGE_STEPS];  // per step: map word, new elements before it
  const uint64_t K = *Kdev;
  const uint64_t total = E + K;
  const unsigned lane = threadIdx.x & 31;
  const uint64_t warp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  const unsigned lt = (1u << lane) - 1u;
  uint2* bm = s_map[threadIdx.x >> 5];
  for (uint64_t sp = warp; sp < nsp; sp += nwarps) {
    const uint64_t wbase = sp * MERGE_SPAN;
    if (wbase >= total) break;
    const uint32_t nout = (uint32_t)(total - wbase < MERGE_SPAN ? total - wbase : MERGE_SPAN);
    const uint64_t b0 = sb[sp];
    const uint32_t cnt = sb[sp + 1] - (uint32_t)b0;
    // span-relative views: output x preceded by y new elements of the span comes from
    // eb[x - y] (old) or nb[y] (new)
    const uint32_t* eb = edges + (wbase - b0);
    const uint32_t* wb = W ? wts + (wbase - b0) : nullptr;
    const uint32_t* nb = nloc + b0;
    const uint32_t* nwb = W ? nw + b0 : nullptr;
    uint32_t* oeb = oe + wbase;
    uint32_t* owb = W ? ow + wbase : nullptr;
    uint32_t* ctb = chunk_tile + wbase / kChunk;
    uint32_t t = ts[sp];
    const uint32_t tlast = ts[sp + 1];
    uint32_t toff = (uint32_t)(wbase - tp[t]);
    uint32_t tend;
    {
      const unsigned long long nx = tp[t + 1] - wbase;
      tend = nx > 0xFFFFFFFFULL ? 0xFFFFFFFFu : (uint32_t)nx;
    }
    // the edge before the span (the first output's predecessor)
    uint32_t plast = 0;
    if (DIR && lane == 0 && wbase > 0) {
      if (b0 > 0 && q[b0 - 1] == wbase - 1) plast = nloc[b0 - 1];
      else plast = edges[wbase - 1 - b0];
    }
    bm[lane].x = 0;
    __syncwarp();
#pragma unroll 4
    for (uint32_t i = lane; i < cnt; i += 32) {
      const uint32_t o = (uint32_t)(q[b0 + i] - wbase);
      atomicOr(&bm[o >> 5].x, 1u << (o & 31));
    }
    __syncwarp();
    const uint32_t word = bm[lane].x;
    uint32_t before = __popc(word);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t x = __shfl_up_sync(0xFFFFFFFFu, before, o);
      if (lane >= (unsigned)o) before += x;
    }
    bm[lane].y = before - __popc(word);
    __syncwarp();
    for (int g = 0; g < MERGE_STEPS; g += MG) {
      if ((uint32_t)g * 32 >= nout) break;
      uint32_t ev[MG], wv[MG];
#pragma unroll
      for (int k = 0; k < MG; ++k) {
        const uint32_t o = (uint32_t)(g + k) * 32 + lane;
        const uint2 m = bm[g + k];
        const uint32_t y = m.y + __popc(m.x & lt);
        const bool fresh = (m.x >> lane) & 1u;
        const uint32_t i = fresh ? y : o - y;
        ev[k] = 0;
        wv[k] = 0;
        if (o < nout) {
          ev[k] = __ldcs((fresh ? nb : eb) + i);
          if (W) wv[k] = __ldcs((fresh ? nwb : wb) + i);
        }
      }
#pragma unroll
      for (int k = 0; k < MG; ++k) {
        const uint32_t o = (uint32_t)(g + k) * 32 + lane;
        if (o < nout) {
          __stcs(oeb + o, ev[k]);
          if (W) __stcs(owb + o, wv[k]);
        }
        // the predecessor: lane 31's edge comes round to lane 0 for the next step
        const uint32_t rot = DIR ? __shfl_sync(0xFFFFFFFFu, ev[k], (lane + 31) & 31) : 0u;
        const uint32_t pv = lane ? rot : plast;
        plast = rot;
        if ((uint32_t)(g + k) * 32 + 31 < min(tend, nout)) {  // the whole step inside one tile
          if ((g + k) % (kChunk / 32) == 0 && lane == 0) ctb[(g + k) / (kChunk / 32)] = t;
          if (DIR && (tend == 0xFFFFFFFFu || tend + toff >= DIR_SMALL)) {
            const uint32_t off = o + toff;
            const int b1 = (int)(ev[k] >> 21);
            const int bs = off == 0 ? 0 : (int)(pv >> 21) + 1;
            uint32_t* dt = dir + (uint64_t)t * (nbw + 1);
            if (bs <= b1) dt[bs] = off;
            if (__any_sync(0xFFFFFFFFu, bs < b1)) dir_runs(dt, 0, bs + 1, b1, off);
          }
        } else {
          merge_index_step(o, nout, ev[k], pv, t, toff, tend, tlast, wbase, tp, ctb, DIR ? dir : nullptr, nbw);
        }
      }
    }
    __syncwarp();  // the map is cleared for the next span
  }
}

__global__ void chunk_tile_kernel(const unsigned long long* __restrict__ tile_ptr, uint64_t ntiles,
                                  uint64_t nchunks, uint32_t* __restrict__ chunk_tile) {
  uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t cix = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; cix <= nchunks; cix += stride) {
    if (cix == nchunks) {
      chunk_tile[cix] = (uint32_t)(ntiles - 1);
      continue;
    }
    unsigned long long e = (unsigned long long)cix * kChunk;
    // last tile t with tile_ptr[t] <= e
    uint64_t lo = 0, hi = ntiles;  // search in tile_ptr[0..ntiles]
    while (lo < hi) {
      uint64_t mid = lo + ((hi - lo + 1) >> 1);
      if (tile_ptr[mid] <= e) lo = mid;
      else hi = mid - 1;
    }
    if (lo >= ntiles) lo = ntiles - 1;
    chunk_tile[cix] = (uint32_t)lo;
  }
}

static int grow_store(Ctx* c, uint64_t need) {
  if (need <= c->cap) return CYTOM_OK;
  join_runs(c);  // the old buffers are freed below
  uint64_t ncap = std::max<uint64_t>(need + need / 2, 1 << 16);
  ncap = (ncap + kChunk - 1) / kChunk * kChunk + kChunk;
  // the chunk tables belong to the capacity: everything is there before anything is replaced
  const uint64_t nch = ncap / kChunk + 2;
  const bool chunks = nch > c->chunk_cap;
  uint32_t *ne = nullptr, *nea = nullptr, *nw = nullptr, *nwa = nullptr, *ct = nullptr, *cta = nullptr;
  cudaError_t e = cy_malloc(&ne, ncap * 4);
  if (e == cudaSuccess) e = cy_malloc(&nea, ncap * 4);
  if (e == cudaSuccess && c->wtype) e = cy_malloc(&nw, ncap * 4);
  if (e == cudaSuccess && c->wtype) e = cy_malloc(&nwa, ncap * 4);
  if (e == cudaSuccess && chunks) e = cy_malloc(&ct, nch * 4);
  if (e == cudaSuccess && chunks) e = cy_malloc(&cta, nch * 4);
  if (e != cudaSuccess) {
    cudaGetLastError();
    cudaFree(ne);
    cudaFree(nea);
    cudaFree(nw);
    cudaFree(nwa);
    cudaFree(ct);
    return set_err(c, CYTOM_ERR_OOM, "tile store growth");
  }
  if (c->E) {
    cudaMemcpyAsync(ne, c->edges, c->E * 4, cudaMemcpyDeviceToDevice, c->stream);
    if (c->wtype) cudaMemcpyAsync(nw, c->wts, c->E * 4, cudaMemcpyDeviceToDevice, c->stream);
  }
  if (chunks) cudaMemcpyAsync(ct, c->chunk_tile, c->chunk_cap * 4, cudaMemcpyDeviceToDevice, c->stream);
  cudaStreamSynchronize(c->stream);
  cudaFree(c->edges);
  cudaFree(c->edges_alt);
  cudaFree(c->wts);
  cudaFree(c->wts_alt);
  c->edges = ne;
  c->edges_alt = nea;
  c->wts = nw;
  c->wts_alt = nwa;
  c->cap = ncap;
  if (chunks) {
    cudaFree(c->chunk_tile);
    cudaFree(c->chunk_tile_alt);
    c->chunk_tile = ct;
    c->chunk_tile_alt = cta;
    c->chunk_cap = nch;
  }
  return upload_store_desc(c);  // the compaction may yet fail
}

int ensure_app_capacity(Ctx* c, uint64_t need) {
  if (need <= c->app_cap) return CYTOM_OK;
  uint64_t ncap = std::max<uint64_t>(need + need / 2, 1 << 16);
  uint64_t *k = nullptr, *ka = nullptr;
  uint32_t *w = nullptr, *wa = nullptr;
  cudaError_t e = cy_malloc(&k, ncap * 8);
  if (e == cudaSuccess) e = cy_malloc(&ka, ncap * 8);
  if (e == cudaSuccess && c->wtype) e = cy_malloc(&w, ncap * 4);
  if (e == cudaSuccess && c->wtype) e = cy_malloc(&wa, ncap * 4);
  if (e != cudaSuccess) {
    cudaGetLastError();
    cudaFree(k);
    cudaFree(ka);
    cudaFree(w);
    cudaFree(wa);
    return set_err(c, CYTOM_ERR_OOM, "append region growth");
  }
  if (c->A) {
    cudaMemcpyAsync(k, c->app_keys, c->A * 8, cudaMemcpyDeviceToDevice, c->stream);
    if (c->wtype) cudaMemcpyAsync(w, c->app_w, c->A * 4, cudaMemcpyDeviceToDevice, c->stream);
  }
  cudaStreamSynchronize(c->stream);
  cudaFree(c->app_keys);
  cudaFree(c->app_keys_alt);
  cudaFree(c->app_w);
  cudaFree(c->app_w_alt);
  c->app_keys = k;
  c->app_keys_alt = ka;
  c->app_w = w;
  c->app_w_alt = wa;
  c->app_cap = ncap;
  return CYTOM_OK;
}

__global__ void dir_tiles_kernel(const unsigned long long* __restrict__ tile_ptr, const uint32_t* __restrict__ edges,
                                 uint64_t ntiles, uint32_t* __restrict__ dir, uint32_t nbw);

int compact(Ctx* c) {
  if (c->A == 0) return CYTOM_OK;
  const uint64_t A = c->A;
  const bool wt = c->wtype != CYTOM_UNWEIGHTED;
  bool in_alt = false;
  int rc = radix_sort_pairs(c, c->app_keys, c->app_keys_alt, wt ? c->app_w : nullptr,
                            wt ? c->app_w_alt : nullptr, A, (int)(2 * (c->lvpt + c->lT)), &in_alt);
  if (rc) return rc;
  const uint64_t* K = in_alt ? c->app_keys_alt : c->app_keys;
  const uint32_t* W = wt ? (in_alt ? c->app_w_alt : c->app_w) : nullptr;
  rc = grow_store(c, c->E + A);
  if (rc) return rc;
  // temporaries
  const uint64_t nsp = (c->E + A + MERGE_SPAN - 1) / MERGE_SPAN;  // merge spans (upper bound)
  size_t bytes = A * (4 + 4 + 8 + 4 + 8 + 4 + 4 + 4) + 64 + 2 * (nsp + 1) * 4 + scan_scratch_words(A) * 4;
  char* tmp = nullptr;
  cudaError_t e = cy_malloc_async((void**)&tmp, bytes, c->stream);
  if (e != cudaSuccess) return set_err(c, CYTOM_ERR_OOM, "compaction temporaries");
  unsigned long long* lb = (unsigned long long*)tmp;
  unsigned long long* q = lb + A;
  uint32_t* keep = (uint32_t*)(q + A);
  uint32_t* P = keep + A;
  uint32_t* wsel = P + A;
  uint32_t* nloc = wsel + A;
  uint32_t* nw = nloc + A;
  uint32_t* ntile = nw + A;
  uint32_t* Kdev = ntile + A;
  uint32_t* sb = Kdev + 16;
  uint32_t* ts = sb + (nsp + 1);
  uint32_t* sscan = ts + (nsp + 1);
  int slot = prof_begin(c, KC_MERGE);
  dedupe_lookup_kernel<<<grid_for(c, A, 256), 256, 0, c->stream>>>(
      K, W, A, c->edges, c->wts, c->tile_ptr,
      c->dir && !c->dir_disabled && c->dir_version == c->version ? c->dir : nullptr, (uint32_t)(c->vpt / 32), c->lvpt,
      keep, lb, wsel);
  c->launches++;
  rc = scan_into(c, keep, P, A, Kdev, sscan);
  if (rc) {
    cudaFreeAsync(tmp, c->stream);
    return rc;
  }
  pack_kept_kernel<<<grid_for(c, A, 256), 256, 0, c->stream>>>(K, A, keep, P, lb, wsel, c->lvpt, q,
                                                               nloc, wt ? nw : nullptr, ntile, c->cmask, c->lT,
                                                               c->lT > 6 ? c->lT - 6 : 0u);
  c->launches++;
  new_tile_ptr_kernel<<<grid_for(c, c->ntiles + 1, 256), 256, 0, c->stream>>>(
      c->tile_ptr, c->ntiles, ntile, Kdev, c->tile_ptr_alt);
  c->launches++;
  // The merge writes only the alternate buffers (store, tile offsets, chunk table and,
  // once the context keeps one, the source directory), so it may overlap runs that still
  // read the installed snapshot.
  uint32_t* mdir = nullptr;
  if (c->dir && !c->dir_disabled) {
    if (!c->dir_alt && cy_malloc(&c->dir_alt, c->dir_entries * 4) != cudaSuccess) {
      cudaGetLastError();
      c->dir_alt = nullptr;
    }
    mdir = c->dir_alt;
  }
  merge_spans_kernel<<<grid_for(c, nsp + 1, 256), 256, 0, c->stream>>>(q, Kdev, c->E, c->tile_ptr_alt, c->ntiles,
                                                                       nsp, sb, ts, c->chunk_tile_alt);
  auto* mg = wt ? (mdir ? merge_gather_kernel<true, true> : merge_gather_kernel<true, false>)
                : (mdir ? merge_gather_kernel<false, true> : merge_gather_kernel<false, false>);
  mg<<<(unsigned)std::max<uint64_t>(1, std::min<uint64_t>((nsp + 7) / 8, (uint64_t)c->num_sms * 8)), 256, 0,
       c->stream>>>(c->edges, c->wts, c->E, q, nloc, nw, Kdev, sb, ts, nsp, c->tile_ptr_alt, c->chunk_tile_alt, mdir,
                    (uint32_t)(c->vpt / 32), c->edges_alt, wt ? c->wts_alt : nullptr);
  c->launches += 2;
  if (wt) {
    fixup_weights_kernel<<<grid_for(c, A, 256), 256, 0, c->stream>>>(lb, wsel, A, q, Kdev, c->wts_alt);
    c->launches++;
  }
  if (mdir) {  // the merge wrote every directory entry up to each tile's last source block
    dir_tiles_kernel<<<grid_for(c, c->ntiles * 32, 256), 256, 0, c->stream>>>(c->tile_ptr_alt, c->edges_alt, c->ntiles,
                                                                              mdir, (uint32_t)(c->vpt / 32));
    c->launches++;
  }
  e = cudaMemcpyAsync(c->h_pinned, Kdev, 4, cudaMemcpyDeviceToHost, c->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
  if (e != cudaSuccess) {
    cudaFreeAsync(tmp, c->stream);
    return cuda_err(c, e, "compaction");
  }
  uint64_t Kn = *(uint32_t*)c->h_pinned;
  prof_end(c, slot, (double)A * (wt ? 44.0 : 36.0) + (double)(c->E + Kn) * (wt ? 16.0 : 8.0));
  rc = pagerank_note_kept(c, nloc, ntile, Kn);  // the PageRank CSC's next build merges these in
  if (rc) {
    cudaFreeAsync(tmp, c->stream);
    return rc;
  }
  // Installing the merged snapshot: runs on the previous one must have finished (everything
  // above wrote to the new snapshot alone). The jobs are then seeded by the merged edges
  // (edgeChanged(INSERT)).
  join_runs(c);
  uint32_t* est = nullptr;  // the estimates' degrees, if the seeding pass brings them up to date
  {
    std::vector<Job*> mp;
    for (Job* j : c->jobs) {
      if (!j || j->fresh) continue;
      if (j->algo == CYTOM_ALGO_BFS || j->algo == CYTOM_ALGO_CC || j->algo == CYTOM_ALGO_SSSP ||
          j->algo == CYTOM_ALGO_SSWP)
        mp.push_back(j);
      else
        rc = job_seed_keys(c, j, K, W, A);  // the PageRank family: a residual round next time
      if (rc) break;
    }
    if (c->est_deg && c->est_version == c->version && !mp.empty()) est = c->est_deg;
    if (!rc && !mp.empty()) rc = minprop_seed_keys_many(c, mp.data(), (int)mp.size(), K, W, A, est);
    if (rc) {
      if (est) c->est_version = ~0ULL;
      cudaFreeAsync(tmp, c->stream);
      return rc;
    }
  }
  cudaFreeAsync(tmp, c->stream);
  if (c->dyn_pending) cudaMemsetAsync(c->dyn_pending, 0, c->ntiles * 4, c->stream);  // nothing appended now
  std::swap(c->edges, c->edges_alt);
  std::swap(c->wts, c->wts_alt);
  std::swap(c->tile_ptr, c->tile_ptr_alt);
  std::swap(c->chunk_tile, c->chunk_tile_alt);
  if (mdir) std::swap(c->dir, c->dir_alt);
  c->E += Kn;
  c->A = 0;
  c->version++;
  if (est) c->est_version = c->version;
  e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_err(c, e, "merge");
  if (mdir) c->dir_version = c->version;
  return upload_store_desc(c);
}

// Compact-vs-sparse flag per tile: distinct sources >= vpt / 2 (tile-manager.h:261-263).
__global__ void count_sources_kernel(const uint32_t* __restrict__ edges,
                                     const unsigned long long* __restrict__ tile_ptr,
                                     uint64_t ntiles, uint64_t vpt, uint8_t* __restrict__ flags) {
  // one warp per tile
  const unsigned lane = threadIdx.x & 31;
  uint64_t warp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  for (uint64_t t = warp; t < ntiles; t += nwarps) {
    uint64_t lo = tile_ptr[t], hi = tile_ptr[t + 1];
    uint32_t cnt = 0;
    for (uint64_t i = lo + lane; i < hi; i += 32) {
      uint32_t s = edges[i] >> 16;
      uint32_t prev = (i == lo) ? 0xFFFFFFFFu : (edges[i - 1] >> 16);
      cnt += (s != prev) ? 1u : 0u;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) cnt += __shfl_xor_sync(0xFFFFFFFFu, cnt, o);
    if (lane == 0) flags[t] = (hi > lo) ? (uint8_t)(cnt >= vpt / 2 ? 1 : 0) : 2;  // 2 = empty
  }
}

// Source directory for sparse rounds. Per edge: the 32-source blocks from just after
// the previous edge's block up to its own start at this edge. Per tile: the blocks after
// the last edge's block (all blocks of an empty tile) hold the tile size.
__global__ void dir_edges_kernel(const StoreDesc* __restrict__ sd, uint32_t* __restrict__ dir, uint32_t nbw) {
  // one warp per 128-edge chunk, four edges per lane; a chunk inside one tile (nearly
  // all of them) takes a 32-bit fast path
  const uint64_t E = sd->E, nchunks = sd->nchunks;
  const unsigned lane = threadIdx.x & 31;
  const uint64_t warp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  for (uint64_t c = warp; c < nchunks; c += nwarps) {
    const uint64_t cbase = c * kChunk;
    const uint64_t e0 = cbase + (uint64_t)lane * 4;
    const uint4 q = *reinterpret_cast<const uint4*>(sd->edges + e0);  // the store has kChunk slack
    uint32_t prev0 = __shfl_up_sync(0xFFFFFFFFu, q.w, 1);
    if (lane == 0) prev0 = cbase > 0 ? sd->edges[cbase - 1] : 0u;
    const uint32_t ev[5] = {prev0, q.x, q.y, q.z, q.w};
    uint32_t t = sd->chunk_tile[c];
    unsigned long long tlo = sd->tile_ptr[t], thi = sd->tile_ptr[t + 1];
    const uint64_t cend = cbase + kChunk < E ? cbase + kChunk : E;
    if (tlo <= cbase && cend <= thi) {
      if (thi - tlo < DIR_SMALL) continue;
      const uint64_t dt = (uint64_t)t * (nbw + 1);
      const uint32_t r0 = (uint32_t)(e0 - tlo);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const bool in = e0 + k < E;
        dir_runs(dir, dt, r0 + k == 0 ? 0 : (int)(ev[k] >> 21) + 1, in ? (int)(ev[k + 1] >> 21) : -1, r0 + k);
      }
      continue;
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const uint64_t e = e0 + k;
      int b0 = 0, b1 = -1;
      if (e < E) {
        while (thi <= e) {
          ++t;
          tlo = thi;
          thi = sd->tile_ptr[t + 1];
        }
        if (thi - tlo >= DIR_SMALL) {
          b1 = (int)(ev[k + 1] >> 21);
          b0 = e == tlo ? 0 : (int)(ev[k] >> 21) + 1;
        }
      }
      dir_runs(dir, (uint64_t)t * (nbw + 1), b0, b1, (uint32_t)(e - tlo));
    }
  }
}

// The end of every tile's directory, and all of it for tiles of fewer than DIR_SMALL edges,
// where an edge may start many blocks. One warp per tile.
__global__ void dir_tiles_kernel(const unsigned long long* __restrict__ tile_ptr, const uint32_t* __restrict__ edges,
                                 uint64_t ntiles, uint32_t* __restrict__ dir, uint32_t nbw) {
  const unsigned lane = threadIdx.x & 31;
  const uint64_t warp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  for (uint64_t t = warp; t < ntiles; t += nwarps) {
    const uint64_t lo = tile_ptr[t], hi = tile_ptr[t + 1];
    const uint32_t m = (uint32_t)(hi - lo);
    const uint64_t dt = t * (nbw + 1);
    const int blast = m ? (int)(edges[hi - 1] >> 21) : -1;
    if (hi - lo < DIR_SMALL) {
      int prev = -1;
      for (uint32_t i = 0; i < m; i += 32) {
        const int b = i + lane < m ? (int)(edges[lo + i + lane] >> 21) : -1;
        int bp = __shfl_up_sync(0xFFFFFFFFu, b, 1);
        if (lane == 0) bp = prev;
        prev = __shfl_sync(0xFFFFFFFFu, b, 31);
        dir_runs(dir, dt, bp + 1, b, i + lane);
      }
    }
    for (int bb = blast + 1 + (int)lane; bb <= (int)nbw; bb += 32) dir[dt + bb] = m;
  }
}

// Column-mask bits of every stored edge (a full directory build): one atomic per run of
// edges with the same source in a tile.
__global__ void cmask_all_kernel(const StoreDesc* __restrict__ sd, unsigned long long* __restrict__ cmask,
                                 uint32_t cshift) {
  const uint64_t E = sd->E, T = sd->T;
  const uint32_t lT = sd->lT, lvpt = sd->lvpt;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; e < E; e += stride) {
    uint64_t t = sd->chunk_tile[e / kChunk];
    while (sd->tile_ptr[t + 1] <= e) ++t;
    const uint32_t src = sd->edges[e] >> 16;
    if (e > sd->tile_ptr[t] && (sd->edges[e - 1] >> 16) == src) continue;
    atomicOr(cmask + (((t >> lT) << lvpt) | src), 1ULL << ((t & (T - 1)) >> cshift));
  }
}

int build_directory(Ctx* c) {
  if (c->dir_version == c->version || c->dir_disabled) return CYTOM_OK;
  const char* env = getenv("CYTOM_SPARSE");  // "0": dense rounds only
  if (c->lvpt < 5 || !c->cfg.enable_adaptive_scheduling || (env && env[0] == '0')) {
    c->dir_disabled = true;
    return upload_store_desc(c);
  }
  const uint64_t nbw = c->vpt / 32;
  const uint64_t entries = c->T * (nbw + 1) * c->T;
  // the directory is worth its memory only while it is small next to the edges
  if (entries * 4 > (4ULL << 30)) {
    c->dir_disabled = true;
    return upload_store_desc(c);
  }
  if (!c->dir) {
    if (cy_malloc(&c->dir, entries * 4) != cudaSuccess) {
      cudaGetLastError();
      c->dir_disabled = true;
      return upload_store_desc(c);
    }
    c->dir_entries = entries;
  }
  // column masks: without memory for them sparse rounds read every item's directory entry
  if (!c->cmask) {
    if (cy_malloc(&c->cmask, c->n * 8) != cudaSuccess) {
      cudaGetLastError();
      c->cmask = nullptr;
    } else {
      cudaMemsetAsync(c->cmask, 0, c->n * 8, c->stream);
    }
  }
  int slot = prof_begin(c, KC_MERGE);
  if (c->E) {
    dir_edges_kernel<<<grid_for(c, (c->E + 3) / 4, 256), 256, 0, c->stream>>>(c->dsd, c->dir, (uint32_t)nbw);
    c->launches++;
    if (c->cmask) {
      cmask_all_kernel<<<grid_for(c, c->E, 256), 256, 0, c->stream>>>(c->dsd, c->cmask, c->lT > 6 ? c->lT - 6 : 0u);
      c->launches++;
    }
  }
  dir_tiles_kernel<<<grid_for(c, c->ntiles * 32, 256), 256, 0, c->stream>>>(c->tile_ptr, c->edges, c->ntiles, c->dir,
                                                                            (uint32_t)nbw);
  c->launches++;
  prof_end(c, slot, (double)c->E * 8.0 + (double)entries * 4.0);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_err(c, e, "directory");
  c->dir_version = c->version;
  return upload_store_desc(c);
}

int compute_compact_flags(Ctx* c, uint8_t* dflags) {
  count_sources_kernel<<<grid_for(c, c->ntiles * 32, 256), 256, 0, c->stream>>>(
      c->edges, c->tile_ptr, c->ntiles, c->vpt, dflags);
  c->launches++;
  return cuda_err(c, cudaGetLastError(), "count_sources");
}


// Deletion of stored edges: the store side of TileManager::deleteEdge and of the
// deleted-edge filter of compactStorage / fillCSR (tile-manager.h:165-173, 249-253,
// 532-535), applied at once instead of kept as a deleted set. Request i finds
// (src[i], tgt[i]) in its tile (binary search over the sorted packed edges); the request
// that sets the edge's kill bit first drops out_deg[src] and in_deg[tgt] by one and
// appends (src, tgt, weight) to the deleted list. A pair that is not stored is skipped.
__global__ void delete_mark_kernel(const StoreDesc* __restrict__ sd, const uint32_t* __restrict__ src,
                                   const uint32_t* __restrict__ tgt, uint64_t count, uint32_t* kill,
                                   uint32_t* out_deg, uint32_t* in_deg, uint32_t* dsrc, uint32_t* dtgt,
                                   uint32_t* dw, unsigned long long* ndel) {
  const uint32_t lvpt = sd->lvpt, lT = sd->lT;
  const uint32_t lmask = (1u << lvpt) - 1u;
  uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += stride) {
    const uint32_t u = src[i], v = tgt[i];
    if ((uint64_t)u >= sd->n || (uint64_t)v >= sd->n) continue;
    const uint64_t t = ((uint64_t)(u >> lvpt) << lT) | (v >> lvpt);
    const uint32_t key = ((u & lmask) << 16) | (v & lmask);
    const uint64_t end = sd->tile_ptr[t + 1];
    uint64_t lo = sd->tile_ptr[t], hi = end;
    while (lo < hi) {
      const uint64_t mid = (lo + hi) >> 1;
      if (sd->edges[mid] < key) lo = mid + 1;
      else hi = mid;
    }
    if (lo >= end || sd->edges[lo] != key) continue;
    const uint32_t bit = 1u << (lo & 31);
    if (atomicOr(kill + (lo >> 5), bit) & bit) continue;  // another request took it
    atomicSub(out_deg + u, 1u);
    atomicSub(in_deg + v, 1u);
    const unsigned long long k = atomicAdd(ndel, 1ULL);
    dsrc[k] = u;
    dtgt[k] = v;
    if (dw) dw[k] = sd->wts[lo];
  }
}

// Kept edges per 32-edge word of the kill bitmap; word nw (one past the last) counts 0,
// so the exclusive scan's entry nw is the new edge count.
__global__ void keep_count_kernel(const uint32_t* __restrict__ kill, uint64_t E, uint64_t nw,
                                  uint32_t* __restrict__ cnt) {
  uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t w = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; w <= nw; w += stride) {
    if (w == nw) {
      cnt[w] = 0;
      continue;
    }
    const unsigned r = (unsigned)(E - w * 32);
    const uint32_t valid = r >= 32 ? 0xFFFFFFFFu : ((1u << r) - 1u);
    cnt[w] = __popc(~kill[w] & valid);
  }
}

// New position of old position p: kept edges before p.
__device__ __forceinline__ uint64_t kept_before(const uint32_t* kill, const uint32_t* P, uint64_t p) {
  const uint64_t w = p >> 5;
  const unsigned b = (unsigned)(p & 31);
  return (uint64_t)P[w] + (b ? (uint64_t)__popc(~kill[w] & ((1u << b) - 1u)) : 0ULL);
}

// Order-preserving gather of the kept edges (each tile stays sorted).
__global__ void delete_gather_kernel(const uint32_t* __restrict__ edges, const uint32_t* __restrict__ wts,
                                     uint64_t E, const uint32_t* __restrict__ kill, const uint32_t* __restrict__ P,
                                     uint32_t* __restrict__ oe, uint32_t* __restrict__ ow) {
  uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < E; i += stride) {
    const uint32_t k = kill[i >> 5];
    const unsigned b = (unsigned)(i & 31);
    if ((k >> b) & 1u) continue;
    const uint64_t o = (uint64_t)P[i >> 5] + __popc(~k & ((1u << b) - 1u));
    oe[o] = edges[i];
    if (ow) ow[o] = wts[i];
  }
}

__global__ void delete_tile_ptr_kernel(const unsigned long long* __restrict__ tile_ptr, uint64_t ntiles,
                                       const uint32_t* __restrict__ kill, const uint32_t* __restrict__ P,
                                       unsigned long long* __restrict__ out) {
  uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; t <= ntiles; t += stride)
    out[t] = kept_before(kill, P, tile_ptr[t]);
}

int minprop_delete_check(Ctx* c, Job* j, const uint32_t* dsrc, const uint32_t* dtgt, const uint32_t* dw,
                         uint64_t count, unsigned* tight);

// Removes the stored (src, tgt) pairs listed (device pointers) after compacting pending
// inserts. The store is rewritten without them in one order-preserving pass; BFS / CC /
// SSSP / SSWP jobs restart only if a deleted edge was tight for them, the PageRank
// family re-converges on the new snapshot (its first round is a residual round).
int delete_edges(Ctx* c, const uint32_t* src, const uint32_t* tgt, uint64_t count, uint64_t* removed) {
  if (removed) *removed = 0;
  int rc = compact(c);
  if (rc) return rc;
  const uint64_t E = c->E;
  if (E == 0 || count == 0) return CYTOM_OK;
  const bool wt = c->wtype != CYTOM_UNWEIGHTED;
  const uint64_t nw = (E + 31) / 32;
  std::vector<Job*> mp;
  for (Job* j : c->jobs)
    if (j && !j->fresh && (j->algo == CYTOM_ALGO_BFS || j->algo == CYTOM_ALGO_CC || j->algo == CYTOM_ALGO_SSSP ||
                           j->algo == CYTOM_ALGO_SSWP))
      mp.push_back(j);
  // temporaries: kill[nw+1], cnt[nw+1], P[nw+1], total, deleted list 3 x count, the scan's
  // scratch (nothing is allocated once the degrees are lowered), ndel, tight flags
  const uint64_t words = 3 * (nw + 1) + 1 + 3 * count + scan_scratch_words(nw + 1);
  const size_t bytes = ((words * 4 + 15) / 16) * 16 + 8 + (mp.size() + 1) * 4;
  char* tmp = nullptr;
  cudaError_t e = cy_malloc_async((void**)&tmp, bytes, c->stream);
  if (e != cudaSuccess) return set_err(c, CYTOM_ERR_OOM, "deletion temporaries");
  uint32_t* kill = (uint32_t*)tmp;
  uint32_t* cnt = kill + (nw + 1);
  uint32_t* P = cnt + (nw + 1);
  uint32_t* total = P + (nw + 1);
  uint32_t* dsrc = total + 1;
  uint32_t* dtgt = dsrc + count;
  uint32_t* dw = dtgt + count;
  uint32_t* sscan = dw + count;
  unsigned long long* ndel = (unsigned long long*)(tmp + ((words * 4 + 15) / 16) * 16);
  unsigned* tight = (unsigned*)(ndel + 1);
  cudaMemsetAsync(kill, 0, (nw + 1) * 4, c->stream);
  cudaMemsetAsync(ndel, 0, 8 + (mp.size() + 1) * 4, c->stream);
  int slot = prof_begin(c, KC_MERGE);
  delete_mark_kernel<<<grid_for(c, count, 256), 256, 0, c->stream>>>(c->dsd, src, tgt, count, kill, c->out_deg,
                                                                       c->in_deg, dsrc, dtgt, wt ? dw : nullptr, ndel);
  c->launches++;
  e = cudaMemcpyAsync(c->h_pinned, ndel, 8, cudaMemcpyDeviceToHost, c->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
  if (e != cudaSuccess) {
    cudaFreeAsync(tmp, c->stream);
    return cuda_err(c, e, "deletion");
  }
  const uint64_t nd = *(unsigned long long*)c->h_pinned;
  if (nd == 0) {
    cudaFreeAsync(tmp, c->stream);
    prof_end(c, slot, (double)count * 8.0);
    return CYTOM_OK;
  }
  keep_count_kernel<<<grid_for(c, nw + 1, 256), 256, 0, c->stream>>>(kill, E, nw, cnt);
  c->launches++;
  rc = scan_into(c, cnt, P, nw + 1, total, sscan);
  if (rc) {
    cudaFreeAsync(tmp, c->stream);
    return rc;
  }
  delete_gather_kernel<<<grid_for(c, E, 256, 16), 256, 0, c->stream>>>(c->edges, c->wts, E, kill, P, c->edges_alt,
                                                                       wt ? c->wts_alt : nullptr);
  c->launches++;
  delete_tile_ptr_kernel<<<grid_for(c, c->ntiles + 1, 256), 256, 0, c->stream>>>(c->tile_ptr, c->ntiles, kill, P,
                                                                                  c->tile_ptr_alt);
  c->launches++;
  for (size_t k = 0; k < mp.size(); ++k) {
    rc = minprop_delete_check(c, mp[k], dsrc, dtgt, wt ? dw : nullptr, nd, tight + k);
    if (rc) {
      cudaFreeAsync(tmp, c->stream);
      return rc;
    }
  }
  std::vector<unsigned> tflags(mp.size() + 1, 0);
  e = cudaMemcpyAsync(tflags.data(), tight, (mp.size() + 1) * 4, cudaMemcpyDeviceToHost, c->stream);
  cudaFreeAsync(tmp, c->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
  if (e != cudaSuccess) return cuda_err(c, e, "deletion");
  prof_end(c, slot, (double)count * 8.0 + (double)E * (wt ? 16.0 : 8.0));
  std::swap(c->edges, c->edges_alt);
  std::swap(c->wts, c->wts_alt);
  std::swap(c->tile_ptr, c->tile_ptr_alt);
  c->E = E - nd;
  c->version++;
  for (size_t k = 0; k < mp.size(); ++k)
    if (tflags[k]) mp[k]->fresh = true;
  if (removed) *removed = nd;
  const uint64_t nch = (c->E + kChunk - 1) / kChunk;
  chunk_tile_kernel<<<grid_for(c, nch + 1, 256), 256, 0, c->stream>>>(c->tile_ptr, c->ntiles, nch, c->chunk_tile);
  c->launches++;
  e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_err(c, e, "chunk_tile");
  return upload_store_desc(c);
}

// Random deletion picks (the reference's deletion_percentage mode,
// meta-tile-manager.h:201-231, with TileManager::deleteRandomEdge, tile-manager.h:175-190):
// pick i chooses a tile uniformly by hash64(hash64(seed) + 2i) and one of its edges
// uniformly by hash64(hash64(seed) + 2i + 1); an empty tile yields no edge (UINT32_MAX
// twice, which the deletion skips).
__global__ void pick_random_kernel(const StoreDesc* __restrict__ sd, uint64_t ntiles, uint64_t count,
                                   uint64_t hs, uint32_t* __restrict__ src, uint32_t* __restrict__ tgt) {
  const uint32_t lvpt = sd->lvpt, lT = sd->lT;
  const uint64_t tmask = (1ULL << lT) - 1ULL;
  uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += stride) {
    const uint64_t t = hash64(hs + 2 * i) % ntiles;
    const uint64_t lo = sd->tile_ptr[t], len = sd->tile_ptr[t + 1] - lo;
    if (len == 0) {
      src[i] = tgt[i] = 0xFFFFFFFFu;
      continue;
    }
    const uint32_t e = sd->edges[lo + hash64(hs + 2 * i + 1) % len];
    src[i] = (uint32_t)((t >> lT) << lvpt) | (e >> 16);
    tgt[i] = (uint32_t)((t & tmask) << lvpt) | (e & 0xFFFFu);
  }
}

int delete_random(Ctx* c, uint64_t count, uint64_t seed, uint32_t* src, uint32_t* tgt, uint64_t* removed) {
  if (removed) *removed = 0;
  int rc = compact(c);
  if (rc || count == 0) return rc;
  pick_random_kernel<<<grid_for(c, count, 256), 256, 0, c->stream>>>(c->dsd, c->ntiles, count, hash64(seed), src,
                                                                     tgt);
  c->launches++;
  rc = cuda_err(c, cudaGetLastError(), "random picks");
  if (rc) return rc;
  return delete_edges(c, src, tgt, count, removed);
}

// Weight update of stored edges: update i finds (src[i], tgt[i]) in its tile (binary
// search over the tile's sorted packed edges) and overwrites its weight; an edge that
// is not stored sets *missing.
__global__ void set_weights_kernel(const StoreDesc* __restrict__ sd, const uint32_t* __restrict__ src,
                                   const uint32_t* __restrict__ tgt, const uint32_t* __restrict__ w, uint64_t count,
                                   uint32_t* wts, unsigned* missing) {
  const uint32_t lvpt = sd->lvpt, lT = sd->lT;
  const uint32_t lmask = (1u << lvpt) - 1u;
  uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += stride) {
    const uint32_t u = src[i], v = tgt[i];
    if ((uint64_t)u >= sd->n || (uint64_t)v >= sd->n) {
      atomicOr(missing, 1u);
      continue;
    }
    const uint64_t t = ((uint64_t)(u >> lvpt) << lT) | (v >> lvpt);
    const uint32_t key = ((u & lmask) << 16) | (v & lmask);
    uint64_t lo = sd->tile_ptr[t], hi = sd->tile_ptr[t + 1];
    while (lo < hi) {
      const uint64_t mid = (lo + hi) >> 1;
      if (sd->edges[mid] < key) lo = mid + 1;
      else hi = mid;
    }
    if (lo < sd->tile_ptr[t + 1] && sd->edges[lo] == key) wts[lo] = w[i];
    else atomicOr(missing, 1u);
  }
}

int set_edge_weights(Ctx* c, const uint32_t* src, const uint32_t* tgt, const uint32_t* w, uint64_t count) {
  int rc = compact(c);
  if (rc) return rc;
  cudaMemsetAsync(c->d_flag, 0, 4, c->stream);
  if (count) {
    set_weights_kernel<<<grid_for(c, count, 256), 256, 0, c->stream>>>(c->dsd, src, tgt, w, count, c->wts,
                                                                          c->d_flag);
    c->launches++;
  }
  unsigned missing = 0;
  cudaError_t e = cudaMemcpyAsync(&missing, c->d_flag, 4, cudaMemcpyDeviceToHost, c->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
  if (e != cudaSuccess) return cuda_err(c, e, "weight update");
  // every weight-dependent structure is rebuilt; SSSP and SSWP jobs restart (a changed
  // weight can worsen a path, which min- or max-propagation cannot undo)
  c->version++;
  rc = upload_store_desc(c);
  if (rc) return rc;
  for (Job* j : c->jobs)
    if (j && (j->algo == CYTOM_ALGO_SSSP || j->algo == CYTOM_ALGO_SSWP)) j->fresh = true;
  if (missing) return set_err(c, CYTOM_ERR_RANGE, "weight update of an edge that is not stored");
  return CYTOM_OK;
}

}  // namespace cytom
