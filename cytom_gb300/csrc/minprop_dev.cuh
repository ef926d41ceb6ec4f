// minprop_dev.cuh — device building blocks of one BFS / CC / SSSP round, shared by the
// one-job kernels (exec_minprop.cu) and the batched persistent executor (exec_batch.cu),
// so both compute the same round with the same arithmetic.
//
// The round is the reference's Jacobi round (src/include/core/continuous-algorithm-executor.h:72-218):
//   gather  — AlgorithmExecutor::executeTile / executeAlgorithmSingleEdge[Weighted]
//             (src/include/core/algorithm-executor.h:214-505): every edge whose source is
//             active relaxes next[tgt] from current[src];
//   apply   — ApplyExecutor::run (src/include/core/apply-executor.h:40-115): changed
//             vertices copy next into current and form the next frontier;
//   control — the convergence test and the swap of the active bitmaps
//             (continuous-algorithm-executor.h:193-218).
//
// Load policy (PERSIST): the one-job kernels read state written by earlier launches through
// the read-only path (0). The cluster kernel of the small rounds writes that state in the same
// launch on other SMs and reads every mutable word through L2 (1). The batched executor also
// writes it in the same launch, but a block reads it only in a phase that it entered by a
// claim and a fence after the phase that wrote it had ended, so ordinary loads see it and may
// hit in L1 (2); words that change within a phase (next) are read through L2 by all.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "engine.h"
#include "ptx.cuh"

namespace cytom {

constexpr int APPLY_T = 256;
constexpr int SG_T = 256;     // threads of a dense-stage block
constexpr int SG_E = 4096;    // edges per dense stage
static_assert(SG_E == SG_T * 16, "16 edges per thread per stage");

// Loads of data that a launch may have written (current values, frontier, changed bits,
// row flags).
template <int PERSIST, class T>
__device__ __forceinline__ T ld_state(const T* p) {
  if constexpr (PERSIST == 1) return __ldcg(p);
  else if constexpr (PERSIST == 2) return *p;
  else return __ldg(p);
}
// The same for words that the one-job kernels also read with plain loads.
template <int PERSIST, class T>
__device__ __forceinline__ T ld_plain(const T* p) {
  if constexpr (PERSIST == 1) return __ldcg(p);
  else return *p;
}

// Programs: ALGO 0 BFS, 1 CC, 2 SSSP, 3 SSWP. SSWP runs on complemented values (v' = ~v),
// which turns its max(v, min(u, w)) into the same min-propagation as the others:
// v' = min(v', max(u', ~w)); unreached (0) is kInf, the start (UINT32_MAX) is 0.
template <int ALGO>
__host__ __device__ constexpr bool mp_weighted() {
  return ALGO >= 2;
}
// The value an edge offers its target from source value c (c != kInf) and weight w.
template <int ALGO>
__device__ __forceinline__ uint32_t mp_cand(uint32_t c, uint32_t w) {
  if (ALGO == 0) return c + 1;
  if (ALGO == 1) return c;
  if (ALGO == 2) {
    const uint32_t sum = c + w;  // c < kInf; a carry out or kInf itself means unreachable
    return (sum < c || sum == kInf) ? kInf : sum;
  }
  return max(c, ~w);
}

// Pre-check of a target's next value before the reduction, through L2. (Any value read
// would do: next only decreases during a round and never exceeds current. Reading the
// one-job kernels' pre-checks through L1 instead measured 2-3 % slower on the RMAT-22
// stream's dense SSSP rounds.)
__device__ __forceinline__ uint32_t ld_next(const uint32_t* p) {
  return __ldcg(p);
}

// Source value of a gather. The asynchronous programs (examples/bfs-async.cc,
// cc-async.cc: ASYNC = true) pull from next[src], which other blocks lower during the
// round (algorithm-executor.h:303-312); read through L2, a value is either the one at
// the round's start or a lower one, and both are valid bounds.
template <int PERSIST>
__device__ __forceinline__ uint32_t ld_src(const JobDesc* __restrict__ jd, bool async, uint64_t u) {
  if (async) return __ldcg(jd->next + u);
  return ld_state<PERSIST>(jd->cur + u);
}

__device__ __forceinline__ unsigned long long row_edges(const StoreDesc* sd, uint64_t x) {
  return sd->tile_ptr[(x + 1) << sd->lT] - sd->tile_ptr[x << sd->lT];
}

// Opening of gather round p: clears the next parity's row flags (threads tid, tid+nthr,
// ...) and, on thread 0, the next parity's counters; adds the round's processed-edge
// count (edges of tile rows with an active source, algorithm-executor.h:424-426).
template <int PERSIST>
__device__ __forceinline__ void round_open(const JobDesc* __restrict__ jd, const StoreDesc* __restrict__ sd,
                                           unsigned p, int adaptive, uint64_t tid, uint64_t nthr) {
  LoopState* ls = jd->ls;
  const uint64_t T = sd->T;
  unsigned* rows_nxt = jd->rows + (p ^ 1u) * T;
  for (uint64_t i = tid; i < T; i += nthr) rows_nxt[i] = 0;
  if (tid == 0) {
    ls->active[p ^ 1u] = 0;
    ls->nact_words[p ^ 1u] = 0;
    ls->teps[p ^ 1u] = 0;
    ls->est[p ^ 1u] = 0;
    atomicAdd(&ls->count_edges, adaptive ? ld_plain<PERSIST>(&ls->teps[p]) : sd->E);
  }
}

// Tile columns in which the active sources of frontier word i (bits w) may have edges:
// the OR of their column masks, read for words with at most four active sources (the
// sparse rounds' words hold about one); all columns for denser words or without masks.
__device__ __forceinline__ unsigned long long word_columns(const StoreDesc* __restrict__ sd, uint64_t i,
                                                           uint32_t w) {
  const unsigned long long* cm = sd->cmask;
  if (!cm || __popc(w) > 4) return ~0ULL;
  unsigned long long m = 0;
  const unsigned long long* row = cm + (i << 5);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    if (w) {
      m |= row[__ffs(w) - 1];
      w &= w - 1;
    }
  }
  return m;
}

// ---- small rounds --------------------------------------------------------
// A round is small when one thread-block cluster finishes it sooner than the grid-wide
// kernels, whose launches cost about 20 us whatever the frontier holds: on a graph of at
// most SMALL_E edges a round of at most SMALL_LISTED frontier words, else a sparse round of at
// most SMALL_ITEMS (word, column) items whose active vertices have at most SMALL_EDGES
// out-edges (LoopState::est). The cluster scans the changed bitmap every round, which bounds the
// vertices (SMALL_WORDS).
// Times of a round, cluster / grid-wide, in us, on graphs whose rounds all look alike:
//   items (2^22 vertices)   1,024: 10.3 / 19.4   8,192: 10.8 / 19.4   65,536: 13.2 / 20.5
//   out-edges (2^20)        4,600: 11.5 / 21.3   66,000: 18.9 / 28.2  263,000: 34 / 55
//   vertices                2^20: 7.6 / 17.6     2^24: 15.6 / 20.9    2^25: 22.0 / 23.3
//   edges, CC's whole run   65,500 (2^15 vertices): 348 / 754   131,000: 231 / 367   262,000: 249 / 289
// so the limits of items, out-edges and edges lie below where the two meet on such graphs. Whole
// workloads with one limit moved: 2^12 items, lattice of 2^18 vertices 19.5 ms, 2^13 17.9, 2^14 and
// 2^16 as long (RMAT-22 stream 54.1, 53.8, 53.7, 53.0); 2^14 out-edges, lattice 23.0, 2^16 17.9, 2^18
// 17.5; 2^14 edges, BFS on RMAT-12 167 us, 2^16 and 2^18 115; 2^16 words, stream 54.6, 2^19 53.8.
// CC from scratch lists every word: with 60,000 edges 2^15 words take 123 us, grid-wide 139,
// 2^16 words 165 / 141, 2^19 words 772 / 420 (three to five rounds).
constexpr uint32_t SMALL_E = 1u << 16;
constexpr uint32_t SMALL_LISTED = 1u << 15;
constexpr uint32_t SMALL_ITEMS = 1u << 13;
constexpr uint32_t SMALL_EDGES = 1u << 16;
constexpr uint32_t SMALL_WORDS = 1u << 19;
constexpr uint32_t EST_MAX = 1u << 20;  // est saturates per block here

// Listed frontier words whose out-edges the estimate needs: with more the round is not a small
// one whatever they hold. (On a graph of at most SMALL_E edges the estimate also chooses a small
// round's gather.)
__device__ __forceinline__ uint32_t est_words(const StoreDesc* __restrict__ sd) {
  return sd->E <= SMALL_E ? SMALL_LISTED : (SMALL_ITEMS >> sd->lT) + 1u;
}

// Out-edges of the active vertices of frontier word i (bits w), their degrees in flight
// together; words past the vertex count (fewer than 32 vertices) one by one.
__device__ __forceinline__ unsigned word_edges(const StoreDesc* __restrict__ sd, uint64_t i, uint32_t w) {
  const uint32_t* deg = sd->out_deg + (i << 5);
  unsigned long long e = 0;
  if (__popc(w) > 4 && ((i + 1) << 5) <= sd->n) {
    uint4 q[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) q[k] = __ldcg(reinterpret_cast<const uint4*>(deg) + k);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const uint32_t m = w >> (4 * k);
      e += (m & 1u ? q[k].x : 0u);
      e += (m & 2u ? q[k].y : 0u);
      e += (m & 4u ? q[k].z : 0u);
      e += (m & 8u ? q[k].w : 0u);
    }
  } else {
    uint32_t d[4];
    do {
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        d[k] = w ? __ldcg(deg + (__ffs(w) - 1)) : 0u;
        w &= w - 1;
      }
      e += (unsigned long long)d[0] + d[1] + d[2] + d[3];
    } while (w);
  }
  return (unsigned)(e < EST_MAX ? e : EST_MAX);
}

// The limits of a small round of `nact` listed words on a graph whose vertex range allows them.
__device__ __forceinline__ bool small_round(uint64_t E, uint32_t lT, bool listed, unsigned nact, unsigned est) {
  return nact <= SMALL_LISTED &&
         (E <= SMALL_E || (listed && ((uint64_t)nact << lT) <= SMALL_ITEMS && est <= SMALL_EDGES));
}

// The gather of a round with `nact` listed frontier words.
__device__ __forceinline__ unsigned pick_mode(const JobDesc* __restrict__ jd, const StoreDesc* __restrict__ sd,
                                              unsigned nact, unsigned est, int allow_small) {
  const uint64_t nwords = (sd->n + 31) >> 5;
  const bool listed = sd->dir_ok && sd->adaptive;
  if (allow_small && sd->small_ok && nwords <= SMALL_WORDS && small_round(sd->E, sd->lT, listed, nact, est)) return 2u;
  const uint32_t div = jd->sparse_div ? jd->sparse_div : sd->sparse_div;
  return (listed && (uint64_t)nact * div <= nwords) ? 1u : 0u;
}

// ---- apply ---------------------------------------------------------------
// One apply step of a block: thread t handles frontier word base + t (base a multiple
// of 32). `initial` apply = the seeding apply before round 0 (writes parity 0).
// rows[parity][x] receives the number of vertices of tile row x that are active in
// the next round (0 = the row is skipped; vpt = every source active, the frontier
// test is skipped). A warp covers 32 consecutive words; when they share one row
// (vpt >= 1024) it adds its row count with a single atomic. The non-zero frontier
// words are listed (warp-ballot compaction) for sparse rounds; those listed first, est_lim
// (est_words) of them, add to the estimate.
template <int PERSIST>
__device__ __forceinline__ void apply_step(const JobDesc* __restrict__ jd, const StoreDesc* __restrict__ sd,
                                           unsigned pw, uint64_t base, uint32_t est_lim, unsigned& cnt,
                                           unsigned long long& teps, unsigned& est) {
  LoopState* ls = jd->ls;
  const uint64_t n = sd->n, T = sd->T;
  const uint32_t lvpt = sd->lvpt;
  const uint64_t nwords = (n + 31) >> 5;
  unsigned* rows_w = jd->rows + pw * T;
  uint32_t* __restrict__ ch = jd->ch;
  uint32_t* __restrict__ fa = jd->fa;
  uint32_t* __restrict__ cur = jd->cur;
  const uint32_t* __restrict__ next = jd->next;
  const unsigned lane = threadIdx.x & 31;
  const uint64_t i = base + threadIdx.x;
  uint32_t w = 0;
  if (i < nwords) {
    w = ld_plain<PERSIST>(ch + i);
    fa[i] = w;
    if (w) {
      ch[i] = 0;
      if (!PERSIST && __popc(w) > 2 && ((i + 1) << 5) <= n) {
        // many changed vertices: the whole word's 32 values in one round trip. A vertex
        // without its changed bit holds next == current (every lowering of next sets
        // the bit), so copying it is a no-op. (Not in the persistent kernel, whose
        // register budget would spill the eight vectors.)
        const uint4* src = reinterpret_cast<const uint4*>(next + (i << 5));
        uint4* dst = reinterpret_cast<uint4*>(cur + (i << 5));
        uint4 q[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) q[k] = ld_plain<PERSIST>(src + k);
#pragma unroll
        for (int k = 0; k < 8; ++k) dst[k] = q[k];
      } else {
        uint32_t bits = w;
        while (bits) {
          const int b = __ffs(bits) - 1;
          bits &= bits - 1;
          const uint64_t v = (i << 5) + b;
          cur[v] = ld_plain<PERSIST>(next + v);
        }
      }
    }
  }
  const unsigned pc = __popc(w);
  cnt += pc;
  {
    const unsigned nz = __ballot_sync(0xFFFFFFFFu, w != 0);
    if (nz) {
      unsigned slot0 = 0;
      if (lane == 0) slot0 = atomicAdd(&ls->nact_words[pw], (unsigned)__popc(nz));
      slot0 = __shfl_sync(0xFFFFFFFFu, slot0, 0);
      if (w) {
        const unsigned slot = slot0 + __popc(nz & ((1u << lane) - 1u));
        jd->aw[slot] = (uint32_t)i;
        jd->awm[slot] = word_columns(sd, i, w);
        if (!PERSIST && slot < est_lim) est = min(est + word_edges(sd, i, w), EST_MAX);
      }
    }
  }
  if (lvpt >= 10) {
    unsigned tot = pc;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) tot += __shfl_xor_sync(0xFFFFFFFFu, tot, o);
    if (lane == 0 && tot) {
      const uint64_t x = ((base + (threadIdx.x & ~31u)) << 5) >> lvpt;
      if (atomicAdd(&rows_w[x], tot) == 0) teps += row_edges(sd, x);
    }
  } else if (w) {
    uint32_t bits = w;
    while (bits) {
      const int b = __ffs(bits) - 1;
      const uint64_t v = (i << 5) + b;
      const uint64_t x = v >> lvpt;
      const uint64_t row_first = x << lvpt;
      const uint64_t row_last = row_first + (1ULL << lvpt);  // exclusive
      uint32_t mrow = bits;
      if (row_last < ((i + 1) << 5)) mrow &= (1u << (uint32_t)(row_last - (i << 5))) - 1u;
      bits &= ~mrow;
      if (atomicAdd(&rows_w[x], (unsigned)__popc(mrow)) == 0) teps += row_edges(sd, x);
    }
  }
}

// Block reduction of the apply counters into the loop state (every thread calls it).
template <int T>
__device__ __forceinline__ void apply_flush(LoopState* ls, unsigned pw, unsigned cnt, unsigned long long teps,
                                            unsigned est) {
  __shared__ unsigned s_cnt[T / 32], s_est[T / 32];
  __shared__ unsigned long long s_teps[T / 32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    cnt += __shfl_xor_sync(0xFFFFFFFFu, cnt, o);
    teps += __shfl_xor_sync(0xFFFFFFFFu, teps, o);
    est = min(est + __shfl_xor_sync(0xFFFFFFFFu, est, o), EST_MAX);
  }
  const unsigned wid = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) {
    s_cnt[wid] = cnt;
    s_teps[wid] = teps;
    s_est[wid] = est;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned c = 0, e = 0;
    unsigned long long t = 0;
    for (int k = 0; k < T / 32; ++k) {
      c += s_cnt[k];
      t += s_teps[k];
      e = min(e + s_est[k], EST_MAX);
    }
    if (c) atomicAdd(&ls->active[pw], c);
    if (t) atomicAdd(&ls->teps[pw], t);
    if (e) atomicAdd(&ls->est[pw], e);
  }
  __syncthreads();
}

// ---- control -------------------------------------------------------------
// Ends a round (or, `initial`, the seeding apply): advances the round counter, ends the
// run when nothing changed or max_iterations rounds ran, and picks the next round's
// gather: sparse (directory, only the listed frontier words) while at most 1/sparse_div
// of the frontier words are non-zero, dense (stream every active row) above.
// The one-job loops (allow_small) run small rounds in one cluster (pick_mode).
__device__ __forceinline__ unsigned control_step(const JobDesc* __restrict__ jd, const StoreDesc* __restrict__ sd,
                                                 int initial, int allow_small) {
  // every word the step reads is loaded before any is used (one L2 round trip); the other
  // blocks' totals are complete and visible when it runs
  LoopState* ls = jd->ls;
  const unsigned was = __ldcg(&ls->cont), it0 = __ldcg(&ls->iter), max_iter = __ldcg(&ls->max_iter);
  const unsigned err = __ldcg(&ls->err);
  const unsigned act[2] = {__ldcg(&ls->active[0]), __ldcg(&ls->active[1])};
  const unsigned nact[2] = {__ldcg(&ls->nact_words[0]), __ldcg(&ls->nact_words[1])};
  const unsigned est[2] = {__ldcg(&ls->est[0]), __ldcg(&ls->est[1])};
  const unsigned long long total = __ldcg(&ls->active_total);
  if (!was) return 0u;
  const unsigned iter = initial ? it0 : it0 + 1;
  const unsigned p = initial ? 0u : (iter & 1u);
  const unsigned a = act[p];
  const unsigned cont = (a > 0 && iter < max_iter && err == 0) ? 1u : 0u;
  volatile LoopState* vls = ls;
  vls->iter = iter;
  vls->active_total = total + a;
  vls->cont = cont;
  vls->mode = pick_mode(jd, sd, nact[p], est[p], allow_small);
  vls->spq_count = 0;
  return cont;
}

// The loop state of a BFS / CC / SSSP / SSWP run before its first round (one thread).
__device__ __forceinline__ void minprop_begin_state(LoopState* ls, unsigned max_iter) {
  ls->iter = 0;
  ls->max_iter = max_iter;
  ls->cont = 1;
  ls->err = 0;
  ls->active[0] = ls->active[1] = 0;
  ls->nact_words[0] = ls->nact_words[1] = 0;
  ls->mode = 0;
  ls->spq_count = 0;
  ls->teps[0] = ls->teps[1] = 0;
  ls->count_edges = 0;
  ls->edges_scanned = 0;
  ls->active_total = 0;
  ls->apply_done = 0;
  ls->sel_rounds = 0;
  ls->items_read = 0;
  ls->est[0] = ls->est[1] = 0;
}

// Tile of edge e of the store: from its chunk's first tile on.
__device__ __forceinline__ uint32_t edge_tile(const uint32_t* __restrict__ chunk_tile,
                                              const unsigned long long* __restrict__ tile_ptr, uint64_t e) {
  uint32_t t = chunk_tile[e >> 7];
  while (tile_ptr[t + 1] <= e) ++t;
  return t;
}

// ---- dense gather: one stage of SG_T * EPT edges ---------------------------
// Processes stage `st` (EPT edges per thread, a multiple of 4) whose edges (and weights) are at eb / wb: shared memory for the
// bulk-copy pipeline, global memory (FROM_GLOBAL, guarded loads) for the persistent
// kernel. Single-row stages (the common case at large vertices-per-tile) take the source
// row from the stage: the frontier test needs no per-edge tile lookup, and only edges
// with an active source look up their target tile. Target updates are fire-and-forget
// red.min / red.or: a candidate below the value read is below current[v] too
// (next <= current), so next[v] ends the round below current[v] and v changed.
template <int ALGO, int PERSIST, bool FROM_GLOBAL, int EPT = 16>
__device__ __forceinline__ void dense_stage(const JobDesc* __restrict__ jd, const StoreDesc* __restrict__ sd,
                                            const uint32_t* eb, const uint32_t* wb, uint64_t st, unsigned p,
                                            int adaptive) {
  const uint64_t T = sd->T;
  const unsigned* rows_cur = jd->rows + p * T;
  const uint32_t* __restrict__ chunk_tile = sd->chunk_tile;
  const unsigned long long* __restrict__ tile_ptr = sd->tile_ptr;
  const uint32_t* fa = jd->fa;
  const bool async = jd->async != 0;
  uint32_t* next = jd->next;
  uint32_t* ch = jd->ch;
  const uint64_t E = sd->E, nchunks = sd->nchunks;
  const uint32_t lT = sd->lT, lvpt = sd->lvpt;
  const uint32_t ymask = (uint32_t)(T - 1);
  constexpr uint32_t SE = SG_T * EPT;  // edges of a stage
  static_assert(EPT % 4 == 0 && EPT <= 32 && SE % kChunk == 0, "stage shape");
  const uint64_t e0 = st * SE;
  const uint64_t rem = E - e0;
  const uint32_t cnt = rem < (uint64_t)SE ? (uint32_t)rem : SE;
  // tiles of the stage's first edge and of the first edge after it
  uint32_t tf, ta;
  {
    const uint64_t c0 = st * (SE / kChunk);
    uint64_t c1 = c0 + SE / kChunk;
    if (c1 > nchunks) c1 = nchunks;
    tf = chunk_tile[c0];
    ta = chunk_tile[c1];
  }
  const bool single_row = (tf >> lT) == (ta >> lT);
  const uint32_t vpt = 1u << lvpt;
  // a stage of at most two tiles in a row: the place of the boundary tells an edge's tile
  const bool two_tiles = ta - tf <= 1u;
  const uint32_t cut = ta == tf ? SE : (uint32_t)min((unsigned long long)SE, tile_ptr[tf + 1] - e0);
  // a fully active row needs no frontier test
  const bool full_row = single_row && (!adaptive || ld_plain<PERSIST>(rows_cur + (tf >> lT)) == vpt);

  // Lanes take consecutive edges: the sources of a warp's 32 edges, sorted in their tile, lie
  // in few cache lines. The round is bound by the requests of its SM to L2 (one a cycle) and by
  // the divergent lines an L1 access walks; with four consecutive edges a lane every load of
  // a source value touched 32 lines (RMAT-24, ids without order, CC and BFS: 10.9 -> 9.8 ms;
  // RMAT-22 stream 72.9 -> 71.3).
  uint32_t qv[EPT], ww[EPT], uu[EPT];
  uint32_t vmask = 0;
#pragma unroll
  for (int k = 0; k < EPT; ++k) {
    const uint32_t i = threadIdx.x + (uint32_t)k * SG_T;
    const bool in = i < cnt;
    qv[k] = (!FROM_GLOBAL || in) ? eb[i] : 0u;
    ww[k] = (mp_weighted<ALGO>() && (!FROM_GLOBAL || in)) ? wb[i] : 0u;
    vmask |= in ? (1u << k) : 0u;
  }
  if (single_row) {
    const uint32_t xb = (tf >> lT) << lvpt;
#pragma unroll
    for (int idx = 0; idx < EPT; ++idx) uu[idx] = xb | (qv[idx] >> 16);
  } else {
    // general path: per-edge tile lookup for the source row
#pragma unroll
    for (int idx = 0; idx < EPT; ++idx) {
      uu[idx] = 0;
      if ((vmask >> idx) & 1u) {
        const uint32_t i = threadIdx.x + (uint32_t)idx * SG_T;
        const uint32_t t = two_tiles ? (i < cut ? tf : ta) : edge_tile(chunk_tile, tile_ptr, e0 + i);
        const uint32_t x = t >> lT;
        uu[idx] = (x << lvpt) | (qv[idx] >> 16);
        if (adaptive && ld_plain<PERSIST>(rows_cur + x) == 0) vmask &= ~(1u << idx);
      }
    }
  }
  uint32_t amask = vmask;
  if (adaptive && !full_row) {
    uint32_t fw[EPT];
#pragma unroll
    for (int idx = 0; idx < EPT; ++idx) fw[idx] = ((vmask >> idx) & 1u) ? ld_state<PERSIST>(fa + (uu[idx] >> 5)) : 0u;
    amask = 0;
#pragma unroll
    for (int idx = 0; idx < EPT; ++idx) amask |= ((fw[idx] >> (uu[idx] & 31)) & 1u) << idx;
    amask &= vmask;
  }
  if (amask) {
    uint32_t cand[EPT], vv[EPT];
#pragma unroll
    for (int idx = 0; idx < EPT; ++idx) cand[idx] = ((amask >> idx) & 1u) ? ld_src<PERSIST>(jd, async, uu[idx]) : kInf;
    if (two_tiles) {
      const uint32_t yb0 = (tf & ymask) << lvpt, yb1 = (ta & ymask) << lvpt;
#pragma unroll
      for (int idx = 0; idx < EPT; ++idx)
        vv[idx] = (threadIdx.x + (uint32_t)idx * SG_T < cut ? yb0 : yb1) | (qv[idx] & 0xFFFFu);
    } else {
      // target tiles of the edges with an active source
#pragma unroll
      for (int idx = 0; idx < EPT; ++idx) {
        vv[idx] = 0;
        if ((amask >> idx) & 1u) {
          const uint32_t t = edge_tile(chunk_tile, tile_ptr, e0 + threadIdx.x + (uint32_t)idx * SG_T);
          vv[idx] = ((t & ymask) << lvpt) | (qv[idx] & 0xFFFFu);
        }
      }
    }
#pragma unroll
    for (int idx = 0; idx < EPT; ++idx)
      if (cand[idx] != kInf) cand[idx] = mp_cand<ALGO>(cand[idx], ww[idx]);
    uint32_t nv[EPT];
#pragma unroll
    for (int idx = 0; idx < EPT; ++idx) nv[idx] = (cand[idx] != kInf) ? ld_next(next + vv[idx]) : 0u;
#pragma unroll
    for (int idx = 0; idx < EPT; ++idx)
      if (cand[idx] != kInf && cand[idx] < nv[idx]) atomicMin(next + vv[idx], cand[idx]);
#pragma unroll
    for (int idx = 0; idx < EPT; ++idx)
      if (cand[idx] != kInf && cand[idx] < nv[idx]) atomicOr(ch + (vv[idx] >> 5), 1u << (vv[idx] & 31));
  }
}

// Whether stage st holds an edge of an active tile row (adaptive scheduling).
template <int PERSIST, int EPT = 16>
__device__ __forceinline__ bool stage_active(const JobDesc* __restrict__ jd, const StoreDesc* __restrict__ sd,
                                             uint64_t st, unsigned p, int adaptive) {
  if (!adaptive) return true;
  const unsigned* rows_cur = jd->rows + p * sd->T;
  const uint64_t nchunks = sd->nchunks;
  constexpr uint32_t SE = SG_T * EPT;
  const uint64_t c0 = st * (SE / kChunk);
  uint64_t c1 = c0 + SE / kChunk;
  if (c1 > nchunks) c1 = nchunks;
  const uint32_t x0 = sd->chunk_tile[c0] >> sd->lT;
  const uint32_t x1 = sd->chunk_tile[c1] >> sd->lT;
  for (uint32_t x = x0; x <= x1; ++x)
    if (ld_plain<PERSIST>(rows_cur + x)) return true;
  return false;
}

// ---- sparse gather -------------------------------------------------------
// Sparse gather: the round restricted to the edges of the listed non-zero frontier
// words. Work item = (frontier word, tile column y); the source directory gives the
// item's edge range inside tile (x, y), x being the word's tile row. A warp takes 32
// items that its words' column masks leave and walks the light items' edges with
// all 32 lanes. Items longer than SP_HEAVY edges, and, when the 32 items of a warp hold
// more than SP_WARP_MAX (SP_BLOCK_MAX where a block shares a list) edges in total, every
// item longer than SP_LIGHT, are cut into SP_CHUNK-edge chunks queued for the chunk pass, so
// no warp is left with more than about that many edges of light items or one chunk per queue
// entry (RMAT hub blocks).
//
// What bounds such a round is the serial chain of its busiest warp, each link an L2 access,
// and was the work done for items that hold nothing: in an RMAT-22 stream 1 to 12 % of (word,
// column) pairs are live, and walking them all took 39 M warp instructions and 100 us where
// 163,000 live items hold 3.3 M edges; numbered through they take 6 M and 44 us, and the
// stream 70.5 -> 60.0 ms. (Live items dealt out by whole words, a warp each: 80 us, a hub's
// 64 items in one warp.) SP_BLOCK_MAX 1024: 61.9 ms, 256: 60.3.
constexpr uint32_t SP_HEAVY = 2048;
constexpr uint32_t SP_CHUNK = 256;
constexpr uint32_t SP_LIGHT = 32;
constexpr uint32_t SP_WARP_MAX = 2048;
constexpr uint32_t SP_BLOCK_MAX = 512;
// Every light item is first narrowed to the edges of its word's active sources
// (sp_narrow). Streaming RMAT-22 by the shortest item narrowed: none 307.6 GTEPS, 64
// edges 313.8, 16 edges 326.7, 4 edges 326-329, every item 335.7. Items up to SP_HEAVY are
// narrowed before they may be queued: 256 edges 61.7 ms for the stream, 512 60.6, 1,024 60.3,
// 2,048 and 8,192 60.0.
constexpr uint32_t SP_NARROW = 0;
constexpr int SP_ILP = 8;   // edges per lane and step of a chunk
constexpr int SP_WILP = 4;  // of a batch of light items (8 and 6: within noise or slower)
constexpr int SP_TAIL = 2;  // steps of a batch's last edges

struct SpItem {
  uint32_t x, y, bits, lo, hi, b;  // b: the word's 32-source block in its tile row
  unsigned long long base;
};

// Item (word w, tile column y): its directory range and tile base.
__device__ __forceinline__ void sp_item_at(const StoreDesc* __restrict__ sd, uint32_t w, uint32_t y, SpItem& r) {
  const uint32_t lT = sd->lT, lnbw = sd->lvpt - 5, nbw = sd->nbw;
  r.y = y;
  r.x = w >> lnbw;
  const uint32_t b = w & (nbw - 1);
  r.b = b;
  const uint64_t dbase = (((uint64_t)r.x << lT) + r.y) * (nbw + 1) + b;
  r.lo = sd->dir[dbase];
  r.hi = sd->dir[dbase + 1];
  r.base = sd->tile_ptr[((uint64_t)r.x << lT) | r.y];
}

template <int PERSIST>
__device__ __forceinline__ SpItem sp_item(const JobDesc* __restrict__ jd, const StoreDesc* __restrict__ sd,
                                          uint64_t it) {
  const uint32_t w = ld_plain<PERSIST>(jd->aw + (it >> sd->lT));
  SpItem r;
  r.bits = ld_state<PERSIST>(jd->fa + w);
  sp_item_at(sd, w, (uint32_t)(it & (sd->T - 1)), r);
  return r;
}

// Relaxes ILP edges per lane whose sources are in their item's frontier word (xy: the item's
// tile, row << 16 | column; a directory exists for up to 2^14 tiles a side only); the
// loads of all ILP edges are issued before any of them is used.
// LAT: a target's value is loaded beside the source's, for every edge with an active source
// (one dependent step less, 53.9 -> 52.7 ms for an RMAT-22 stream; otherwise only for edges
// that offer a value).
template <int ALGO, int PERSIST, int ILP, bool LAT = false>
__device__ __forceinline__ void sp_batch(const JobDesc* __restrict__ jd, const StoreDesc* __restrict__ sd,
                                         const uint32_t (&xy)[ILP], const uint32_t (&bits)[ILP],
                                         const unsigned long long (&pos)[ILP], uint32_t valid) {
  const uint32_t lvpt = sd->lvpt;
  const bool async = jd->async != 0;
  uint32_t pk[ILP], wv[ILP], cand[ILP], nv[ILP];
#pragma unroll
  for (int k = 0; k < ILP; ++k) pk[k] = ((valid >> k) & 1u) ? sd->edges[pos[k]] : 0u;
  // the weight is read only for an edge whose source is in the frontier, beside its
  // source value (one dependent step, as before; most listed edges have inactive sources)
#pragma unroll
  for (int k = 0; k < ILP; ++k) {
    const uint32_t sl = pk[k] >> 16;
    const bool act = ((valid >> k) & 1u) && ((bits[k] >> (sl & 31)) & 1u);
    cand[k] = act ? ld_src<PERSIST>(jd, async, ((xy[k] >> 16) << lvpt) | sl) : kInf;
    wv[k] = (mp_weighted<ALGO>() && act) ? sd->wts[pos[k]] : 0u;
    if (LAT) nv[k] = act ? ld_next(jd->next + (((xy[k] & 0xFFFFu) << lvpt) | (pk[k] & 0xFFFFu))) : 0u;
  }
#pragma unroll
  for (int k = 0; k < ILP; ++k)
    if (cand[k] != kInf) cand[k] = mp_cand<ALGO>(cand[k], wv[k]);
#pragma unroll
  for (int k = 0; k < ILP && !LAT; ++k)
    nv[k] = (cand[k] != kInf) ? ld_next(jd->next + (((xy[k] & 0xFFFFu) << lvpt) | (pk[k] & 0xFFFFu))) : 0u;
#pragma unroll
  for (int k = 0; k < ILP; ++k) {
    if (cand[k] != kInf && cand[k] < nv[k]) {
      const uint32_t v = ((xy[k] & 0xFFFFu) << lvpt) | (pk[k] & 0xFFFFu);
      atomicMin(jd->next + v, cand[k]);
      atomicOr(jd->ch + (v >> 5), 1u << (v & 31));
    }
  }
}

// Narrows item m to the edges whose sources lie between the lowest and the highest
// active source of its word: an item's edges are sorted by (source, target) and packed
// as source << 16 | target, so two lower-bound searches (run side by side) on
// (source << 16) find the span. Sources outside it are inactive; their edges would only
// be read and dropped.
__device__ __forceinline__ void sp_narrow(const StoreDesc* __restrict__ sd, SpItem& m) {
  const uint32_t smin = (m.b << 5) + (uint32_t)(__ffs(m.bits) - 1);
  const uint32_t smax = (m.b << 5) + (31u - (uint32_t)__clz(m.bits));
  const uint32_t klo = smin << 16;
  const bool top = smax == 0xFFFFu;  // the tile's last source: the span runs to the end
  const uint32_t khi = top ? 0u : (smax + 1u) << 16;
  const uint32_t* e = sd->edges + m.base;
  uint32_t a0 = m.lo, a1 = m.hi, c0 = m.lo, c1 = top ? m.lo : m.hi;
  while (a0 < a1 || c0 < c1) {
    const uint32_t ma = (a0 + a1) >> 1, mc = (c0 + c1) >> 1;
    const uint32_t va = a0 < a1 ? e[ma] : 0u;
    const uint32_t vc = c0 < c1 ? e[mc] : 0u;
    if (a0 < a1) {
      if (va < klo) a0 = ma + 1;
      else a1 = ma;
    }
    if (c0 < c1) {
      if (vc < khi) c0 = mc + 1;
      else c1 = mc;
    }
  }
  m.lo = a0;
  m.hi = top ? m.hi : c0;
}

// sp_narrow with seven probes of each search per step: a third of the dependent loads, for
// rounds whose time is their latency.
__device__ __forceinline__ void sp_narrow_wide(const StoreDesc* __restrict__ sd, SpItem& m) {
  const uint32_t smin = (m.b << 5) + (uint32_t)(__ffs(m.bits) - 1);
  const uint32_t smax = (m.b << 5) + (31u - (uint32_t)__clz(m.bits));
  const uint32_t klo = smin << 16;
  const bool top = smax == 0xFFFFu;
  const uint32_t khi = top ? 0u : (smax + 1u) << 16;
  const uint32_t* e = sd->edges + m.base;
  uint32_t a0 = m.lo, a1 = m.hi, c0 = m.lo, c1 = top ? m.lo : m.hi;
  while (a0 < a1 || c0 < c1) {
    const uint32_t la = a1 - a0, lc = c1 - c0;
    uint32_t va[7], vc[7];
#pragma unroll
    for (int k = 0; k < 7; ++k) {
      va[k] = la ? e[a0 + ((la * (uint32_t)(k + 1)) >> 3)] : 0u;
      vc[k] = lc ? e[c0 + ((lc * (uint32_t)(k + 1)) >> 3)] : 0u;
    }
    // the probes ascend: the span after the last one below the key, up to the first at or above it
    uint32_t na = 0, nc = 0;
#pragma unroll
    for (int k = 0; k < 7; ++k) {
      na += va[k] < klo ? 1u : 0u;
      nc += vc[k] < khi ? 1u : 0u;
    }
    if (la) {
      const uint32_t b = a0;
      if (na < 7) a1 = b + ((la * (na + 1)) >> 3);
      if (na > 0) a0 = b + ((la * na) >> 3) + 1;
    }
    if (lc) {
      const uint32_t b = c0;
      if (nc < 7) c1 = b + ((lc * (nc + 1)) >> 3);
      if (nc > 0) c0 = b + ((lc * nc) >> 3) + 1;
    }
  }
  m.lo = a0;
  m.hi = top ? m.hi : c0;
}

// Position of the r-th set bit of m (r < its set bits).
__device__ __forceinline__ uint32_t nth_bit(unsigned long long m, uint32_t r) {
  uint32_t lo = (uint32_t)m, pos = 0;
  const uint32_t c0 = (uint32_t)__popc(lo);
  if (r >= c0) {
    r -= c0;
    lo = (uint32_t)(m >> 32);
    pos = 32;
  }
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) {
    const uint32_t c = (uint32_t)__popc(lo & ((1u << s) - 1u));
    if (r >= c) {
      r -= c;
      lo >>= s;
      pos += s;
    }
  }
  return pos;
}

// Lane whose run holds element f: the least j with incl[j] > f (incl: the lanes' inclusive
// prefix sums).
__device__ __forceinline__ uint32_t lane_of(uint32_t incl, uint32_t f) {
  uint32_t j = 0;
#pragma unroll
  for (int step = 16; step > 0; step >>= 1) {
    const uint32_t probe = __shfl_sync(0xFFFFFFFFu, incl, j + step - 1);
    if (probe <= f) j += step;
  }
  return j;
}
__device__ __forceinline__ uint32_t warp_incl_scan(uint32_t v) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, v, o);
    if ((threadIdx.x & 31) >= (unsigned)o) v += y;
  }
  return v;
}

// Light edges [f0, f0 + 32 ILP) of a batch of items, one item per lane: the batch's edges are
// numbered 0..total-1 by `incl`, the prefix sums of the items' lengths `mine`.
template <int ALGO, int PERSIST, int ILP, bool LAT>
__device__ __forceinline__ void sp_light(const JobDesc* __restrict__ jd, const StoreDesc* __restrict__ sd,
                                         const SpItem& m, uint32_t incl, uint32_t mine, uint32_t f0, uint32_t total) {
  const uint32_t mxy = (m.x << 16) | m.y;
  const unsigned long long first = m.base + m.lo - (incl - mine);  // of edge number 0
  uint32_t xy[ILP], bits[ILP];
  unsigned long long pos[ILP];
  uint32_t valid = 0;
#pragma unroll
  for (int k = 0; k < ILP; ++k) {
    const uint32_t f = f0 + (threadIdx.x & 31) + 32u * k;
    const uint32_t j = lane_of(incl, f);
    xy[k] = __shfl_sync(0xFFFFFFFFu, mxy, j);
    bits[k] = __shfl_sync(0xFFFFFFFFu, m.bits, j);
    pos[k] = __shfl_sync(0xFFFFFFFFu, first, j) + f;
    valid |= (f < total) ? (1u << k) : 0u;
  }
  sp_batch<ALGO, PERSIST, ILP, LAT>(jd, sd, xy, bits, pos, valid);
}

// Loads item (word w with frontier bits m.bits, tile column y) into m, narrowed if it is light.
template <bool WIDE>
__device__ __forceinline__ uint32_t sp_load(const StoreDesc* __restrict__ sd, uint32_t w, uint32_t y, SpItem& m) {
  sp_item_at(sd, w, y, m);
  uint32_t len = m.hi > m.lo ? m.hi - m.lo : 0u;
  if (len > SP_NARROW && len <= SP_HEAVY) {
    if (WIDE) sp_narrow_wide(sd, m);
    else sp_narrow(sd, m);
    len = m.hi > m.lo ? m.hi - m.lo : 0u;
  }
  return len;
}

// Walks a batch of up to 32 items, lane k's being m of len edges (0: none) with the number it;
// returns the light edges walked. Items of more than SP_HEAVY edges and, when the batch holds
// more than WMAX, those of more than SP_LIGHT, are queued for the chunk pass. nes warps share
// the batch: they deal out its light edges in steps of 32 * ILP; the first of them (es 0) alone
// queues the heavy items, and if the queue overflowed it walks every light edge of the batch
// itself (the others' share is then walked twice, which changes nothing).
template <int ALGO, int PERSIST, int ILP, uint32_t WMAX, bool LAT>
__device__ __forceinline__ uint32_t sp_walk(const JobDesc* __restrict__ jd, const StoreDesc* __restrict__ sd,
                                            const SpItem& m, uint32_t len, uint32_t it, uint32_t es, uint32_t nes) {
  uint32_t tot = len;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) tot += __shfl_xor_sync(0xFFFFFFFFu, tot, o);
  const bool heavy = len > SP_HEAVY || (tot > WMAX && len > SP_LIGHT);
  bool queued = heavy && es != 0;  // the first warp queues; the others leave those items to it
  bool overflow = false;
  if (heavy && es == 0) {
    const uint32_t nch = (len + SP_CHUNK - 1) / SP_CHUNK;
    const unsigned slot = atomicAdd(&jd->ls->spq_count, nch);
    if ((uint64_t)slot + nch <= jd->spq_cap) {
      for (uint32_t k = 0; k < nch; ++k) jd->spq[slot + k] = make_uint2(it, k);
      queued = true;
    } else {
      overflow = true;
    }
  }
  const bool walk_all = nes > 1 && es == 0 && __any_sync(0xFFFFFFFFu, overflow);
  const uint32_t mine = (len > 0 && !queued) ? len : 0u;
  const uint32_t incl = warp_incl_scan(mine);
  const uint32_t total = __shfl_sync(0xFFFFFFFFu, incl, 31);
  const uint32_t step0 = walk_all ? 0u : es, nstep = walk_all ? 1u : nes;
  for (uint32_t f0 = step0 * 32 * ILP; f0 < total; f0 += nstep * 32 * ILP) {
    if (total - f0 <= 32 * SP_TAIL) sp_light<ALGO, PERSIST, SP_TAIL, LAT>(jd, sd, m, incl, mine, f0, total);
    else sp_light<ALGO, PERSIST, ILP, LAT>(jd, sd, m, incl, mine, f0, total);
  }
  return es == 0 ? mine : 0u;
}

// Column mask of list entry e, as a number of items: bits of columns, times the columns of a bit.
template <int PERSIST>
__device__ __forceinline__ unsigned long long sp_columns(const JobDesc* __restrict__ jd,
                                                         const StoreDesc* __restrict__ sd, uint32_t e) {
  const unsigned long long cols = ld_plain<PERSIST>(jd->awm + e);
  return sd->lT < 6 ? cols & ((1ULL << (1u << sd->lT)) - 1ULL) : cols;
}
// Column of item r of an entry.
__device__ __forceinline__ uint32_t sp_column(unsigned long long cols, uint32_t r, uint32_t cshift) {
  return (nth_bit(cols, r >> cshift) << cshift) | (r & ((1u << cshift) - 1u));
}

// The frontier list of a round is walked by items (word, tile column), and an item is taken up
// only where the word's column mask says that an active source may have edges there: in late
// rounds of a stream a word reaches 1 to 8 of 64 columns, hubs' words all. The live items
// of a share of the list are numbered through and warps take them 32 at a time, one per lane.
//
// sparse_words: up to 32 entries e0 + k estep, k < ne, for the calling warp, or for nslice warps
// that share them: these deal out the batches of 32 items, and the light edges of a batch
// where there are fewer batches than warps. Returns the light edges walked and adds the
// items whose directory entries it read to `nread`.
template <int ALGO, int PERSIST, int ILP = SP_WILP, bool WIDE = false>
__device__ __forceinline__ uint32_t sparse_words(const JobDesc* __restrict__ jd, const StoreDesc* __restrict__ sd,
                                                 uint32_t e0, uint32_t estep, uint32_t ne, uint32_t& nread,
                                                 uint32_t slice = 0, uint32_t nslice = 1) {
  const unsigned lane = threadIdx.x & 31;
  const uint32_t cshift = sd->cshift;
  uint32_t w = 0, wbits = 0, ni = 0;
  unsigned long long cols = 0;
  if (lane < ne) {
    const uint32_t e = e0 + lane * estep;
    w = ld_plain<PERSIST>(jd->aw + e);
    cols = sp_columns<PERSIST>(jd, sd, e);
    wbits = ld_state<PERSIST>(jd->fa + w);
    ni = (uint32_t)__popcll(cols) << cshift;
  }
  const uint32_t iincl = warp_incl_scan(ni);
  const uint32_t nitems = __shfl_sync(0xFFFFFFFFu, iincl, 31);
  uint32_t nb = 1;  // batches that run side by side, each with nslice / nb slices
  while (nb < nslice && nb * 32 < nitems) nb *= 2;
  const uint32_t es = slice / nb, nes = nslice / nb;
  uint32_t walked = 0;
  for (uint32_t i0 = (slice % nb) * 32; i0 < nitems; i0 += nb * 32) {
    const uint32_t f = i0 + lane;
    const uint32_t j = lane_of(iincl, f);
    const uint32_t r = f - __shfl_sync(0xFFFFFFFFu, iincl - ni, j);
    const unsigned long long cj = __shfl_sync(0xFFFFFFFFu, cols, j);
    const uint32_t wj = __shfl_sync(0xFFFFFFFFu, w, j);
    SpItem m{};
    m.bits = __shfl_sync(0xFFFFFFFFu, wbits, j);
    uint32_t len = 0;
    if (f < nitems) {
      nread += es == 0 ? 1u : 0u;
      len = sp_load<WIDE>(sd, wj, sp_column(cj, r, cshift), m);
    }
    walked += sp_walk<ALGO, PERSIST, ILP, SP_WARP_MAX, WIDE>(jd, sd, m, len, ((e0 + j * estep) << sd->lT) | m.y, es,
                                                             nes);
  }
  return walked;
}

// Split of a list of nact entries over nwarps warps for sparse_words: `units` shares of at most
// 32 entries (entry e belongs to unit e % units, so that the hubs' words, which lie side by
// side, go to different warps); with few entries nslice warps on each.
__device__ __forceinline__ void sparse_split(uint32_t nact, uint32_t nwarps, uint32_t& units, uint32_t& nslice) {
  units = min(nact, max(nwarps, (nact + 31) / 32));
  nslice = 1;
  while (nslice < 8 && units * nslice * 2 <= nwarps) nslice *= 2;
}

// sparse_block: the same for up to NT entries and the calling block of NT threads, which share
// them all, so that a hub's 64 items don't keep one warp busy when the others are done.
template <int NT>
struct SparseList {
  unsigned long long cols[NT];
  uint32_t w[NT], bits[NT], incl[NT];  // incl: live items up to and with this entry
  uint32_t wsum[NT / 32];
};

template <int ALGO, int PERSIST, int NT, int ILP = SP_WILP>
__device__ __forceinline__ uint32_t sparse_block(const JobDesc* __restrict__ jd, const StoreDesc* __restrict__ sd,
                                                 SparseList<NT>& sl, uint32_t e0, uint32_t estep, uint32_t ne,
                                                 uint32_t& nread) {
  constexpr uint32_t NW = NT / 32;
  const unsigned tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t cshift = sd->cshift;
  uint32_t ni = 0;
  if (tid < ne) {
    const uint32_t e = e0 + tid * estep;
    const uint32_t w = ld_plain<PERSIST>(jd->aw + e);
    const unsigned long long cols = sp_columns<PERSIST>(jd, sd, e);
    ni = (uint32_t)__popcll(cols) << cshift;
    sl.w[tid] = w;
    sl.cols[tid] = cols;
    sl.bits[tid] = ld_state<PERSIST>(jd->fa + w);
  }
  uint32_t iincl = warp_incl_scan(ni);
  if (lane == 31) sl.wsum[warp] = iincl;
  __syncthreads();
  uint32_t nitems = 0;
#pragma unroll
  for (uint32_t k = 0; k < NW; ++k) {
    const uint32_t x = sl.wsum[k];
    iincl += k < warp ? x : 0u;
    nitems += x;
  }
  sl.incl[tid] = iincl;
  __syncthreads();
  uint32_t nb = 1;  // batches that run side by side, each by NW / nb warps
  while (nb < NW && nb * 32 < nitems) nb *= 2;
  const uint32_t es = warp / nb, nes = NW / nb;
  uint32_t walked = 0;
  for (uint32_t i0 = (warp % nb) * 32; i0 < nitems; i0 += nb * 32) {
    const uint32_t f = i0 + lane;
    SpItem m{};
    uint32_t len = 0, ent = 0;
    if (f < nitems) {
      nread += es == 0 ? 1u : 0u;
#pragma unroll
      for (uint32_t step = NT / 2; step > 0; step >>= 1)
        if (sl.incl[ent + step - 1] <= f) ent += step;
      const unsigned long long cols = sl.cols[ent];
      const uint32_t r = f - (sl.incl[ent] - ((uint32_t)__popcll(cols) << cshift));
      m.bits = sl.bits[ent];
      len = sp_load<false>(sd, sl.w[ent], sp_column(cols, r, cshift), m);
    }
    walked += sp_walk<ALGO, PERSIST, ILP, SP_BLOCK_MAX, true>(jd, sd, m, len,
                                                               ((e0 + ent * estep) << sd->lT) | m.y, es, nes);
  }
  return walked;
}

// Queue entry q (a chunk of a heavy item) for the calling warp; returns the edges walked
// (lane 0). Sources are sorted inside an item, so a chunk whose first and last edges
// span no source of the item's frontier word is skipped after two loads. (A skipped chunk of
// an item that its neighbours made heavy still counts as walked, so that the count does not
// hang on the order of the frontier list.)
template <int ALGO, int PERSIST>
__device__ __forceinline__ uint32_t sparse_chunk(const JobDesc* __restrict__ jd, const StoreDesc* __restrict__ sd,
                                                 uint64_t q, uint64_t items) {
  const unsigned lane = threadIdx.x & 31;
  const uint2 c = ld_plain<PERSIST>(jd->spq + q);
  if (c.x >= items) return 0;  // never indexes outside this round's items
  SpItem m = sp_item<PERSIST>(jd, sd, c.x);
  const bool own = m.hi > m.lo && m.hi - m.lo > SP_HEAVY;  // queued for its own length
  // the item as sp_walk cut it into chunks: narrowed by the same rule
  if (!own && m.hi > m.lo) sp_narrow(sd, m);
  const uint32_t e0 = m.lo + c.y * SP_CHUNK;
  const uint32_t e1 = min(m.hi, e0 + SP_CHUNK);
  if (e0 >= e1) return 0;
  uint32_t bound = 0;
  if (lane == 0) bound = sd->edges[m.base + e0];
  if (lane == 1) bound = sd->edges[m.base + e1 - 1];
  const uint32_t s_first = (__shfl_sync(0xFFFFFFFFu, bound, 0) >> 16) & 31u;
  const uint32_t s_last = (__shfl_sync(0xFFFFFFFFu, bound, 1) >> 16) & 31u;
  const uint32_t span = (s_last >= 31u ? 0xFFFFFFFFu : ((2u << s_last) - 1u)) & ~((1u << s_first) - 1u);
  if ((m.bits & span) == 0) return own || lane != 0 ? 0u : e1 - e0;
  uint32_t xy[SP_ILP], bits[SP_ILP];
#pragma unroll
  for (int k = 0; k < SP_ILP; ++k) {
    xy[k] = (m.x << 16) | m.y;
    bits[k] = m.bits;
  }
  for (uint32_t e = e0 + lane; e < e1; e += 32 * SP_ILP) {
    unsigned long long pos[SP_ILP];
    uint32_t valid = 0;
#pragma unroll
    for (int k = 0; k < SP_ILP; ++k) {
      const uint32_t ek = e + 32u * k;
      pos[k] = m.base + ek;
      valid |= (ek < e1) ? (1u << k) : 0u;
    }
    sp_batch<ALGO, PERSIST, SP_ILP>(jd, sd, xy, bits, pos, valid);
  }
  return lane == 0 ? e1 - e0 : 0u;
}

}  // namespace cytom
