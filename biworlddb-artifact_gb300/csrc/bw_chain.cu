// bw_chain.cu -- single-pass replay of a linear version chain (see bw_chain.cuh).
//
// Sweep (k_chain_sweep, one CTA per state block; 128-512 threads, tiles of 512-1024
// events, three tiles or two in shared memory, the geometry picked per workload by occupancy):
//   * the block's events (an equal share, or, where queries are many, such that events and
//     queries together are an equal share) stream through the ring, each tile one
//     cp.async.bulk copy from global memory into shared memory completed on the
//     stage's mbarrier (bounded waits);
//   * the running key histogram of the block is an exact int32 window H[key] in
//     shared memory (plus int32 totals of 32-key chunks when the key domain is
//     larger than 4,096 keys).  A window holds events whose absolute sum stays
//     below 2^28 + 2^29, so every partial sum of it is exact in int32; before it
//     can grow past that it is folded into the block's key prefix row in global
//     memory (P[k] = sum of the folded events below key k, int64).  Tiles holding a
//     delta outside (-2^19, 2^19) bypass the window: their events go to a per-block
//     int64 key histogram with global atomics, folded into P before the next tile;
//   * a tile owns the queries whose position (number of events at or before their
//     state) falls inside it: state < state of the tile's last event.  Their local
//     answer = P[hi] - P[lo] + the window over [lo, hi) before the tile is applied,
//     plus the tile's first `pos` events inside [lo, hi); one warp per query,
//     int32 lane sums reduced with redux.sync;
//   * one warp (the last) finds the next tile's queries and their positions while
//     the others answer the current tile's: the query records come through a
//     32-record window that cp.async fills one tile ahead, and land in a
//     double-buffered shared query buffer.
// Carry (k_chain_carry): exclusive column scan over the blocks' final prefix rows, in
// place: row b becomes the key prefix of the events of blocks 0 .. b-1.
// Fix-up (k_chain_fixup): every query of block b >= 1 adds row[hi] - row[lo].
#include <cuda_runtime.h>
#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <mutex>
#include <type_traits>

#include "bw_gpu.h"
#include "bw_common.cuh"
#include "bw_chain.cuh"

namespace bw {
namespace {

constexpr int TE = kChainTile;   // largest tile (the shared-memory ring is sized per geometry)
constexpr int QB = kChainQBuf;
constexpr int kMaxWarps = kChainThreads / 32;
constexpr int kChunkShift = 5;                   // chunk totals cover 32 keys each
constexpr uint32_t kFlatKeys = 4096;             // key domains up to this size keep no chunk totals
constexpr uint32_t kWaitLimit = 1u << 22;        // mbarrier polls before a stage is declared lost
// A query costs a sweep CTA about what 64 events do.  Where the queries outweigh the events
// the blocks are cut by both: a reference-native chain (300,000 states, an edit of 1,700 keys
// every 75th, two queries a state) had its queries in few of its equal event ranges (sweep
// 499 -> 318 us; 32 events a query 336, 128 315, 256 331), 6,636 states 96 -> 29 us.  Chains
// with both spread evenly pay the search of the cut, some 3 us; hence not below.
constexpr int32_t kQueryWeight = 64;
constexpr uint32_t kFoldAt = 1u << 28;           // window |delta| sum that triggers a fold
// A tile is int32-safe when every delta lies in (-2^19, 2^19): with at most 1024
// events its absolute sum is then below 2^29.

struct ChainParams {
  const uint4* ev;        // events as 16-byte records (state, key, delta lo, delta hi)
  const BwQuery* qs;
  int64_t* ans;
  const int32_t* parent;
  int64_t E, Q;
  int32_t S;
  uint32_t C;
  int32_t B;
  int32_t nch;
  int32_t qweight;        // events a query counts for in the cut of the blocks (0: events only)
  int64_t* rows;          // B rows of C+1 int64: key prefixes (row[k] = sum below key k)
  int64_t* wide;          // B rows of C int64: key histogram of the block's wide tiles
  int64_t* btab;          // B x (first query, end query)
  int32_t* status;
};

// Shared words written in one tile and read in the next are double-buffered by
// tile parity: a fast warp may already write the next tile's copy while a slow one
// still reads this tile's.
struct Misc {
  uint32_t wsum[2][kMaxWarps];   // per-warp |delta| sum of a tile's window updates
  int64_t tq[2][2];              // queries [tq0, tq1) of a tile
  int64_t tail_q0;
  unsigned long long scan[kMaxWarps];   // warp totals of the fold's key scan
};

// Dynamic shared memory of the sweep, every region 16-byte aligned.
struct SweepSmem {
  size_t ring, kd, st, H, T, qbuf, qpre, bar, misc, bytes;
};
__host__ __device__ inline size_t al16(size_t x) { return (x + 15) & ~size_t(15); }
// hw: bytes of a window entry (4: int32 window, 8: int64 window).  With the int32 window the
// current tile lies in its compact form, and the ring holds the ns - 1 tiles after it.
__host__ __device__ inline SweepSmem sweep_smem(uint32_t C, int nch, int te, int ns, int hw) {
  SweepSmem L;
  size_t o = 0;
  L.ring = o;  o = al16(o + (size_t)(hw == 4 ? ns - 1 : ns) * te * 16);
  L.kd = o;    o = al16(o + (hw == 4 ? (size_t)te * 8 : 0));
  L.st = o;    o = al16(o + (hw == 4 ? (size_t)te * 4 : 0));
  L.H = o;     o = al16(o + (size_t)C * hw);
  L.T = o;     o = al16(o + (size_t)nch * hw);
  L.qbuf = o;  o = al16(o + 2 * (size_t)QB * 16);   // two tiles' query records
  L.qpre = o;  o = al16(o + 32 * 12);                // prefetched window of 32 query records
  L.bar = o;   o = al16(o + (size_t)ns * 8);
  L.misc = o;  o = al16(o + sizeof(Misc));
  L.bytes = o;
  return L;
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}
// Bounded wait for phase `parity` of a stage barrier; false when it never completed.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
  const uint32_t a = smem_u32(bar);
  for (uint32_t i = 0; i < kWaitLimit; ++i) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(a), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return false;
}

__device__ __forceinline__ void set_status(int32_t* st, int32_t code) {
  if (*reinterpret_cast<volatile int32_t*>(st) == 0) atomicCAS(st, 0, code);
}

// delta in (-2^19, 2^19): its high word is the sign extension of its low word
__device__ __forceinline__ bool small_delta(const uint4& e) {
  const int32_t lo = (int32_t)e.z;
  return e.w == (uint32_t)(lo >> 31) && (uint32_t)(lo + (1 << 19)) < (1u << 20);
}

__device__ __forceinline__ uint64_t warp_sum_u64(uint64_t v) {
#pragma unroll
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Lane share of the window sum over keys [lo, hi) (lo < hi <= C): the partial
// chunks at either end from H (fewer than 32 keys each), the whole chunks from T.
__device__ __forceinline__ int32_t probe32(const int32_t* H, const int32_t* T, uint32_t lo, uint32_t hi, int lane) {
  const uint32_t clo = (lo + 31) >> kChunkShift, chi = hi >> kChunkShift;
  int32_t s = 0;
  if (clo >= chi) {   // fewer than 64 keys
    for (uint32_t k = lo + lane; k < hi; k += 32) s += H[k];
    return s;
  }
  const uint32_t a = lo + lane, z = (chi << kChunkShift) + lane;
  if (a < (clo << kChunkShift)) s += H[a];
  if (z < hi) s += H[z];
  for (uint32_t c = clo + lane; c < chi; c += 32) s += T[c];
  return s;
}

// Lane share of the window sum over keys [lo, hi) (lo < hi <= C) without chunk
// totals: 128-bit reads of H, four keys per lane, masked to the interval.  H is
// 16-byte aligned and padded to a multiple of four keys, so the last read stays in
// the region; padding keys fall outside [lo, hi).
__device__ __forceinline__ int32_t probe_flat(const int32_t* H, uint32_t lo, uint32_t hi, int lane) {
  const uint32_t w = hi - lo;
  int32_t s = 0;
#pragma unroll 2
  for (uint32_t k = (lo & ~3u) + 4 * lane; k < hi; k += 128) {
    const int4 v = *reinterpret_cast<const int4*>(H + k);
    const uint32_t d = k - lo;
    s += (d < w ? v.x : 0) + (d + 1 < w ? v.y : 0) + (d + 2 < w ? v.z : 0) + (d + 3 < w ? v.w : 0);
  }
  return s;
}

// The int64 window's counterparts: lane shares of the sum over [lo, hi) (lo < hi <= C)
// from 32-key chunk totals plus the partial chunks, or flat 128-bit reads of two
// keys each (H 16-byte aligned and padded to an even key count).
__device__ __forceinline__ uint64_t probe_chunks64(const unsigned long long* H, const unsigned long long* T,
                                                   uint32_t lo, uint32_t hi, int lane) {
  const uint32_t clo = (lo + 31) >> kChunkShift, chi = hi >> kChunkShift;
  uint64_t s = 0;
  if (clo >= chi) {
    for (uint32_t k = lo + lane; k < hi; k += 32) s += H[k];
    return s;
  }
  const uint32_t a = lo + lane, z = (chi << kChunkShift) + lane;
  if (a < (clo << kChunkShift)) s += H[a];
  if (z < hi) s += H[z];
  for (uint32_t c = clo + lane; c < chi; c += 32) s += T[c];
  return s;
}
__device__ __forceinline__ uint64_t probe_flat64(const unsigned long long* H, uint32_t lo, uint32_t hi, int lane) {
  const uint32_t w = hi - lo;
  uint64_t s = 0;
#pragma unroll 2
  for (uint32_t k = (lo & ~1u) + 2 * lane; k < hi; k += 64) {
    const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(H + k);
    const uint32_t d = k - lo;
    s += (d < w ? v.x : 0ull) + (d + 1 < w ? v.y : 0ull);
  }
  return s;
}

// Position of a query in its tile: the number of the tile's events at or before
// its state (upper bound over the tile's sorted states).
__device__ __forceinline__ uint32_t state_of(const uint4& e) { return e.x; }
__device__ __forceinline__ uint32_t state_of(uint32_t s) { return s; }
template <typename R>
__device__ __forceinline__ uint32_t tile_pos(const R* tile, int n, uint32_t qst) {
  uint32_t lo = 0, hi = (uint32_t)n;
  while (lo < hi) {
    const uint32_t mid = (lo + hi) >> 1;
    if (state_of(tile[mid]) <= qst) lo = mid + 1; else hi = mid;
  }
  return lo;
}

// First query index in [0, Q) whose state is >= x (Q when none), found by the
// whole CTA in rounds of one probe per thread.
__device__ int64_t first_query_at_or_after(const BwQuery* qs, int64_t Q, uint32_t x) {
  const int nt = blockDim.x;
  int64_t lo = 0, hi = Q;
  while (true) {
    const int64_t n = hi - lo;
    if (n <= 0) return lo;
    const int64_t step = (n + nt - 1) / nt;
    const int64_t pos = lo + (int64_t)threadIdx.x * step;
    const bool lt = pos < hi && qs[pos].state < x;
    const int cnt = __syncthreads_count(lt);
    if (step == 1) return lo + cnt;
    const int64_t nlo = cnt ? lo + (int64_t)(cnt - 1) * step + 1 : lo;
    hi = min(hi, lo + (int64_t)cnt * step);
    lo = nlo;
  }
}

// Events [e[0], e[1]) of block b where a query counts for p.qweight events: the points where
// the walk through events and queries in state order (an event before the queries of its
// state) has done b and b + 1 shares of the work.  Found on those diagonals by the whole
// CTA, one probe of each per thread and round; ascending in b for sorted input, inside
// [0, E] for any (so every event is in some block even then).
__device__ void weighted_cut(const ChainParams& p, int64_t b, int64_t (&e)[2]) {
  const int64_t K = p.qweight, nt = blockDim.x;
  // queries after the last event belong to the last block whatever the cut, and cost it little: they are
  // left out where they are many (1M events, 441,437 queries all on the last state, 17 blocks: 1.14 ms, 3.75
  // with them counted, as the events then went into two blocks)
  int64_t Q = p.Q;
  const uint32_t end = p.ev[p.E - 1].x;
  if (p.qs[Q - 1 - Q / 16].state >= end) Q = first_query_at_or_after(p.qs, Q, end);
  const int64_t work = p.E + K * Q;
  int64_t target[2], hi[2];
  bool done[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    target[i] = work / p.B * (b + i) + work % p.B * (b + i) / p.B;
    e[i] = max((int64_t)0, target[i] - K * Q);
    hi[i] = min(target[i], p.E);
    done[i] = false;
  }
  while (!done[0] || !done[1]) {
    bool before[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int64_t pos = e[i] + (int64_t)threadIdx.x * ((hi[i] - e[i] + nt - 1) / nt);
      before[i] = false;
      if (pos < hi[i]) {
        const int64_t q = (target[i] - pos) / K;
        before[i] = q >= Q || p.ev[pos].x <= p.qs[q].state;
      }
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int cnt = __syncthreads_count(before[i]);
      const int64_t step = (hi[i] - e[i] + nt - 1) / nt;
      if (step == 1) {
        e[i] += cnt;
        hi[i] = e[i];
      } else if (step > 1) {
        const int64_t lo = cnt ? e[i] + (int64_t)(cnt - 1) * step + 1 : e[i];
        hi[i] = min(hi[i], e[i] + (int64_t)cnt * step);
        e[i] = lo;
      }
      done[i] = hi[i] <= e[i];
    }
  }
}

// First query index in [from, Q) whose state is >= x (Q when none), found by one warp:
// doubling steps, then 32 probes a round.
__device__ int64_t next_query_at_or_after(const BwQuery* qs, int64_t Q, int64_t from, uint32_t x, int lane) {
  int64_t pos = from + ((int64_t)32 << lane);
  uint32_t lt = __ballot_sync(0xffffffffu, pos < Q && qs[pos].state < x);
  int k = lt == 0xffffffffu ? 32 : __ffs(~lt) - 1;
  int64_t lo = k ? from + ((int64_t)32 << (k - 1)) + 1 : from;
  int64_t hi = k < 32 ? min(Q, from + ((int64_t)32 << k)) : Q;
  while (hi > lo) {
    const int64_t step = (hi - lo + 31) / 32;
    pos = lo + lane * step;
    k = __popc(__ballot_sync(0xffffffffu, pos < hi && qs[pos].state < x));
    if (step == 1) return lo + k;
    const int64_t nlo = k ? lo + (k - 1) * step + 1 : lo;
    hi = min(hi, lo + k * step);
    lo = nlo;
  }
  return lo;
}

// The query warp's window of the next 32 query records, copied into shared memory
// with cp.async one tile before it is read (so the copy's latency stays hidden).
__device__ __forceinline__ void qpre_issue(uint32_t* qpre, const BwQuery* qs, int64_t Q, int64_t base, int lane) {
  const int64_t i = base + lane;
  if (i < Q) {
    const uint32_t* src = reinterpret_cast<const uint32_t*>(qs + i);
#pragma unroll
    for (int j = 0; j < 3; ++j)
      asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(qpre + 3 * lane + j)), "l"(src + j)
                   : "memory");
  } else {
    qpre[3 * lane] = 0xffffffffu;   // past the last query
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
}

// Query warp: the queries of a tile (n events, the last with state x) are those
// from qcur on with state < x.  Their records and positions in the tile go to qbuf
// (the first QB), their range to tq; qcur advances past them.  `pbase` is the first
// query of the window in flight.
__device__ void find_tile_queries(const ChainParams& p, uint32_t* qpre, int64_t& pbase, int64_t& qcur,
                                  const uint4* tile, int n, uint32_t* qbuf, int64_t* tq, int lane) {
  const uint32_t x = tile[n - 1].x;
  const int64_t tq0 = qcur;
  while (true) {
    if (pbase != qcur) {
      qpre_issue(qpre, p.qs, p.Q, qcur, lane);
      pbase = qcur;
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    const uint32_t st = qpre[3 * lane], lo = qpre[3 * lane + 1], hi = qpre[3 * lane + 2];
    const bool valid = qcur + lane < p.Q;
    const uint32_t ball = __ballot_sync(0xffffffffu, valid && st < x);
    const int k = ball == 0xffffffffu ? 32 : __ffs(~ball) - 1;
    if (lane < k) {
      const int64_t slot = qcur - tq0 + lane;
      if (slot < QB) {
        uint4 r;
        r.x = st;
        r.y = lo;
        r.z = hi;
        r.w = tile_pos(tile, n, st);
        reinterpret_cast<uint4*>(qbuf)[slot] = r;
      }
    }
    __syncwarp();   // every lane has read the window before it is refilled
    qcur += k;
    if (k < 32) break;
    if (qcur - tq0 >= QB) {   // no more records are staged: only the end is asked for
      qcur = next_query_at_or_after(p.qs, p.Q, qcur, x, lane);
      break;
    }
  }
  if (lane == 0) {
    tq[0] = tq0;
    tq[1] = qcur;
  }
  qpre_issue(qpre, p.qs, p.Q, qcur, lane);   // read at the next tile
  pbase = qcur;
}

// The same with the int64 window (no folded row: it only fills at the end).
__device__ __forceinline__ int64_t answer_one64(const ChainParams& p, const unsigned long long* H,
                                                const unsigned long long* T, const uint4* tile, uint32_t pos,
                                                uint32_t lo, uint32_t hi, int lane) {
  lo = min(lo, p.C);
  hi = min(hi, p.C);
  if (lo >= hi) return 0;
  const uint32_t w = hi - lo;
  uint64_t part = p.nch ? probe_chunks64(H, T, lo, hi, lane) : probe_flat64(H, lo, hi, lane);
#pragma unroll 4
  for (uint32_t j = lane; j < pos; j += 32) {
    const uint4 e = tile[j];
    if (e.y - lo < w) part += ((uint64_t)e.w << 32) | e.z;
  }
  return (int64_t)warp_sum_u64(part);
}

// Answer of one query by one warp, valid in lane 0: the folded key prefix row
// (P[hi] - P[lo], when it holds data), the window probe, and the tile's first `pos` events
// inside [lo, hi): from the compact tile, two (key, delta) pairs a lane and read; those of
// a wide tile, whose deltas do not fit it, from global memory.
__device__ __forceinline__ int64_t answer_one(const ChainParams& p, const int32_t* H, const int32_t* T,
                                              const int64_t* P, bool rows_live, const uint2* kd, const uint4* wide_tile,
                                              uint32_t pos, uint32_t lo, uint32_t hi, int lane) {
  lo = min(lo, p.C);
  hi = min(hi, p.C);
  if (lo >= hi) return 0;
  const uint32_t w = hi - lo;
  uint64_t pv = 0;
  if (rows_live && lane < 2) pv = (uint64_t)__ldcg(P + (lane ? hi : lo));   // both ends in flight at once
  int32_t part = p.nch ? probe32(H, T, lo, hi, lane) : probe_flat(H, lo, hi, lane);
  uint64_t wide = 0;
  if (wide_tile) {
    for (uint32_t j = lane; j < pos; j += 32) {
      const uint4 e = wide_tile[j];
      if (e.y - lo < w) wide += ((uint64_t)e.w << 32) | e.z;
    }
  } else {
#pragma unroll 4
    for (uint32_t j = 2 * lane; j < pos; j += 64) {
      const uint4 e = *reinterpret_cast<const uint4*>(kd + j);   // (key, delta) of events j and j + 1
      if (e.x - lo < w) part += (int32_t)e.y;
      if (j + 1 < pos && e.z - lo < w) part += (int32_t)e.w;
    }
  }
  uint64_t total = (uint64_t)(int64_t)(int32_t)__reduce_add_sync(0xffffffffu, (uint32_t)part);
  if (wide_tile) total += warp_sum_u64(wide);
  const uint64_t phi = __shfl_down_sync(0xffffffffu, pv, 1);
  return (int64_t)(total + phi - pv);
}

// Fold of the window (and of the wide tiles' histogram) into the block's key
// prefix row: P[k+1] += sum of H[j] + wide[j] over j <= k.  Each thread takes a
// contiguous key segment; a CTA-wide exclusive scan of the segment sums gives its
// base.  H, T and the consumed wide entries return to zero.  All threads call it.
template <int NT, typename HT>
__device__ void fold(const ChainParams& p, HT* H, HT* T, int64_t* P, int64_t* wide, bool rows_live,
                     bool wide_live, Misc* m) {
  constexpr int NW = NT / 32;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t C = p.C, per = (C + NT - 1) / NT;
  const uint32_t k0 = min(C, (uint32_t)tid * per), k1 = min(C, k0 + per);
  uint64_t s = 0;
  for (uint32_t k = k0; k < k1; ++k) {
    s += (uint64_t)(int64_t)H[k];   // sign-extends an int32 window entry
    if (wide_live) s += (uint64_t)__ldcg(wide + k);
  }
  uint64_t incl = s;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint64_t t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) m->scan[warp] = incl;
  __syncthreads();
  uint64_t run = incl - s;
#pragma unroll
  for (int w = 0; w < NW; ++w)
    if (w < warp) run += m->scan[w];
  for (uint32_t k = k0; k < k1; ++k) {
    run += (uint64_t)(int64_t)H[k];
    H[k] = 0;
    if (wide_live) {
      run += (uint64_t)__ldcg(wide + k);
      wide[k] = 0;
    }
    P[k + 1] = rows_live ? (int64_t)((uint64_t)__ldcg(P + k + 1) + run) : (int64_t)run;
  }
  if (tid == 0 && !rows_live) P[0] = 0;
  for (int c = tid; c < p.nch; c += NT) T[c] = 0;
  __syncthreads();
}

// Tile geometry: NT threads, EPT events per thread, TL = NT * EPT events per tile
// (<= 1024, so an int32-safe tile's absolute sum stays below 2^29); MINB CTAs per SM;
// NS tiles in the shared-memory ring.  W64: the window is int64 (two 32-bit shared
// atomics per update, exact modulo 2^64 at any delta size): no window folds, no wide
// tiles -- the mode for chains whose deltas mostly exceed the int32-safe range.
template <int NT, int EPT, int MINB, int NS, bool W64>
__global__ void __launch_bounds__(NT, MINB) k_chain_sweep(ChainParams p) {
  constexpr int NW = NT / 32, QW = NW - 1, TL = NT * EPT;
  // int32 window: every tile is copied into its compact form when its events are loaded,
  // which frees its place in the ring a tile earlier and halves what a query's scan reads (the
  // shared-memory pipe and issue bound the sweep: 100M events, 1M queries 893 -> 859 us; 20M
  // events, 2M queries 922 -> 789)
  constexpr bool kCompact = !W64;
  constexpr int RS = kCompact ? NS - 1 : NS;
  chain_wait();
  static_assert(TL <= TE && NW <= kMaxWarps && NW >= 2, "tile geometry");
  extern __shared__ __align__(128) unsigned char sm[];
  const uint32_t C = p.C;
  using HT = typename std::conditional<W64, unsigned long long, int32_t>::type;
  const SweepSmem SL = sweep_smem(C, p.nch, TL, NS, (int)sizeof(HT));
  uint4* ring = reinterpret_cast<uint4*>(sm + SL.ring);
  uint2* kd = reinterpret_cast<uint2*>(sm + SL.kd);          // the tile's (key, delta)
  uint32_t* kst = reinterpret_cast<uint32_t*>(sm + SL.st);   // ... and states
  HT* H = reinterpret_cast<HT*>(sm + SL.H);
  HT* T = reinterpret_cast<HT*>(sm + SL.T);
  uint32_t* qbuf = reinterpret_cast<uint32_t*>(sm + SL.qbuf);   // [2][QB] uint4, by tile parity
  uint32_t* qpre = reinterpret_cast<uint32_t*>(sm + SL.qpre);
  uint64_t* bar = reinterpret_cast<uint64_t*>(sm + SL.bar);
  Misc* m = reinterpret_cast<Misc*>(sm + SL.misc);
  auto qbuf_of = [&](int t) { return qbuf + (size_t)(t & 1) * QB * 4; };

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int b = blockIdx.x;
  int64_t cut[2] = {(int64_t)b * p.E / p.B, (int64_t)(b + 1) * p.E / p.B};
  if (p.qweight) weighted_cut(p, b, cut);
  const int64_t e0 = cut[0], ne = cut[1] - cut[0];   // (no tile below 1)
  const int ntiles = ne > 0 ? (int)((ne + TL - 1) / TL) : 0;
  int64_t* P = p.rows + (int64_t)b * (C + 1);
  int64_t* wrow = p.wide + (int64_t)b * C;
  auto tile_n = [&](int t) { return (int)min((int64_t)TL, ne - (int64_t)t * TL); };

  for (uint32_t i = tid; i < C; i += NT) H[i] = 0;
  for (int i = tid; i < p.nch; i += NT) T[i] = 0;
  if (tid < 2 * kMaxWarps) m->wsum[tid / kMaxWarps][tid % kMaxWarps] = 0;
  if (tid == 0) {
    for (int s = 0; s < RS; ++s) mbar_init(&bar[s], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  int issued = 0;   // tiles whose copy was issued (thread 0)
  if (tid == 0) {
    for (; issued < RS && issued < ntiles; ++issued)
      bulk_load(ring + (issued % RS) * TL, p.ev + e0 + (int64_t)issued * TL, (uint32_t)tile_n(issued) * 16u,
                &bar[issued % RS]);
  }
  // input checks spread over every sweep thread: parent[v] = v - 1, and every query
  // (sorted by state, state and bounds in range) -- queries behind an out-of-order
  // one may never be reached by a tile, so they are checked here, not when consumed
  for (int64_t v = (int64_t)b * NT + tid; v < p.S; v += (int64_t)p.B * NT)
    if (p.parent[v] != (int32_t)(v - 1)) set_status(p.status, BW_STATUS_BAD_PARENT);
  for (int64_t i = (int64_t)b * NT + tid; i < p.Q; i += (int64_t)p.B * NT) {
    const uint32_t* r = reinterpret_cast<const uint32_t*>(p.qs + i);
    const uint32_t qst = r[0], lo = r[1], hi = r[2];
    if (i > 0 && qst < p.qs[i - 1].state) set_status(p.status, BW_STATUS_QUERIES_UNSORTED);
    if (qst >= (uint32_t)p.S) set_status(p.status, BW_STATUS_STATE_RANGE);
    if (lo > C || hi > C) set_status(p.status, BW_STATUS_QUERY_RANGE);
  }
  // the block's first query: position >= e0, i.e. state >= state of event e0 - 1
  uint32_t last = e0 > 0 ? p.ev[e0 - 1].x : 0u;   // state of the event before the tile to be loaded
  const int64_t qstart = e0 > 0 ? first_query_at_or_after(p.qs, p.Q, last) : 0;

  int64_t qcur = qstart, pbase = qstart;
  if (warp == QW) qpre_issue(qpre, p.qs, p.Q, qcur, lane);

  uint4 cur[EPT];
  bool rows_live = false;   // the prefix row holds data (set by the first fold)
  bool wide_init = false;   // the wide histogram row has been zeroed
  bool wide_live = false;   // a wide tile was applied since the last fold
  uint32_t win = 0;         // |delta| sum in the int32 window (the same in every thread)
  int bigp = 0, lost = 0;
  uint32_t bad = 0;         // event defects seen by this thread (reported at the end)
  // this thread's events of the tile in ring place `rt`: into registers and the compact
  // tile, with their order checked (the state before each comes from the previous lane;
  // lane 0 reads it from the tile, for the first event it is the last tile's)
  auto load_tile = [&](const uint4* rt, int n) -> int {
    int wide = 0;
#pragma unroll
    for (int k = 0; k < EPT; ++k) {
      const int idx = tid + k * NT;
      cur[k] = idx < n ? rt[idx] : make_uint4(0, 0, 0, 0);
      const uint32_t up = __shfl_up_sync(0xffffffffu, cur[k].x, 1);
      if (idx < n) {
        const uint32_t prev = lane ? up : (idx ? rt[idx - 1].x : last);
        bad |= (cur[k].x < prev ? 1u : 0u) | (cur[k].x >= (uint32_t)p.S ? 2u : 0u);
        if (kCompact) {
          kd[idx] = make_uint2(cur[k].y, cur[k].z);
          kst[idx] = cur[k].x;
        }
      }
      if (!W64) wide |= !small_delta(cur[k]);
    }
    last = rt[n - 1].x;
    return wide;
  };
  if (ntiles > 0) {
    if (!mbar_wait(&bar[0], 0)) {
      set_status(p.status, BW_STATUS_TIMEOUT);
      lost = 1;
    } else {
      const int n = tile_n(0);
      bigp = load_tile(ring, n);
      if (warp == QW) find_tile_queries(p, qpre, pbase, qcur, ring, n, qbuf_of(0), m->tq[0], lane);
    }
  }
  // end-of-tile barrier: OR of the next tile's wide flag and of lost waits (a
  // second barrier separates the two only when the first is set)
  auto tile_barrier = [&](int wide, int gone, int& big_out) -> bool {
    if (!__syncthreads_or(wide | gone)) {
      big_out = 0;
      return false;
    }
    const bool ab = __syncthreads_or(gone);
    big_out = __syncthreads_or(wide);
    return ab;
  };
  int big = 0;
  bool aborted = tile_barrier(bigp, lost, big);

  int t = 0;
  for (; t < ntiles && !aborted; ++t) {
    const int n = tile_n(t);
    const uint4* tile = ring + (t % RS) * TL;   // (int64 window)
    if (tid == 0 && (kCompact || t >= 1) && issued < ntiles) {
      // the place of tile t (compact) or t - 1 was released by the barrier that ended tile t-1
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      bulk_load(ring + (issued % RS) * TL, p.ev + e0 + (int64_t)issued * TL, (uint32_t)tile_n(issued) * 16u,
                &bar[issued % RS]);
      ++issued;
    }
    const int64_t tq0 = m->tq[t & 1][0], tq1 = m->tq[t & 1][1];
    if (t > 0) {   // window updates of the previous tile, summed over its warps
      const uint32_t v = lane < NW ? m->wsum[(t - 1) & 1][lane] : 0u;
      win += __reduce_add_sync(0xffffffffu, v);
    }
    // fold the window into the prefix row before it could overflow, and after a
    // wide tile (whose events went to the wide histogram)
    if (!W64 && (win >= kFoldAt || wide_live)) {
      fold<NT>(p, H, T, P, wrow, rows_live, wide_live, m);
      win = 0;
      rows_live = true;
      wide_live = false;
    }
    if (!W64 && big && !wide_init) {
      for (uint32_t k = tid; k < C; k += NT) wrow[k] = 0;
      wide_init = true;
      __syncthreads();
    }
    // the tile's queries, one warp each; meanwhile the query warp waits for the next
    // tile and finds its queries (into the other query buffer)
    const bool has_q = tq1 > tq0;
    bool next_found = false;
    if (has_q) {
      if (warp == QW) {
        if (t + 1 < ntiles) {
          const uint4* nt = ring + ((t + 1) % RS) * TL;
          if (!mbar_wait(&bar[(t + 1) % RS], (uint32_t)(((t + 1) / RS) & 1))) {
            set_status(p.status, BW_STATUS_TIMEOUT);
            lost = 1;
          } else {
            find_tile_queries(p, qpre, pbase, qcur, nt, tile_n(t + 1), qbuf_of(t + 1), m->tq[(t + 1) & 1], lane);
          }
        }
        next_found = true;
      }
      const uint4* qb = reinterpret_cast<const uint4*>(qbuf_of(t));
      for (int64_t i = tq0 + warp; warp < QW && i < tq1; i += QW) {
        uint32_t lo, hi, pos;
        if (i - tq0 < QB) {
          const uint4 r = qb[i - tq0];
          lo = r.y;
          hi = r.z;
          pos = r.w;
        } else {
          const uint32_t* r = reinterpret_cast<const uint32_t*>(p.qs + i);
          lo = r[1];
          hi = r[2];
          pos = kCompact ? tile_pos(kst, n, r[0]) : tile_pos(tile, n, r[0]);
        }
        int64_t a;
        if constexpr (W64) a = answer_one64(p, H, T, tile, pos, lo, hi, lane);
        else a = answer_one(p, H, T, P, rows_live, kd, big ? p.ev + e0 + (int64_t)t * TL : nullptr, pos, lo, hi, lane);
        if (lane == 0) p.ans[i] = a;
      }
      __syncthreads();
    }
    // apply the tile
    uint32_t wsum = 0;
#pragma unroll
    for (int k = 0; k < EPT; ++k) {
      const int idx = tid + k * NT;
      if (idx < n) {
        const uint4 e = cur[k];
        if (e.y >= C) {
          bad |= 4u;
        } else if (W64) {
          const uint64_t d = ((uint64_t)e.w << 32) | e.z;
          shared_add_u64(reinterpret_cast<unsigned long long*>(&H[e.y]), d);
          if (p.nch) shared_add_u64(reinterpret_cast<unsigned long long*>(&T[e.y >> kChunkShift]), d);
        } else if (!big) {
          const int32_t d = (int32_t)e.z;
          atomicAdd(reinterpret_cast<int32_t*>(&H[e.y]), d);
          if (p.nch) atomicAdd(reinterpret_cast<int32_t*>(&T[e.y >> kChunkShift]), d);
          wsum += (uint32_t)(d < 0 ? -d : d);
        } else {
          atomicAdd(reinterpret_cast<unsigned long long*>(wrow + e.y), ((unsigned long long)e.w << 32) | e.z);
        }
      }
    }
    wide_live |= big != 0;
    {
      const uint32_t ws = __reduce_add_sync(0xffffffffu, wsum);
      if (lane == 0) m->wsum[t & 1][warp] = ws;
    }
    // next tile: wait for its copy, load this thread's events (and, when no query
    // phase ran, let the query warp find the next tile's queries)
    bigp = 0;
    if (t + 1 < ntiles) {
      const int nn = tile_n(t + 1);
      const uint4* nt = ring + ((t + 1) % RS) * TL;
      if (!mbar_wait(&bar[(t + 1) % RS], (uint32_t)(((t + 1) / RS) & 1))) {
        set_status(p.status, BW_STATUS_TIMEOUT);
        lost = 1;
      } else {
        bigp = load_tile(nt, nn);
        if (warp == QW && !next_found)
          find_tile_queries(p, qpre, pbase, qcur, nt, nn, qbuf_of(t + 1), m->tq[(t + 1) & 1], lane);
      }
    }
    aborted = tile_barrier(bigp, lost, big);
  }

  if (bad)
    set_status(p.status, (bad & 1u) ? BW_STATUS_EVENTS_UNSORTED
                                    : (bad & 2u) ? BW_STATUS_STATE_RANGE : BW_STATUS_EVENT_KEY_RANGE);
  // the query warp's last window copy lands before its shared memory goes away
  if (warp == QW) asm volatile("cp.async.wait_all;" ::: "memory");
  if (aborted) {
    // wait (bounded) for the copies still in flight before the CTA exits: tiles
    // from the one whose wait gave up to the last one issued
    if (tid == 0)
      for (int u = t; u < issued; ++u) mbar_wait(&bar[u % RS], (uint32_t)((u / RS) & 1));
    __syncthreads();
    return;
  }
  // final fold: the block's whole key histogram as a key prefix row
  if (warp == QW && lane == 0) m->tail_q0 = qcur;
  fold<NT>(p, H, T, P, wrow, rows_live && !W64, wide_live && !W64, m);
  // last block: the queries after its last event see every event of the chain,
  // all of it now in the prefix row
  if (b == p.B - 1) {
    for (int64_t i = m->tail_q0 + tid; i < p.Q; i += NT) {
      const uint32_t* r = reinterpret_cast<const uint32_t*>(p.qs + i);
      const uint32_t lo = min(r[1], C), hi = min(r[2], C);
      p.ans[i] = lo < hi ? (int64_t)((uint64_t)__ldcg(P + hi) - (uint64_t)__ldcg(P + lo)) : 0;
    }
    if (warp == QW) qcur = p.Q;
  }
  if (warp == QW && lane == 0) {
    p.btab[2 * b] = qstart;
    p.btab[2 * b + 1] = qcur;
  }
}

// Rows become exclusive column prefixes: row b = the key prefix of the carry of blocks
// 0 .. b-1.  A CTA takes 32 columns, a warp of 32 columns one of 32 ranges of the rows:
// range sums, their prefix through shared memory, then the rows again (from the L2).
// Bound by memory latency at few rows: 152 rows of 4,097 took 23 us as two kernels that
// walked 16 rows (and up to nine segment sums) one after the other, 12 us so (both with
// the fix-up; 608 rows 50 -> 26 us, 456 rows of 1,700 40 -> 21 us).
__global__ void __launch_bounds__(1024) k_chain_carry(ChainParams p) {
  chain_wait();
  __shared__ uint64_t s_sum[32][33];
  const int x = threadIdx.x & 31, y = threadIdx.x >> 5;
  const uint32_t k = blockIdx.x * 32 + x + 1;   // column 0 is always 0
  const int b0 = (int)((int64_t)p.B * y / 32), b1 = (int)((int64_t)p.B * (y + 1) / 32);
  const int64_t w = (int64_t)p.C + 1;
  int64_t* col = p.rows + k;
  constexpr int kBatch = 8;
  uint64_t sum = 0, v[kBatch];
  if (k <= p.C)
    for (int b = b0; b < b1; b += kBatch) {
#pragma unroll
      for (int i = 0; i < kBatch; ++i) v[i] = b + i < b1 ? (uint64_t)col[(b + i) * w] : 0;
#pragma unroll
      for (int i = 0; i < kBatch; ++i) sum += v[i];
    }
  s_sum[y][x] = sum;
  __syncthreads();
  if (k > p.C) return;
  uint64_t run = 0;
  for (int i = 0; i < y; ++i) run += s_sum[i][x];
  for (int b = b0; b < b1; b += kBatch) {
    if (b1 - b0 > kBatch) {   // (else the batch is still at hand)
#pragma unroll
      for (int i = 0; i < kBatch; ++i) v[i] = b + i < b1 ? (uint64_t)col[(b + i) * w] : 0;
    }
#pragma unroll
    for (int i = 0; i < kBatch; ++i) {
      if (b + i < b1) col[(b + i) * w] = (int64_t)run;
      run += v[i];
    }
  }
}

// Block b >= 1: every query of the block adds the carry inside [lo, hi).
__global__ void __launch_bounds__(kChainThreads) k_chain_fixup(ChainParams p) {
  chain_wait();
  const int b = blockIdx.x + 1;
  const int64_t* row = p.rows + (int64_t)b * (p.C + 1);
  const int64_t q0 = p.btab[2 * b], q1 = p.btab[2 * b + 1];
  for (int64_t i = q0 + threadIdx.x; i < q1; i += blockDim.x) {
    const BwQuery q = p.qs[i];
    const uint32_t lo = min(q.lo, p.C), hi = min(q.hi, p.C);
    if (lo < hi) p.ans[i] = (int64_t)((uint64_t)p.ans[i] + (uint64_t)row[hi] - (uint64_t)row[lo]);
  }
}

// Sweep geometries: threads per CTA, events per thread, CTAs per SM the kernel is
// compiled for.  Smaller CTAs give more state blocks and shorter per-tile
// barriers; larger ones amortise the query warp over more appliers.
struct Geometry {
  int threads, ept, minb, stages;
};
constexpr Geometry kGeometries[] = {{128, 4, 5, 3}, {256, 4, 3, 3}, {512, 2, 2, 3},
                                    {256, 4, 4, 2}, {256, 3, 4, 3}, {384, 2, 3, 3}};
constexpr int kNumGeometries = 6;

// (`stages` counts the tile in work, which the int32 window keeps in its compact form.)
// BW_CHAIN_GEOMETRY=<index into kGeometries> pins the geometry (tuning runs).
// Otherwise, when the events fill every CTA with full state blocks, the first that fits of
//   384 x 2 (threads x events), two CTAs an SM or more: int32 window, dense queries, chunk
//     totals (8,000 keys, 12 events a query: 554 us against 625 to 800; 16,000 keys 623
//     against 751 to 851; with 1,000 and 4,096 keys, where 256 x 3 gets four CTAs, it is no
//     faster: 533 / 509, 540 / 536);
//   256 x 4, three: int32 window, few queries (4,096 keys, 1,000 events a query: 108 us
//     against 114; 100 events a query 157 against 159 to 162);
//   256 x 3, four CTAs (three with the int64 window); 256 x 4 and two stages, three (or 256 x
//     3 where it gets as many: 131 against 133);
//   256 x 4, two.
// 384 x 2 takes the place of the last but one and of 256 x 3 where those get three CTAs
// and it does too, with the int64 window (4,000 keys: 94 us against 102 to 109) or a query in
// 256 events and more (8,000 keys, 100 events a query: 180 against 202; 400: 152 against
// 131).  All 16M events, sweep alone.
// Where only one CTA of 512 fits but two of these do, two of 384 x 2 take its place with the
// int64 window (8,000 keys: 168 -> 123 us), two of 256 x 4 else.
// Else (few, short state blocks) 512 threads x 2 events, whose wide CTAs finish each block
// soonest, with one block per SM while every block keeps at least 512 events.  Tiles always
// stay large: smaller tiles shorten the in-tile scans but cost more per tile than they
// save, even on query-dense chains.
int geometry_override() {
  static const int g = [] {
    const char* v = std::getenv("BW_CHAIN_GEOMETRY");
    if (!v || !*v) return -1;
    const int i = std::atoi(v);
    return i >= 0 && i < kNumGeometries ? i : -1;
  }();
  return g;
}

std::once_flag g_attr_once;
cudaError_t g_attr_err = cudaSuccess;

}  // namespace

bool chain_selected(const BwReplayArgs* a) {
  if (!(a->flags & BW_REPLAY_CHAIN_HINT) || (a->flags & BW_REPLAY_GENERAL)) return false;
  if (a->n_keys > kChainMaxKeys || a->n_states < 1) return false;
  if (a->events && (reinterpret_cast<uintptr_t>(a->events) & 15) != 0) return false;
  return (a->flags & BW_REPLAY_CHAIN_KERNEL) || a->n_queries * 8 <= a->n_events;
}

int chain_spec(const BwReplayArgs* a, int sms, ChainSpec& s) {
  s.S = a->n_states;
  s.C = a->n_keys;
  s.E = a->n_events;
  s.Q = a->n_queries;
  // query-dense chains (more than one query per 64 events) keep chunk totals at any
  // domain size: their intervals are probed often, and a probe over chunk totals
  // reads ~width/1024 words per lane instead of ~width/128
  const bool dense = s.Q * 64 > s.E;
  s.nch = (s.C > kFlatKeys || dense) ? (int32_t)((s.C + 31) >> 5) : 0;
  s.w64 = (a->flags & BW_REPLAY_WIDE) && s.C <= kChainMaxKeys64;
  const int hw = s.w64 ? 8 : 4;
  int pin = geometry_override();
  int fit[kNumGeometries];
  size_t need[kNumGeometries];
  for (int g = 0; g < kNumGeometries; ++g) {
    const Geometry& G = kGeometries[g];
    need[g] = sweep_smem(s.C, s.nch, G.threads * G.ept, G.stages, hw).bytes;
    fit[g] = (int)(kSmemPerSM / (need[g] + 1024));
    if (fit[g] > G.minb) fit[g] = G.minb;
  }
  if (pin >= 0 && fit[pin] < 1) pin = -1;
  const bool pinned = pin >= 0;
  auto full = [&](int g, int ctas) { return fit[g] >= ctas && s.E >= (int64_t)sms * fit[g] * kChainMinBlockEvents; };
  if (pin < 0 && !s.w64 && dense && s.C > kFlatKeys && full(5, 2)) pin = 5;
  if (pin < 0 && !s.w64 && !dense && full(1, 3)) pin = 1;
  if (pin < 0 && full(4, s.w64 ? 3 : 4)) pin = 4;
  if (pin < 0 && full(3, 3)) pin = 3;
  if (pin < 0 && full(1, 2)) pin = 1;
  if (!pinned && (pin == 4 || pin == 3) && fit[pin] == 3 && fit[5] >= 3 && (s.w64 || s.Q * 256 > s.E)) pin = 5;
  if (!pinned && pin == 3 && fit[4] >= fit[3]) pin = 4;
  const int two = s.w64 ? 5 : 3;
  const bool pair = pin < 0 && full(two, 2);
  if (pair) pin = two;
  // too few events to fill the GPU with full blocks: the widest CTA (512 threads)
  // finishes each short block soonest (measured on the 1M-event plain chain)
  const bool few = pin < 0;
  if (few && fit[2] >= 1) pin = 2;
  int best = -1, best_threads = 0;
  for (int g = 0; g < kNumGeometries; ++g) {
    const Geometry& G = kGeometries[g];
    const size_t smem = need[g];
    const int ctas = fit[g];
    if (ctas < 1) continue;
    if (pin >= 0 ? g == pin : ctas * G.threads >= best_threads) {
      best = g;
      best_threads = ctas * G.threads;
      s.threads = G.threads;
      s.ept = G.ept;
      s.geometry = g;
      s.smem = smem;
      s.ctas_per_sm = ctas;
    }
  }
  if (best < 0) return BW_EINVAL;
  int64_t B = (s.E + kChainMinBlockEvents - 1) / kChainMinBlockEvents;
  int64_t floor = B;
  // few events: one block per SM when every block still gets 512 events or more (25,000
  // events: 12 blocks 25 us a replay, 48 blocks 21 us); but a single block, without carry and
  // fix-up, up to some 4,000 events, a query counted as 16 and sixteen keys of a row as one (1 / 4
  // blocks, us: 2,200 events, 1 query, 100 keys 11.8 / 13.9, 32,000 keys 31.4 / 45.3; 45 queries, 10,000
  // keys 23.1 / 27.0; 2,200 queries, 100 keys 198 / 60; 4,400 events, 1 query, 100 keys 13.9 / 14.3, 32,000
  // keys 33.4 / 45.8; 8,800 events, 32,000 keys 73 / 47)
  if (few && B < sms) {
    floor = std::min<int64_t>(sms, std::max<int64_t>(B, s.E / 2048));
    B = std::min<int64_t>(sms, std::max<int64_t>(B, s.E / 512));
    if (s.E + 16 * s.Q < 4096 + (int64_t)s.C / 16) B = 1;
  } else if (pair) {
    floor = std::min<int64_t>(B, sms);
  }
  B = std::min<int64_t>(B, (int64_t)sms * s.ctas_per_sm);
  // (the blocks that these rules add to `floor` take no more than the 32 MiB that the replay
  // without allocations has)
  const int64_t row_bytes = (int64_t)s.C * 16 + 24, small = ((int64_t)32 << 20) - 1024;
  if (floor * row_bytes <= small) B = std::min(B, std::max(floor, small / row_bytes));
  if (a->blocks > 0) B = a->blocks;
  if (B > s.E) B = s.E;
  if (B < 1) B = 1;
  if (B > (1 << 20)) return BW_EINVAL;
  s.B = (int32_t)B;
  auto al = [](size_t x) { return (x + 255) & ~size_t(255); };
  size_t o = 256;   // status word
  s.off_btab = o;  o = al(o + (size_t)s.B * 16);
  s.off_rows = o;  o = al(o + (size_t)s.B * (s.C + 1) * 8);
  s.off_wide = o;  o = al(o + (size_t)s.B * s.C * 8);
  s.total = o;
  return 0;
}

int chain_enqueue(const ChainSpec& s, const BwReplayArgs* a, EventSet* evs, int* kernels) {
  std::call_once(g_attr_once, [] {
    const cudaFuncAttribute A = cudaFuncAttributeMaxDynamicSharedMemorySize;
    const void* fns[] = {(const void*)k_chain_sweep<128, 4, 5, 3, false>, (const void*)k_chain_sweep<256, 4, 3, 3, false>,
                         (const void*)k_chain_sweep<512, 2, 2, 3, false>, (const void*)k_chain_sweep<256, 4, 4, 2, false>,
                         (const void*)k_chain_sweep<256, 3, 4, 3, false>, (const void*)k_chain_sweep<128, 4, 5, 3, true>,
                         (const void*)k_chain_sweep<256, 4, 3, 3, true>, (const void*)k_chain_sweep<512, 2, 2, 3, true>,
                         (const void*)k_chain_sweep<256, 4, 4, 2, true>, (const void*)k_chain_sweep<256, 3, 4, 3, true>,
                         (const void*)k_chain_sweep<384, 2, 3, 3, false>, (const void*)k_chain_sweep<384, 2, 3, 3, true>};
    for (const void* f : fns)
      if (g_attr_err == cudaSuccess) g_attr_err = cudaFuncSetAttribute(f, A, kSmemLimit);
  });
  if (g_attr_err != cudaSuccess) return report(g_attr_err, "chain sweep attribute");
  cudaStream_t st = static_cast<cudaStream_t>(a->stream);
  char* ws = static_cast<char*>(a->workspace);
  ChainParams p;
  p.ev = reinterpret_cast<const uint4*>(a->events);
  p.qs = a->queries;
  p.ans = a->answers;
  p.parent = a->parent;
  p.E = s.E;
  p.Q = s.Q;
  p.S = s.S;
  p.C = s.C;
  p.B = s.B;
  p.nch = s.nch;
  p.qweight = s.B > 1 && s.Q * kQueryWeight > s.E ? kQueryWeight : 0;   // (one block has nothing to cut)
  p.rows = reinterpret_cast<int64_t*>(ws + s.off_rows);
  p.wide = reinterpret_cast<int64_t*>(ws + s.off_wide);
  p.btab = reinterpret_cast<int64_t*>(ws + s.off_btab);
  p.status = reinterpret_cast<int32_t*>(ws);
  int rc = report(cudaMemsetAsync(ws, 0, 4, st), "status reset");
  if (rc) return rc;
  if (evs) {
    for (int i = 0; i <= BW_STAGE_SWEEP; ++i)
      if ((rc = report(cudaEventRecord(evs->ev[i], st), "event record"))) return rc;
  }
  switch (s.geometry * 2 + (s.w64 ? 1 : 0)) {
    case 0: k_chain_sweep<128, 4, 5, 3, false><<<s.B, 128, s.smem, st>>>(p); break;
    case 1: k_chain_sweep<128, 4, 5, 3, true><<<s.B, 128, s.smem, st>>>(p); break;
    case 2: k_chain_sweep<256, 4, 3, 3, false><<<s.B, 256, s.smem, st>>>(p); break;
    case 3: k_chain_sweep<256, 4, 3, 3, true><<<s.B, 256, s.smem, st>>>(p); break;
    case 4: k_chain_sweep<512, 2, 2, 3, false><<<s.B, 512, s.smem, st>>>(p); break;
    case 5: k_chain_sweep<512, 2, 2, 3, true><<<s.B, 512, s.smem, st>>>(p); break;
    case 6: k_chain_sweep<256, 4, 4, 2, false><<<s.B, 256, s.smem, st>>>(p); break;
    case 7: k_chain_sweep<256, 4, 4, 2, true><<<s.B, 256, s.smem, st>>>(p); break;
    case 8: k_chain_sweep<256, 3, 4, 3, false><<<s.B, 256, s.smem, st>>>(p); break;
    case 9: k_chain_sweep<256, 3, 4, 3, true><<<s.B, 256, s.smem, st>>>(p); break;
    case 10: k_chain_sweep<384, 2, 3, 3, false><<<s.B, 384, s.smem, st>>>(p); break;
    default: k_chain_sweep<384, 2, 3, 3, true><<<s.B, 384, s.smem, st>>>(p); break;
  }
  int k = 1;
  if ((rc = report(cudaGetLastError(), "chain sweep launch"))) return rc;
  if (evs && (rc = report(cudaEventRecord(evs->ev[BW_STAGE_SWEEP + 1], st), "event record"))) return rc;
  if (s.B > 1) {
    // (1M events, 152 blocks: 39.4 -> 36.0 us a replay launched chained; 7M events and more,
    // whose blocks do not end together: 1 to 2% slower)
    const bool early = s.E < ((int64_t)1 << 22);
    if ((rc = report(launch_chained(early, k_chain_carry, (s.C + 31) / 32, 1024, 0, st, p), "chain carry launch")))
      return rc;   // (columns 1 .. C)
    if ((rc = report(launch_chained(early, k_chain_fixup, s.B - 1, kChainThreads, 0, st, p), "chain fix-up launch")))
      return rc;
    k += 2;
  }
  if (evs) {
    evs->chain = 1;
    if ((rc = report(cudaEventRecord(evs->ev[BW_STAGE_COUNT + 1], st), "event record"))) return rc;
  }
  if (kernels) *kernels += k;
  return 0;
}

}  // namespace bw
