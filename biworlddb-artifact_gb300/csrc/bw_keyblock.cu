// bw_keyblock.cu -- one-tree replay over large key domains, by key blocks.
//
// The state-block pipeline (bw_pipeline.cu) carries one dense key-prefix row per
// state block: over a domain of millions of keys the rows bound it to a few dozen
// blocks (80 MB a row at 10M keys), and each block sweeps its events once per rank
// slice that fits shared memory.  Here the axes are exchanged.  The keys are cut into
// blocks of m events and the dense rows run over the states that are asked about
// ("columns", in tour order), so a row entry is one int64 per (column, key block):
//
//   answer(v, lo, hi) = R[v][blk(hi)] - R[v][blk(lo)]        whole key blocks
//                     + L(blk(hi), v, hi) - L(blk(lo), v, lo)  part of a block
//
// R[v][b] sums the root path's events in the key blocks before b, L(b, v, k) those in
// block b with a key below k.  Stages, on the ranked tour of pipe_tour():
//
//   columns   k_kb_steps, k_kb_cols   a step's time = the queries answered before it;
//             a state's events count from its enter to its exit (two signed points),
//             and not at all when no query lies between.
//   keys      k_kb_key_hist + scan    pos[k] = events with a key below k: an event's
//             slot, and with it its key block pos / m and slot in the block.
//   points    k_kb_point_count / scan / k_kb_point_scatter   signed points grouped by
//             key block, in tour order (a stable partition of up to 4,096 digits).
//   rows      k_kb_seg, k_kb_segscan, k_kb_rows   R, in two passes over the tour cut in
//             equal segments (net sum per segment and block, then the running vector
//             in shared memory, written out scanned over the blocks at every column).
//   probes    k_kb_probe_count / scan / k_kb_probe_scatter   both bounds of every query
//             grouped by key block, in tour order; the whole-block part goes to acc.
//   sweep     k_kb_sweep   one CTA per key block: L of every probe (below).
//   answers   k_kb_answers  acc, kept in tour order, to the queries' own places.
//
// Measured on 20M events over 10M keys, 100k states, 100M range queries (the
// versioned sparse-key workload): see k_kb_sweep and kb_select.
#include <cuda_runtime.h>
#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <mutex>

#include "bw_gpu.h"
#include "bw_common.cuh"
#include "bw_pipeline.cuh"
#include "bw_keyblock.cuh"

namespace bw {
namespace {

constexpr uint32_t kAll = 0xffffffffu;
constexpr uint32_t kNone = 0xffffffffu;

struct KbParams {
  const BwEvent* ev;
  const BwQuery* qs;
  int64_t* answers;
  const int64_t *eoff, *qoff;
  const uint64_t* rank;
  const int64_t* cnt;
  const int32_t *ehead, *xhead;
  int32_t* step;        // 2S: v on the enter of v, ~v on its exit
  int64_t* w;           // 2S: inclusive (columns << 32) + queries up to the step
  int64_t* ep;          // 2S: inclusive events that count, up to the step
  uint32_t* time;       // 2S: queries answered before the step
  int32_t* colstate;    // per column: its state,
  uint32_t* coltime;    //   the queries before it (and after the last column: all),
  int32_t* colstep;     //   and its enter step
  uint32_t* pos;        // C + 1
  uint32_t* pthist;
  uint4* pts;           // {time, slot, delta}
  uint64_t* seg;        // segs x B
  int64_t* rows;        // columns x B
  uint32_t* prhist;
  uint2* prs;           // {query in tour order, slot | lower bound << 31}
  unsigned long long* acc;   // per query in tour order
  const int32_t* status;
  int32_t* ticket;
  int64_t E, Q, pt_tiles, pr_tiles;
  int32_t S, B, segs;
  uint32_t C, m;
};

// Tour steps of state v's enter and exit (one tree: the tour ends at step 2S).
__device__ __forceinline__ void kb_steps_of(const KbParams& p, int32_t v, int64_t& pe, int64_t& px) {
  const int64_t He = (uint32_t)(uint64_t)p.cnt[p.S - 1], base = 2 * (int64_t)p.S;
  const uint64_t c = (uint64_t)p.cnt[v], cp = v ? (uint64_t)p.cnt[v - 1] : 0ull;
  const int64_t eid = (int64_t)(uint32_t)c - 1;
  const int64_t xid = (int64_t)(cp >> 32);   // exit heads below v
  pe = base - (int64_t)(uint32_t)p.rank[eid] + (v - p.ehead[eid]);
  px = base - (int64_t)(uint32_t)p.rank[He + xid] + (p.xhead[xid] - v);
}

__device__ __forceinline__ int64_t kb_own(const KbParams& p, int32_t v) {
  const int64_t nq = p.qoff[v + 1] - p.qoff[v];
  return nq > 0 ? ((int64_t)1 << 32) + nq : 0;
}

__global__ void k_kb_steps(KbParams p) {
  if (*p.status) return;
  for (int32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < p.S; v += gridDim.x * blockDim.x) {
    int64_t pe, px;
    kb_steps_of(p, v, pe, px);
    p.step[pe] = v;
    p.step[px] = ~v;
    p.w[pe] = kb_own(p, v);
    p.w[px] = 0;
  }
}

__global__ void k_kb_cols(KbParams p) {
  if (*p.status) return;
  for (int32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < p.S; v += gridDim.x * blockDim.x) {
    int64_t pe, px;
    kb_steps_of(p, v, pe, px);
    const int64_t own = kb_own(p, v), a = p.w[pe] - own, z = p.w[px];
    const uint32_t ta = (uint32_t)a, tz = (uint32_t)z;
    const int64_t ne = p.eoff[v + 1] - p.eoff[v];
    p.time[pe] = ta;
    p.time[px] = tz;
    p.ep[pe] = ta != tz ? ne : 0;                          // a query lies below v
    p.ep[px] = ta != tz && (int64_t)tz < p.Q ? ne : 0;     // and another one after it
    if (own) {
      const int32_t c = (int32_t)(a >> 32);
      p.colstate[c] = v;
      p.coltime[c] = ta;
      p.colstep[c] = (int32_t)pe;
    }
    if (v == 0) p.coltime[z >> 32] = (uint32_t)p.Q;        // the root leaves last
  }
}

__device__ __forceinline__ int32_t kb_columns(const KbParams& p) { return (int32_t)(p.w[2 * (int64_t)p.S - 1] >> 32); }
__device__ __forceinline__ int64_t kb_points(const KbParams& p) { return p.ep[2 * (int64_t)p.S - 1]; }

// pos[k + 1] counts the events of key k (one atomic per distinct key of a warp's 32
// events: a hot key would otherwise serialise at the L2).
__global__ void k_kb_key_hist(KbParams p) {
  if (*p.status) return;
  const int64_t n32 = (p.E + 31) & ~(int64_t)31;
  const int lane = threadIdx.x & 31;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n32; i += (int64_t)gridDim.x * blockDim.x) {
    const uint32_t k = i < p.E ? p.ev[i].key : kNone;
    const unsigned peers = __match_any_sync(kAll, k);
    if (i < p.E && (peers & ((1u << lane) - 1u)) == 0) atomicAdd(p.pos + k + 1, (unsigned)__popc(peers));
  }
}

// First step in [lo, hi] with ep[step] > j (there is one).
__device__ __forceinline__ int32_t kb_find_step(const int64_t* ep, int32_t lo, int32_t hi, int64_t j) {
  while (lo < hi) {
    const int32_t mid = (lo + hi) >> 1;
    if (ep[mid] > j) hi = mid; else lo = mid + 1;
  }
  return lo;
}
// Last column in [lo, hi] with coltime <= j.
__device__ __forceinline__ int32_t kb_find_col(const uint32_t* coltime, int32_t lo, int32_t hi, uint32_t j) {
  while (lo < hi) {
    const int32_t mid = (lo + hi + 1) >> 1;
    if (coltime[mid] <= j) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// Point j of the tour: event of step t, negated on an exit.
struct KbPoint {
  uint32_t time, key;
  uint64_t delta;
};
__device__ __forceinline__ KbPoint kb_point(const KbParams& p, int32_t t, int64_t j) {
  const int32_t v = p.step[t], s = v < 0 ? ~v : v;
  const uint4 e = __ldg(reinterpret_cast<const uint4*>(p.ev) + (p.eoff[s + 1] - (p.ep[t] - j)));
  const uint64_t d = ((uint64_t)e.w << 32) | e.z;
  return KbPoint{p.time[t], e.y, v < 0 ? (uint64_t)0 - d : d};
}

// Step range [s_t[0], s_t[1]] holding the points [j0, j1), j0 < j1 (whole CTA).
__device__ __forceinline__ void kb_step_range(const KbParams& p, int64_t j0, int64_t j1, int32_t* s_t) {
  if (threadIdx.x < 2) s_t[threadIdx.x] = kb_find_step(p.ep, 0, 2 * p.S - 1, threadIdx.x ? j1 - 1 : j0);
  __syncthreads();
}
__device__ __forceinline__ void kb_col_range(const KbParams& p, int64_t j0, int64_t j1, int32_t* s_c) {
  if (threadIdx.x < 2)
    s_c[threadIdx.x] = kb_find_col(p.coltime, 0, kb_columns(p) - 1, (uint32_t)(threadIdx.x ? j1 - 1 : j0));
  __syncthreads();
}

// An event of the last key of its key block lies below no probe of the block: it
// counts in the rows only (which also keeps a hot key out of the sweep).
__device__ __forceinline__ bool kb_swept(const KbParams& p, uint32_t key, uint32_t b) { return p.pos[key + 1] / p.m == b; }

// Stable rank of a warp's ITEMS x 32 digits (kNone: no item) within the warp; wc: the
// warp's counters, zeroed.  r[j] = earlier items of the warp with the same digit.
template <int ITEMS>
__device__ __forceinline__ void kb_rank(uint16_t* wc, const uint32_t (&d)[ITEMS], uint16_t (&r)[ITEMS]) {
  const unsigned lt = (1u << (threadIdx.x & 31)) - 1u;
#pragma unroll
  for (int j = 0; j < ITEMS; ++j) {
    const unsigned peers = __match_any_sync(kAll, d[j]);
    const uint32_t old = d[j] != kNone ? wc[d[j]] : 0u;
    __syncwarp();
    r[j] = (uint16_t)(old + __popc(peers & lt));
    if (d[j] != kNone && (peers & lt) == 0) wc[d[j]] = (uint16_t)(old + __popc(peers));
    __syncwarp();
  }
}
// Counters of the CTA's NW warps -> output position of each warp's first item per digit.
template <int NW>
__device__ __forceinline__ void kb_bases(uint16_t* wc, uint32_t* base, int32_t B, int32_t Bp, const uint32_t* hist,
                                         int64_t ntiles) {
  __syncthreads();
  for (int32_t d = threadIdx.x; d < B; d += NW * 32) {
    uint32_t run = 0;
#pragma unroll
    for (int w = 0; w < NW; ++w) {
      const uint32_t c = wc[w * Bp + d];
      wc[w * Bp + d] = (uint16_t)run;
      run += c;
    }
    base[d] = hist[(int64_t)d * ntiles + blockIdx.x] - run;   // inclusive counts
  }
  __syncthreads();
}
__device__ __forceinline__ void kb_write_hist(const uint32_t* h, int32_t B, uint32_t* hist, int64_t ntiles) {
  __syncthreads();
  for (int32_t d = threadIdx.x; d < B; d += blockDim.x) hist[(int64_t)d * ntiles + blockIdx.x] = h[d];
}

constexpr int kPtWarps = 16, kPtItems = kKbPtTile / (kPtWarps * 32);
constexpr int kPrWarps = 16, kPrItems = 2 * kKbPrTile / (kPrWarps * 32);
inline size_t kb_scatter_smem(int32_t B, int warps) { return (size_t)B * 4 + (size_t)warps * ((B + 7) & ~7) * 2 + 16; }

__global__ void __launch_bounds__(kPtWarps * 32) k_kb_point_count(KbParams p) {
  if (*p.status) return;
  extern __shared__ __align__(16) uint32_t h[];
  __shared__ int32_t s_t[2];
  for (int32_t i = threadIdx.x; i < p.B; i += blockDim.x) h[i] = 0;
  __syncthreads();
  const int64_t j0 = (int64_t)blockIdx.x * kKbPtTile, j1 = imin64(j0 + kKbPtTile, kb_points(p));
  if (j0 < j1) {
    kb_step_range(p, j0, j1, s_t);
    for (int64_t j = j0 + threadIdx.x; j < j1; j += blockDim.x) {
      const int32_t t = kb_find_step(p.ep, s_t[0], s_t[1], j);
      const KbPoint x = kb_point(p, t, j);
      const uint32_t b = p.pos[x.key] / p.m;
      if (kb_swept(p, x.key, b)) atomicAdd(h + b, 1u);
    }
  }
  kb_write_hist(h, p.B, p.pthist, p.pt_tiles);
}

__global__ void __launch_bounds__(kPtWarps * 32, 2) k_kb_point_scatter(KbParams p) {
  if (*p.status) return;
  extern __shared__ __align__(16) uint32_t base[];
  __shared__ int32_t s_t[2];
  const int32_t Bp = (p.B + 7) & ~7;
  uint16_t* wc = reinterpret_cast<uint16_t*>(base + ((p.B + 3) & ~3));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t j0 = (int64_t)blockIdx.x * kKbPtTile, j1 = imin64(j0 + kKbPtTile, kb_points(p));
  if (j0 >= j1) return;
  for (int32_t i = threadIdx.x; i < kPtWarps * Bp / 2; i += blockDim.x) reinterpret_cast<uint32_t*>(wc)[i] = 0;
  kb_step_range(p, j0, j1, s_t);
  uint32_t d[kPtItems], slot[kPtItems], time[kPtItems];
  uint64_t delta[kPtItems];
  uint16_t r[kPtItems];
#pragma unroll
  for (int i = 0; i < kPtItems; ++i) {
    const int64_t j = j0 + (warp * kPtItems + i) * 32 + lane;
    d[i] = kNone;
    if (j < j1) {
      const KbPoint x = kb_point(p, kb_find_step(p.ep, s_t[0], s_t[1], j), j);
      const uint32_t ps = p.pos[x.key], b = ps / p.m;
      if (kb_swept(p, x.key, b)) d[i] = b;
      slot[i] = ps - b * p.m;
      time[i] = x.time;
      delta[i] = x.delta;
    }
  }
  kb_rank<kPtItems>(wc + warp * Bp, d, r);
  kb_bases<kPtWarps>(wc, base, p.B, Bp, p.pthist, p.pt_tiles);
#pragma unroll
  for (int i = 0; i < kPtItems; ++i)
    if (d[i] != kNone)
      p.pts[(size_t)base[d[i]] + wc[warp * Bp + d[i]] + r[i]] =
          make_uint4(time[i], slot[i], (uint32_t)delta[i], (uint32_t)(delta[i] >> 32));
}

// ------------------------------------------------------------------ rows
__device__ __forceinline__ void kb_add_points(const KbParams& p, unsigned long long* vec, int64_t j0, int64_t j1,
                                              int32_t t0, int32_t t1) {
  for (int64_t j = j0 + threadIdx.x; j < j1; j += blockDim.x) {
    const KbPoint x = kb_point(p, kb_find_step(p.ep, t0, t1, j), j);
    shared_add_u64(vec + p.pos[x.key] / p.m, x.delta);
  }
}
__device__ __forceinline__ int64_t kb_seg_start(const KbParams& p, int32_t g) {
  return (int64_t)(((__int128)kb_points(p) * g) / p.segs);
}

// Net delta of every tour segment in every key block.
__global__ void __launch_bounds__(256) k_kb_seg(KbParams p) {
  if (*p.status) return;
  extern __shared__ __align__(16) unsigned long long vec[];
  __shared__ int32_t s_t[2];
  for (int32_t i = threadIdx.x; i < p.B; i += blockDim.x) vec[i] = 0;
  __syncthreads();
  const int64_t j0 = kb_seg_start(p, blockIdx.x), j1 = kb_seg_start(p, blockIdx.x + 1);
  if (j0 < j1) {
    kb_step_range(p, j0, j1, s_t);
    kb_add_points(p, vec, j0, j1, s_t[0], s_t[1]);
  }
  __syncthreads();
  for (int32_t i = threadIdx.x; i < p.B; i += blockDim.x) p.seg[(size_t)blockIdx.x * p.B + i] = vec[i];
}

// Exclusive prefix over the segments, per key block: 32 blocks x 32 segment ranges a CTA.
__global__ void __launch_bounds__(1024) k_kb_segscan(KbParams p) {
  if (*p.status) return;
  __shared__ uint64_t s[32][33];
  const int x = threadIdx.x & 31, y = threadIdx.x >> 5;
  const int32_t b = blockIdx.x * 32 + x;
  const int32_t g0 = (int32_t)((int64_t)p.segs * y / 32), g1 = (int32_t)((int64_t)p.segs * (y + 1) / 32);
  uint64_t sum = 0;
  if (b < p.B)
    for (int32_t g = g0; g < g1; ++g) sum += p.seg[(size_t)g * p.B + b];
  s[y][x] = sum;
  __syncthreads();
  uint64_t run = 0;
  for (int i = 0; i < y; ++i) run += s[i][x];
  if (b < p.B)
    for (int32_t g = g0; g < g1; ++g) {
      const uint64_t v = p.seg[(size_t)g * p.B + b];
      p.seg[(size_t)g * p.B + b] = run;
      run += v;
    }
}

// First column whose points (all up to its enter step) number more than j.
__device__ __forceinline__ int32_t kb_col_after(const KbParams& p, int32_t nc, int64_t j) {
  int32_t lo = 0, hi = nc;
  while (lo < hi) {
    const int32_t mid = (lo + hi) >> 1;
    if (p.ep[p.colstep[mid]] > j) hi = mid; else lo = mid + 1;
  }
  return lo;
}

// A segment's columns: the running vector over the key blocks (shared memory) takes
// the points up to the column and is written out scanned.  Bound by the row writes.
__global__ void __launch_bounds__(256) k_kb_rows(KbParams p) {
  if (*p.status) return;
  extern __shared__ __align__(16) unsigned long long vec[];
  unsigned long long* out = vec + p.B;
  __shared__ int32_t s_c[2];
  const int64_t j0 = kb_seg_start(p, blockIdx.x), j1 = kb_seg_start(p, blockIdx.x + 1);
  if (threadIdx.x < 2) {
    const bool last = blockIdx.x + 1 == (unsigned)p.segs;
    const int32_t nc = kb_columns(p);
    // columns of the segment: point counts in (j0, j1], and those without points in the first one
    s_c[threadIdx.x] = threadIdx.x ? (last ? nc : kb_col_after(p, nc, j1)) : (blockIdx.x ? kb_col_after(p, nc, j0) : 0);
  }
  for (int32_t i = threadIdx.x; i < p.B; i += blockDim.x) vec[i] = p.seg[(size_t)blockIdx.x * p.B + i];
  __syncthreads();
  const int32_t per = ((p.B + 255) / 256) | 1;   // odd: a thread's entries start in different banks
  const int32_t i0 = min(p.B, (int32_t)threadIdx.x * per), i1 = min(p.B, i0 + per);
  int64_t j = j0;
  int32_t t = 0;
  if (s_c[0] < s_c[1]) t = kb_find_step(p.ep, 0, 2 * p.S - 1, j0);
  for (int32_t c = s_c[0]; c < s_c[1]; ++c) {
    const int32_t tc = p.colstep[c];
    const int64_t je = p.ep[tc];
    kb_add_points(p, vec, j, je, t, tc);
    j = je;
    t = tc;
    __syncthreads();
    uint64_t s = 0;
    for (int32_t i = i0; i < i1; ++i) s += vec[i];
    uint64_t run = block_exclusive_scan<uint64_t>(s);
    for (int32_t i = i0; i < i1; ++i) {
      out[i] = run;
      run += vec[i];
    }
    __syncthreads();
    int64_t* row = p.rows + (size_t)c * p.B;
    for (int32_t i = threadIdx.x; i < p.B; i += blockDim.x) row[i] = (int64_t)out[i];
    __syncthreads();
  }
}

// ------------------------------------------------------------------ probes
// acc[j] = the slots of query j's bounds (both 0 when the interval is empty), and the
// probes of every key block; a probe at the first slot of its block has nothing below.
__global__ void __launch_bounds__(512) k_kb_probe_count(KbParams p) {
  if (*p.status) return;
  extern __shared__ __align__(16) uint32_t h[];
  __shared__ int32_t s_c[2];
  for (int32_t i = threadIdx.x; i < p.B; i += blockDim.x) h[i] = 0;
  const int64_t j0 = (int64_t)blockIdx.x * kKbPrTile, j1 = imin64(j0 + kKbPrTile, p.Q);
  kb_col_range(p, j0, j1, s_c);
  for (int64_t j = j0 + threadIdx.x; j < j1; j += blockDim.x) {
    const int32_t c = kb_find_col(p.coltime, s_c[0], s_c[1], (uint32_t)j);
    const int64_t q = p.qoff[p.colstate[c]] + (j - p.coltime[c]);
    const uint32_t lo = p.qs[q].lo, hi = p.qs[q].hi;
    uint32_t a = 0, z = 0;
    if (lo < hi) {
      a = __ldg(p.pos + lo);
      z = __ldg(p.pos + hi);
    }
    p.acc[j] = ((unsigned long long)z << 32) | a;
    if (a != z) {
      const uint32_t ba = a / p.m, bz = z / p.m;
      if (a != ba * p.m) atomicAdd(h + ba, 1u);
      if (z != bz * p.m) atomicAdd(h + bz, 1u);
    }
  }
  kb_write_hist(h, p.B, p.prhist, p.pr_tiles);
}

// Lanes 2i and 2i + 1 hold the lower and upper bound of a query, so that a warp's
// probes are in tour order.
__global__ void __launch_bounds__(kPrWarps * 32, 2) k_kb_probe_scatter(KbParams p) {
  if (*p.status) return;
  extern __shared__ __align__(16) uint32_t base[];
  __shared__ int32_t s_c[2];
  const int32_t Bp = (p.B + 7) & ~7;
  uint16_t* wc = reinterpret_cast<uint16_t*>(base + ((p.B + 3) & ~3));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t j0 = (int64_t)blockIdx.x * kKbPrTile, j1 = imin64(j0 + kKbPrTile, p.Q);
  for (int32_t i = threadIdx.x; i < kPrWarps * Bp / 2; i += blockDim.x) reinterpret_cast<uint32_t*>(wc)[i] = 0;
  kb_col_range(p, j0, j1, s_c);
  uint32_t d[kPrItems], slot[kPrItems];
  uint16_t r[kPrItems];
#pragma unroll
  for (int i = 0; i < kPrItems; ++i) {
    const int64_t j = j0 + (warp * kPrItems + i) * 16 + (lane >> 1);
    d[i] = kNone;
    slot[i] = 0;
    if (j < j1) {
      const unsigned long long az = p.acc[j];
      const uint32_t a = (uint32_t)az, z = (uint32_t)(az >> 32);
      const uint32_t x = (lane & 1) ? z : a, b = x / p.m;
      slot[i] = x - b * p.m;
      if (a != z && slot[i]) d[i] = b;
    }
  }
  kb_rank<kPrItems>(wc + warp * Bp, d, r);
  kb_bases<kPrWarps>(wc, base, p.B, Bp, p.prhist, p.pr_tiles);
#pragma unroll
  for (int i = 0; i < kPrItems; ++i) {
    const int64_t j = j0 + (warp * kPrItems + i) * 16 + (lane >> 1);
    if (d[i] != kNone)
      p.prs[(size_t)base[d[i]] + wc[warp * Bp + d[i]] + r[i]] =
          make_uint2((uint32_t)j, slot[i] | ((lane & 1) ? 0u : 0x80000000u));
    if (j < j1 && !(lane & 1)) {
      const unsigned long long az = p.acc[j];
      const uint32_t ba = (uint32_t)az / p.m, bz = (uint32_t)(az >> 32) / p.m;
      uint64_t v = 0;
      if (ba != bz) {
        const int64_t* row = p.rows + (size_t)kb_find_col(p.coltime, s_c[0], s_c[1], (uint32_t)j) * p.B;
        v = (uint64_t)row[bz] - (uint64_t)row[ba];
      }
      p.acc[j] = v;   // read by this lane pair only, both reads above
    }
    __syncwarp();
  }
}

// ------------------------------------------------------------------ sweep
// One key block at a time per CTA: its points (signed deltas at slots) and probes
// (prefixes over the slots), both in tour order.  The points before the current tile
// of 32 are held as a prefix structure of radix 32 over the slots: T0[s] = sum of the
// slots below s in s's group of 32, T1 = sum of the groups below in the warp's range,
// W = the warps' totals.  A probe is one read of each plus its correction inside the
// tile, tab[points before it in time][points below it by slot], for which a seventeenth
// warp sorts the next tile's slots and sums its table while the tile is probed.  Sixteen
// warps own m / 16 slots each and apply the tile's points in their range without atomics:
// the 32 lanes add to the tail of the point's group, T1 stays in registers.
constexpr int kSwWarps = 16, kSwThreads = kSwWarps * 32 + 32, kSwPage = kSwWarps * 32;
struct KbSweepSmem {
  unsigned long long T1[kKbMaxSlots / 32];
  unsigned long long W[kSwWarps];
  unsigned long long tab[2][32 * 32];       // [x - 1][y - 1]
  uint4 pt[2][32];                           // {time, slot, delta}
  uint32_t tm[2][32], sorted[2][32];
  uint32_t next_time[2];                     // time of the tile after (kNone: none)
  int32_t block;
};

// Values of v[0..32) (ascending) that are < x (kLess) or <= x.
template <bool kLess>
__device__ __forceinline__ int kb_below(const uint32_t* v, uint32_t x) {
  int n = 0;
#pragma unroll
  for (int s = 16; s; s >>= 1) {
    const uint32_t y = v[n + s - 1];
    if (kLess ? y < x : y <= x) n += s;
  }
  const uint32_t y = v[n];
  return n + ((kLess ? y < x : y <= x) ? 1 : 0);
}

__global__ void __launch_bounds__(kSwThreads, 2) k_kb_sweep(KbParams p) {
  if (*p.status) return;
  extern __shared__ __align__(16) unsigned long long T0[];   // m slots
  __shared__ KbSweepSmem sm;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bool builder = warp == kSwWarps;
  const uint32_t g = p.m / kKbSlotStep, span = g * 32;       // groups and slots of a warp
  const uint32_t inv = 65536u / g + 1u;                      // x / g = x * inv >> 16 for x < 320
  for (;;) {
    __syncthreads();
    if (tid == 0) sm.block = atomicAdd(p.ticket, 1);
    __syncthreads();
    const int32_t b = sm.block;
    if (b >= p.B) break;
    const uint32_t p0 = b ? p.pthist[(int64_t)b * p.pt_tiles - 1] : 0u, p1 = p.pthist[(int64_t)(b + 1) * p.pt_tiles - 1];
    const uint32_t q0 = b ? p.prhist[(int64_t)b * p.pr_tiles - 1] : 0u, q1 = p.prhist[(int64_t)(b + 1) * p.pr_tiles - 1];
    if (p0 == p1 || q0 == q1) continue;
    const uint32_t nt = (p1 - p0 + 31) / 32;
    for (uint32_t i = tid; i < p.m / 2; i += kSwThreads) reinterpret_cast<uint4*>(T0)[i] = make_uint4(0, 0, 0, 0);
    for (uint32_t i = tid; i < p.m / 32; i += kSwThreads) sm.T1[i] = 0;
    if (tid < kSwWarps) sm.W[tid] = 0;
    // the builder's points of a tile; past the end: at a time after every query
    auto load_point = [&](uint32_t k) -> uint4 {
      const uint32_t i = p0 + 32 * k + lane;
      return k < nt && i < p1 ? __ldg(p.pts + i) : make_uint4(kNone, kNone, 0u, 0u);
    };
    auto build = [&](uint32_t k, uint4 x, uint32_t next_first) {
      const int f = k & 1;
      int below = 0, at = 0;   // points with a smaller slot; its place among the sorted
#pragma unroll 8
      for (int i = 0; i < 32; ++i) {
        const uint32_t y = __shfl_sync(kAll, x.y, i);
        below += y < x.y;
        at += y < x.y || (y == x.y && i < lane);
      }
      sm.pt[f][lane] = x;
      sm.tm[f][lane] = x.x;
      sm.sorted[f][at] = x.y;
      if (lane == 0) sm.next_time[f] = next_first;
      uint64_t acc = 0;        // column lane + 1: points taken so far among the lane + 1 lowest slots
#pragma unroll 8
      for (int i = 0; i < 32; ++i) {
        const int r = __shfl_sync(kAll, below, i);
        const uint64_t d = ((uint64_t)__shfl_sync(kAll, x.w, i) << 32) | __shfl_sync(kAll, x.z, i);
        acc += r <= lane ? d : 0;
        sm.tab[f][i * 32 + lane] = acc;
      }
    };
    uint4 nx = make_uint4(0, 0, 0, 0), nx2 = nx;   // builder: tiles k + 1 and k + 2
    if (builder) {
      const uint4 x = load_point(0);
      nx = load_point(1);
      nx2 = load_point(2);
      build(0, x, __shfl_sync(kAll, nx.x, 0));
    }
    auto load_probe = [&](uint32_t i) -> uint2 {
      return !builder && i < q1 ? __ldg(p.prs + i) : make_uint2(0u, kNone);
    };
    uint32_t page = q0;
    uint2 pr = load_probe(page + tid), pn = load_probe(page + kSwPage + tid);
    bool done = pr.y == kNone;                       // (slots stay below 2^31 - 1)
    uint64_t t1 = 0, wtot = 0;                       // lane's group sum below, warp total
    __syncthreads();
    for (uint32_t k = 0; k < nt; ++k) {
      const int f = k & 1;
      const uint32_t limit = sm.next_time[f];
      uint64_t wpre = 0;                             // totals of the warps below `lane`
      if (!builder) {
        const uint64_t own = lane < kSwWarps ? sm.W[lane] : 0;
        wpre = own;
#pragma unroll
        for (int o = 1; o < kSwWarps; o <<= 1) {
          const uint64_t y = __shfl_up_sync(kAll, wpre, o);
          if (lane >= o) wpre += y;
        }
        wpre -= own;
      }
      bool more = true;
      for (bool first = true; more; first = false) {
        if (builder) {
          if (first && k + 1 < nt) {
            const uint4 x = nx;
            nx = nx2;
            nx2 = load_point(k + 3);
            build(k + 1, x, __shfl_sync(kAll, nx.x, 0));
          }
        } else {
          const bool in = !done && pr.x < limit;
          if (__any_sync(kAll, in)) {
            const uint32_t r = pr.y & 0x7fffffffu, rs = in ? r : 0u;
            const uint64_t w = __shfl_sync(kAll, wpre, (int)(((rs >> 5) * inv) >> 16));
            if (in) {
              uint64_t v = w + sm.T1[r >> 5] + T0[r];
              const int x = kb_below<false>(sm.tm[f], pr.x), y = kb_below<true>(sm.sorted[f], r);
              if (x && y) v += sm.tab[f][(x - 1) * 32 + y - 1];
              if (v) atomicAdd(p.acc + pr.x, (unsigned long long)((pr.y >> 31) ? (uint64_t)0 - v : v));
              done = true;
            }
          }
        }
        more = __syncthreads_and(builder || done);   // the whole page is answered
        if (more) {
          page += kSwPage;
          if (page >= q1) break;
          pr = pn;
          pn = load_probe(page + kSwPage + tid);
          done = pr.y == kNone;
        }
      }
      if (more) break;                               // no probes are left
      if (!builder) {                                // the tile's points into the prefixes
        const uint32_t s = sm.pt[f][lane].y;
        uint32_t hit = __ballot_sync(kAll, s - warp * span < span);
        if (hit) {
          do {
            const int i = __ffs(hit) - 1;
            hit &= hit - 1;
            const uint4 x = sm.pt[f][i];
            const uint64_t d = ((uint64_t)x.w << 32) | x.z;
            const uint32_t q = x.y & 31u;
            if (lane > (int)q) T0[(x.y & ~31u) + lane] += d;
            if (lane > (int)((x.y >> 5) - warp * g)) t1 += d;
            wtot += d;
            __syncwarp();
          } while (hit);
          if (lane < (int)g) sm.T1[warp * g + lane] = t1;
          if (lane == 0) sm.W[warp] = wtot;
        }
      }
      __syncthreads();
    }
  }
}

__global__ void __launch_bounds__(256) k_kb_answers(KbParams p) {
  if (*p.status) return;
  __shared__ int32_t s_c[2];
  const int64_t j0 = (int64_t)blockIdx.x * kKbPrTile, j1 = imin64(j0 + kKbPrTile, p.Q);
  kb_col_range(p, j0, j1, s_c);
  for (int64_t j = j0 + threadIdx.x; j < j1; j += blockDim.x) {
    const int32_t c = kb_find_col(p.coltime, s_c[0], s_c[1], (uint32_t)j);
    p.answers[p.qoff[p.colstate[c]] + (j - p.coltime[c])] = (int64_t)p.acc[j];
  }
}

inline size_t al256(size_t x) { return (x + 255) & ~size_t(255); }

// Workspace of the replay with blocks of k.m slots.
void kb_layout(const PipeSpec& s, KbSpec& k) {
  k.B = (int32_t)(s.E / k.m + 1);   // a bound past every event has slot E: its block is E / m
  k.segs = 8 * s.sms;
  k.pt_tiles = (2 * s.E + kKbPtTile - 1) / kKbPtTile;
  k.pr_tiles = (s.Q + kKbPrTile - 1) / kKbPrTile;
  const size_t S = (size_t)s.S, S2 = 2 * S, B = (size_t)k.B;
  const size_t cols = (size_t)std::min<int64_t>(s.S, s.Q);
  const size_t scan_n = std::max({S2, (size_t)s.Cmax + 1, B * (size_t)k.pt_tiles, B * (size_t)k.pr_tiles});
  size_t o = 0;
  auto take = [&](int i, size_t bytes) { k.off[i] = o; o = al256(o + bytes); };
  take(KB_SOFF, 8); take(KB_TEOFF, 16); take(KB_TQOFF, 16); take(KB_TC, 4); take(KB_TBOFF, 8); take(KB_TBITS, 8);
  take(KB_TCARRY, 8); take(KB_TGSUM, 8); take(KB_LASTQ, 4);
  take(KB_MISC, 256);
  take(KB_EOFF, (S + 1) * 8); take(KB_QOFF, (S + 1) * 8);
  take(KB_FORK, S * 4); take(KB_NEXT, S * 4); take(KB_CNT, S * 8); take(KB_EHEAD, S * 4); take(KB_XHEAD, S * 4);
  take(KB_RANK, S2 * 8);
  take(KB_SCAN, scan_tmp_bytes(scan_n));
  take(KB_STEP, S2 * 4); take(KB_W, S2 * 8); take(KB_EP, S2 * 8); take(KB_TIME, S2 * 4);
  take(KB_COLSTATE, cols * 4); take(KB_COLTIME, (cols + 1) * 4); take(KB_COLSTEP, cols * 4);
  take(KB_POS, ((size_t)s.Cmax + 2) * 4);
  take(KB_PTHIST, B * (size_t)k.pt_tiles * 4);
  take(KB_PTS, 2 * (size_t)s.E * 16);
  take(KB_SEG, (size_t)k.segs * B * 8);
  take(KB_ROWS, cols * B * 8);
  take(KB_PRHIST, B * (size_t)k.pr_tiles * 4);
  take(KB_PRS, 2 * (size_t)s.Q * 8);
  take(KB_ACC, (size_t)s.Q * 8);
  k.total = o;
}

// Shared-memory opt-ins, once per device (the largest request of each kernel).
int kb_attrs() {
  static std::mutex mu;
  static bool done[64] = {false};
  int dev = 0;
  int rc = report(cudaGetDevice(&dev), "cudaGetDevice");
  if (rc) return rc;
  std::lock_guard<std::mutex> g(mu);
  if (dev >= 0 && dev < 64 && done[dev]) return 0;
  const struct { const void* f; size_t bytes; } need[] = {
      {(const void*)k_kb_point_scatter, kb_scatter_smem(kKbMaxBlocks, kPtWarps)},
      {(const void*)k_kb_probe_scatter, kb_scatter_smem(kKbMaxBlocks, kPrWarps)},
      {(const void*)k_kb_rows, (size_t)kKbMaxBlocks * 16},
      {(const void*)k_kb_sweep, (size_t)kKbMaxSlots * 8}};
  for (const auto& n : need)
    if ((rc = report(cudaFuncSetAttribute(n.f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)n.bytes), "smem attr")))
      return rc;
  if (dev >= 0 && dev < 64) done[dev] = true;
  return 0;
}

}  // namespace

bool kb_select(const BwReplayArgs* a, const PipeSpec& s, size_t general_bytes, KbSpec& k) {
  if (s.T != 1 || s.Cmax <= kKbMinKeys || a->blocks > 0 || (a->flags & BW_REPLAY_GENERAL)) return false;
  if (s.E < 1 || s.Q < 1 || s.Q >= ((int64_t)1 << 30)) return false;
  k = KbSpec();
  k.S = s.S; k.C = s.Cmax; k.E = s.E; k.Q = s.Q;
  // about four blocks per sweep CTA (two CTAs an SM), larger ones where the rows would
  // not fit.  Never more scratch than twice the state-block pipeline's or 32 MiB, and nothing
  // that fits the allocation-free entry's 32 MiB there may outgrow them here.
  const size_t small = (size_t)32 << 20;
  const size_t limit = general_bytes > small ? 2 * general_bytes : small;
  int64_t steps = std::min<int64_t>(s.E / (8 * (int64_t)s.sms * kKbSlotStep) + 1, kKbMaxSlots / kKbSlotStep);
  for (; steps * kKbSlotStep <= kKbMaxSlots; ++steps) {
    k.m = (int32_t)steps * kKbSlotStep;
    if (s.E / k.m + 1 > kKbMaxBlocks) continue;
    kb_layout(s, k);
    if (k.total <= limit) return true;
  }
  return false;
}

const int32_t* kb_status_word(const KbSpec& k, const void* workspace) {
  return reinterpret_cast<const int32_t*>(static_cast<const char*>(workspace) + k.off[KB_MISC]) + M_STATUS;
}

int kb_enqueue(const KbSpec& k, const PipeSpec& s, const BwReplayArgs* a, EventSet* timing, int* kernels_out) {
  if ((reinterpret_cast<uintptr_t>(a->events) & 15u) != 0) {
    std::fprintf(stderr, "bw replay: events must be 16-byte aligned (got %p)\n", static_cast<const void*>(a->events));
    return BW_EINVAL;
  }
  cudaStream_t st = static_cast<cudaStream_t>(a->stream);
  char* ws = static_cast<char*>(a->workspace);
  auto at = [&](int i) { return ws + k.off[i]; };
  TourArrays ta;
  ta.tt.soff = (int32_t*)at(KB_SOFF); ta.tt.eoff = (int64_t*)at(KB_TEOFF); ta.tt.qoff = (int64_t*)at(KB_TQOFF);
  ta.tt.C = (uint32_t*)at(KB_TC); ta.tt.boff = (int32_t*)at(KB_TBOFF); ta.tt.bits = (int64_t*)at(KB_TBITS);
  ta.tt.carry = (int64_t*)at(KB_TCARRY); ta.tt.gsum = (int64_t*)at(KB_TGSUM); ta.tt.last_q = (int32_t*)at(KB_LASTQ);
  ta.misc = (int32_t*)at(KB_MISC); ta.eoff = (int64_t*)at(KB_EOFF); ta.qoff = (int64_t*)at(KB_QOFF);
  ta.gpar = nullptr; ta.fork_head = (int32_t*)at(KB_FORK); ta.next_sib = (int32_t*)at(KB_NEXT);
  ta.cnt = (int64_t*)at(KB_CNT); ta.ehead = (int32_t*)at(KB_EHEAD); ta.xhead = (int32_t*)at(KB_XHEAD);
  ta.rank = (uint64_t*)at(KB_RANK); ta.scan_tmp = (int64_t*)at(KB_SCAN);
  KbParams p;
  p.ev = a->events; p.qs = a->queries; p.answers = a->answers;
  p.eoff = ta.eoff; p.qoff = ta.qoff; p.rank = ta.rank; p.cnt = ta.cnt; p.ehead = ta.ehead; p.xhead = ta.xhead;
  p.step = (int32_t*)at(KB_STEP); p.w = (int64_t*)at(KB_W); p.ep = (int64_t*)at(KB_EP); p.time = (uint32_t*)at(KB_TIME);
  p.colstate = (int32_t*)at(KB_COLSTATE); p.coltime = (uint32_t*)at(KB_COLTIME); p.colstep = (int32_t*)at(KB_COLSTEP);
  p.pos = (uint32_t*)at(KB_POS); p.pthist = (uint32_t*)at(KB_PTHIST); p.pts = (uint4*)at(KB_PTS);
  p.seg = (uint64_t*)at(KB_SEG); p.rows = (int64_t*)at(KB_ROWS); p.prhist = (uint32_t*)at(KB_PRHIST);
  p.prs = (uint2*)at(KB_PRS); p.acc = (unsigned long long*)at(KB_ACC);
  p.status = ta.misc + M_STATUS; p.ticket = ta.misc + M_SWEEP_TICKET;
  p.E = k.E; p.Q = k.Q; p.pt_tiles = k.pt_tiles; p.pr_tiles = k.pr_tiles;
  p.S = k.S; p.B = k.B; p.segs = k.segs; p.C = k.C; p.m = (uint32_t)k.m;

  const size_t pt_smem = kb_scatter_smem(k.B, kPtWarps), pr_smem = kb_scatter_smem(k.B, kPrWarps);
  const size_t row_smem = (size_t)k.B * 16, sweep_smem = (size_t)k.m * 8;
  int rc = kb_attrs();
  if (rc) return rc;
  int kernels = 0;
  auto chk = [&](const char* what) { ++kernels; return report(cudaGetLastError(), what); };
  auto mark = [&](int i) { return timing ? report(cudaEventRecord(timing->ev[i], st), "event record") : 0; };
  const int grid = s.sms * 8;
  if (timing) timing->chain = 0;
  if ((rc = mark(0))) return rc;
  if ((rc = pipe_tour(s, false, ta, a->parent, a->events, a->queries, st, timing, kernels))) return rc;
  k_kb_steps<<<grid, 256, 0, st>>>(p);
  if ((rc = chk("k_kb_steps"))) return rc;
  if ((rc = device_inclusive_scan_i64(p.w, 2 * (int64_t)k.S, ta.scan_tmp, st, kernels))) return report((cudaError_t)rc, "scan");
  k_kb_cols<<<grid, 256, 0, st>>>(p);
  if ((rc = chk("k_kb_cols"))) return rc;
  if ((rc = device_inclusive_scan_i64(p.ep, 2 * (int64_t)k.S, ta.scan_tmp, st, kernels))) return report((cudaError_t)rc, "scan");
  if ((rc = mark(2))) return rc;
  if ((rc = report(cudaMemsetAsync(p.pos, 0, ((size_t)k.C + 1) * 4, st), "memset"))) return rc;
  k_kb_key_hist<<<grid, 256, 0, st>>>(p);
  if ((rc = chk("k_kb_key_hist"))) return rc;
  if ((rc = device_inclusive_scan<uint32_t>(p.pos, (int64_t)k.C + 1, ta.scan_tmp, st, kernels)))
    return report((cudaError_t)rc, "scan");
  if ((rc = mark(3))) return rc;
  k_kb_point_count<<<(unsigned)k.pt_tiles, kPtWarps * 32, (size_t)k.B * 4, st>>>(p);
  if ((rc = chk("k_kb_point_count"))) return rc;
  if ((rc = device_inclusive_scan<uint32_t>(p.pthist, (int64_t)k.B * k.pt_tiles, ta.scan_tmp, st, kernels)))
    return report((cudaError_t)rc, "scan");
  k_kb_point_scatter<<<(unsigned)k.pt_tiles, kPtWarps * 32, pt_smem, st>>>(p);
  if ((rc = chk("k_kb_point_scatter"))) return rc;
  if ((rc = mark(4))) return rc;
  k_kb_seg<<<k.segs, 256, (size_t)k.B * 8, st>>>(p);
  if ((rc = chk("k_kb_seg"))) return rc;
  k_kb_segscan<<<(k.B + 31) / 32, 1024, 0, st>>>(p);
  if ((rc = chk("k_kb_segscan"))) return rc;
  k_kb_rows<<<k.segs, 256, row_smem, st>>>(p);
  if ((rc = chk("k_kb_rows"))) return rc;
  if ((rc = mark(5))) return rc;
  k_kb_probe_count<<<(unsigned)k.pr_tiles, 512, (size_t)k.B * 4, st>>>(p);
  if ((rc = chk("k_kb_probe_count"))) return rc;
  if ((rc = device_inclusive_scan<uint32_t>(p.prhist, (int64_t)k.B * k.pr_tiles, ta.scan_tmp, st, kernels)))
    return report((cudaError_t)rc, "scan");
  k_kb_probe_scatter<<<(unsigned)k.pr_tiles, kPrWarps * 32, pr_smem, st>>>(p);
  if ((rc = chk("k_kb_probe_scatter"))) return rc;
  k_kb_sweep<<<std::min(k.B, 2 * s.sms), kSwThreads, sweep_smem, st>>>(p);
  if ((rc = chk("k_kb_sweep"))) return rc;
  k_kb_answers<<<(unsigned)k.pr_tiles, 256, 0, st>>>(p);
  if ((rc = chk("k_kb_answers"))) return rc;
  if ((rc = mark(6))) return rc;
  if (kernels_out) *kernels_out = kernels;
  return 0;
}

}  // namespace bw
