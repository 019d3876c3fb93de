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
//             segments of equal work (net sum per segment and block, then the running vector
//             in shared memory, written out scanned over the blocks at every column).
//   probes    k_kb_probe_count / scan / k_kb_probe_scatter   both bounds of every query
//             grouped by key block, in tour order; the whole-block part goes to acc.
//   sweep     k_kb_sweep   one CTA per key block: L of every probe (below).
//   answers   k_kb_answers  acc, kept in tour order, to the queries' own places.
//
// Measured on 20M events over 10M keys, 100k states and 100M range queries: 15.7 ms
// (sweep 6.9, probe scatter 3.9, rows 1.2, probe count 1.1, points 1.3) against 624 ms
// on the state-block pipeline.
#include <cuda_runtime.h>
#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <mutex>

#include "bw_gpu.h"
#include "bw_common.cuh"
#include "bw_pipeline.cuh"
#include "bw_keyblock.cuh"
#include "bw_search.cuh"

namespace bw {
namespace {

constexpr uint32_t kAll = 0xffffffffu;
constexpr uint32_t kNone = 0xffffffffu;

struct KbCut {
  int64_t j;            // points
  int64_t c;            // and columns before the segment
};

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
  uint4* tour;          // 2E: the points in tour order, {time, pos, delta}
  uint32_t *pthist, *ptoff;   // tiles x B digit counts (then starts), B + 1 block starts
  uint4* pts;           // the swept points by key block, {time, slot, delta}
  uint64_t* seg;        // segs x B
  KbCut* cut;           // segs + 1
  int64_t* rows;        // columns x Bs
  uint32_t *prhist, *proff;
  uint32_t* more;       // B + 1: parts of the key blocks before this one, beyond one each
  uint2* prs;           // {query in tour order, slot | lower bound << 31}
  unsigned long long* acc;   // per query in tour order
  const int32_t* status;
  int32_t* ticket;
  int64_t E, Q, pt_tiles, pr_tiles;
  int32_t S, B, Bs, segs;   // Bs: B rounded up to whole 32-byte sectors of a row
  uint32_t C, m, part;  // part: probes that a CTA of the sweep takes at a time (whole pages)
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
  return first_after(lo, hi, [&](int32_t t) { return ep[t] > j; });
}
// Last column in [lo, hi] with coltime <= j.
__device__ __forceinline__ int32_t kb_find_col(const uint32_t* coltime, int32_t lo, int32_t hi, uint32_t j) {
  while (lo < hi) {
    const int32_t mid = (lo + hi + 1) >> 1;
    if (coltime[mid] <= j) lo = mid; else hi = mid - 1;
  }
  return lo;
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

// ------------------------------------------------------------------ digit starts
// hist[tile][d] = items of digit d in the tile -> output position of the first of them
// (all items of smaller digits, then those of earlier tiles), off[d] = start of the
// digit, off[B] = all items.  Column sums and column prefixes over chunks of tiles, so
// that every access runs along the digits (a digit-major matrix cost a sector per count).
constexpr int kStartChunks = 64;
__device__ __forceinline__ void kb_chunk(int64_t tiles, int64_t& t0, int64_t& t1) {
  t0 = tiles * blockIdx.y / kStartChunks;
  t1 = tiles * (blockIdx.y + 1) / kStartChunks;
}
__global__ void __launch_bounds__(128) k_kb_start_sum(const uint32_t* __restrict__ hist, int32_t B, int64_t tiles,
                                                      uint32_t* __restrict__ part, const int32_t* status) {
  const int32_t d = blockIdx.x * 128 + threadIdx.x;
  if (*status || d >= B) return;
  int64_t t0, t1;
  kb_chunk(tiles, t0, t1);
  uint32_t s = 0;
#pragma unroll 8
  for (int64_t t = t0; t < t1; ++t) s += hist[t * B + d];
  part[(int64_t)blockIdx.y * B + d] = s;
}
// `more` (probes): the parts of `per` items that each digit takes beyond its first, as starts.
__global__ void __launch_bounds__(1024) k_kb_start_scan(uint32_t* part, int32_t B, uint32_t* off, uint32_t* more,
                                                        uint32_t per, const int32_t* status) {
  if (*status) return;
  uint32_t carry = 0, parts = 0;
  for (int32_t d0 = 0; d0 < B; d0 += 1024) {
    const int32_t d = d0 + threadIdx.x;
    uint32_t n = 0, total = 0;
    if (d < B) {
#pragma unroll 8
      for (int c = 0; c < kStartChunks; ++c) n += part[(int64_t)c * B + d];
    }
    uint32_t run = carry + block_exclusive_scan<uint32_t>(n, &total);
    if (d < B) {
      off[d] = run;
#pragma unroll 8
      for (int c = 0; c < kStartChunks; ++c) {
        const uint32_t x = part[(int64_t)c * B + d];
        part[(int64_t)c * B + d] = run;
        run += x;
      }
    }
    carry += total;
    if (more) {
      const uint32_t before = block_exclusive_scan<uint32_t>(n ? (n - 1) / per : 0, &total);
      if (d < B) more[d] = parts + before;
      parts += total;
    }
  }
  if (threadIdx.x == 0) {
    off[B] = carry;
    if (more) more[B] = parts;
  }
}
__global__ void __launch_bounds__(128) k_kb_start_apply(uint32_t* __restrict__ hist, int32_t B, int64_t tiles,
                                                        const uint32_t* __restrict__ part, const int32_t* status) {
  const int32_t d = blockIdx.x * 128 + threadIdx.x;
  if (*status || d >= B) return;
  int64_t t0, t1;
  kb_chunk(tiles, t0, t1);
  uint32_t run = part[(int64_t)blockIdx.y * B + d];
  for (int64_t t = t0; t < t1; t += 16) {   // in place: a batch is loaded before it is written
    uint32_t x[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) x[i] = t + i < t1 ? hist[(t + i) * B + d] : 0u;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      if (t + i < t1) hist[(t + i) * B + d] = run;
      run += x[i];
    }
  }
}

// ------------------------------------------------------------------ points
// An event of the last key of its key block lies below no probe of the block: it
// counts in the rows only (which also keeps a hot key out of the sweep).
__device__ __forceinline__ bool kb_swept(const KbParams& p, uint32_t key, uint32_t b) { return p.pos[key + 1] / p.m == b; }
constexpr uint32_t kRowsOnly = 0x80000000u;   // in a tour point's pos (positions stay below 2^31)

// The points of a tile, written out in tour order, and the swept ones counted by block.
__global__ void __launch_bounds__(256) k_kb_points(KbParams p) {
  if (*p.status) return;
  extern __shared__ __align__(16) uint32_t h[];
  __shared__ int32_t s_t[2];
  for (int32_t i = threadIdx.x; i < p.B; i += blockDim.x) h[i] = 0;
  __syncthreads();
  const int64_t j0 = (int64_t)blockIdx.x * kKbPtTile, j1 = imin64(j0 + kKbPtTile, kb_points(p));
  if (j0 < j1) {
    kb_step_range(p, j0, j1, s_t);
    const int32_t ta = s_t[0], tz = s_t[1];
#pragma unroll 4
    for (int64_t j = j0 + threadIdx.x; j < j1; j += 256) {
      const int32_t t = kb_find_step(p.ep, ta, tz, j);
      const int32_t v = p.step[t], s = v < 0 ? ~v : v;
      const uint4 e = __ldg(reinterpret_cast<const uint4*>(p.ev) + (p.eoff[s + 1] - (p.ep[t] - j)));
      const uint64_t d = ((uint64_t)e.w << 32) | e.z, sd = v < 0 ? (uint64_t)0 - d : d;
      const uint32_t ps = p.pos[e.y], b = ps / p.m;
      const bool swept = kb_swept(p, e.y, b);
      if (swept) atomicAdd(h + b, 1u);
      p.tour[j] = make_uint4(p.time[t], ps | (swept ? 0u : kRowsOnly), (uint32_t)sd, (uint32_t)(sd >> 32));
    }
  }
  __syncthreads();
  for (int32_t d = threadIdx.x; d < p.B; d += blockDim.x) p.pthist[(int64_t)blockIdx.x * p.B + d] = h[d];
}

// Stable scatter by key block: four warps, 1,024 consecutive points each, ranked by
// ballots over the digit's bits (__match_any_sync took some 400 cycles with 32 distinct
// digits) in per-warp counters.
constexpr int kPtWarps = 4, kPtRounds = kKbPtTile / (kPtWarps * 32);
inline size_t kb_scatter_smem(int32_t B) { return (size_t)((B + 3) & ~3) * 4 + (size_t)kPtWarps * ((B + 7) & ~7) * 2; }
__global__ void __launch_bounds__(kPtWarps * 32, 10) k_kb_point_scatter(KbParams p, int bits) {
  if (*p.status) return;
  extern __shared__ __align__(16) uint32_t base[];
  const int32_t Bp = (p.B + 7) & ~7;
  uint16_t* wall = reinterpret_cast<uint16_t*>(base + ((p.B + 3) & ~3));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint16_t* wc = wall + warp * Bp;
  const unsigned lt = (1u << lane) - 1u;
  const int64_t j0 = (int64_t)blockIdx.x * kKbPtTile, j1 = imin64(j0 + kKbPtTile, kb_points(p));
  if (j0 >= j1) return;
  for (int32_t i = threadIdx.x; i < kPtWarps * Bp / 8; i += blockDim.x) reinterpret_cast<uint4*>(wall)[i] = make_uint4(0, 0, 0, 0);
  for (int32_t i = threadIdx.x; i < p.B; i += blockDim.x) base[i] = p.pthist[(int64_t)blockIdx.x * p.B + i];
  __syncthreads();
  const int64_t w0 = j0 + warp * (kPtRounds * 32) + lane;
  uint32_t r[kPtRounds / 2];   // rank inside the warp, two rounds a word
  uint32_t batch[8];           // positions of the next rounds, read ahead of the ranking
#pragma unroll
  for (int i = 0; i < kPtRounds; ++i) {
    if (i % 8 == 0) {
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const int64_t j = w0 + (i + k) * 32;
        batch[k] = j < j1 ? __ldg(&p.tour[j].y) : kRowsOnly;
      }
    }
    const uint32_t ps = batch[i % 8];
    const bool in = !(ps & kRowsOnly);
    const uint32_t d = ps / p.m;
    unsigned peers = __ballot_sync(kAll, in);
    for (int k = 0; k < bits; ++k) {
      const bool one = (d >> k) & 1u;
      const unsigned m = __ballot_sync(kAll, one);
      peers &= one ? m : ~m;
    }
    const uint32_t old = in ? wc[d] : 0u;
    __syncwarp();
    const uint32_t rk = old + __popc(peers & lt);
    if (i & 1) r[i / 2] |= rk << 16; else r[i / 2] = rk;
    if (in && (peers & lt) == 0) wc[d] = (uint16_t)(old + __popc(peers));
    __syncwarp();
  }
  __syncthreads();
  for (int32_t d = threadIdx.x; d < p.B; d += blockDim.x) {
    uint32_t run = 0;
#pragma unroll
    for (int w = 0; w < kPtWarps; ++w) {
      const uint32_t c = wall[w * Bp + d];
      wall[w * Bp + d] = (uint16_t)run;
      run += c;
    }
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kPtRounds; ++i) {
    const int64_t j = w0 + i * 32;
    if (j >= j1) continue;
    uint4 x = __ldg(p.tour + j);
    if (x.y & kRowsOnly) continue;
    const uint32_t d = x.y / p.m;
    x.y -= d * p.m;
    p.pts[(size_t)base[d] + wc[d] + ((r[i / 2] >> (16 * (i & 1))) & 0xffffu)] = x;
  }
}

// ------------------------------------------------------------------ rows
__device__ __forceinline__ void kb_add_points(const KbParams& p, unsigned long long* vec, int64_t j0, int64_t j1) {
#pragma unroll 4
  for (int64_t j = j0 + threadIdx.x; j < j1; j += blockDim.x) {
    const uint4 x = __ldg(p.tour + j);
    shared_add_u64(vec + (x.y & ~kRowsOnly) / p.m, ((uint64_t)x.w << 32) | x.z);
  }
}
// Segment g of the tour: an equal share of points and columns, a column counted as
// kColPoints points (each column of a segment is written out in turn, some 0.6 us and more; cut by
// points alone, the columns of 74,000 states with 12 events met in a dozen CTAs and the
// rows took 11 ms).  The walk takes a column once all points up to its enter step are
// taken.  Whole warp.
constexpr int64_t kColPoints = 256;
__device__ __forceinline__ KbCut kb_cut(const KbParams& p, int32_t g, int lane) {
  const int32_t nc = kb_columns(p);
  const int64_t np = kb_points(p), total = np + kColPoints * nc;
  const int64_t d = total / p.segs * g + total % p.segs * g / p.segs;
  int32_t lo = 0, hi = nc;   // the columns wholly before the cut, 32 probes a round
  while (lo < hi) {
    const int32_t step = (hi - lo + 31) / 32, c = lo + lane * step;   // (columns stay below 2^30)
    const int n = __popc(__ballot_sync(kAll, c < hi && p.ep[p.colstep[c]] + kColPoints * ((int64_t)c + 1) <= d));
    if (!n) break;
    const int32_t last = lo + (n - 1) * step;
    hi = n < 32 && last + step < hi ? last + step : hi;
    lo = last + 1;
  }
  return KbCut{min(d - kColPoints * lo, lo < nc ? p.ep[p.colstep[lo]] : np), lo};
}

// The cuts, and the net delta of every segment in every key block.
__global__ void __launch_bounds__(512) k_kb_seg(KbParams p) {
  if (*p.status) return;
  extern __shared__ __align__(16) unsigned long long vec[];
  __shared__ int64_t s_j[2];
  for (int32_t i = threadIdx.x; i < p.B; i += blockDim.x) vec[i] = 0;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (warp < 2) {
    const KbCut x = kb_cut(p, blockIdx.x + warp, lane);
    if (lane == 0) {
      s_j[warp] = x.j;
      if (warp == 0 || blockIdx.x + 1 == (unsigned)p.segs) p.cut[blockIdx.x + warp] = x;
    }
  }
  __syncthreads();
  kb_add_points(p, vec, s_j[0], s_j[1]);
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

// A segment's columns: the running vector over the key blocks (shared memory) takes
// the points up to the column and is written out scanned, four entries a thread and
// pass.  Two barriers a column: the vector is complete; the warps' sums are written
// (and the vector read, so that the next column's points may follow).
constexpr int kRowThreads = 512;
__global__ void __launch_bounds__(kRowThreads, 3) k_kb_rows(KbParams p) {
  if (*p.status) return;
  extern __shared__ __align__(16) unsigned long long vec[];   // Bs
  __shared__ uint64_t s_sum[2][2][kRowThreads / 32];          // by column parity and pass
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int32_t i = threadIdx.x; i < p.Bs; i += kRowThreads) vec[i] = i < p.B ? p.seg[(size_t)blockIdx.x * p.B + i] : 0;
  __syncthreads();
  int64_t j = p.cut[blockIdx.x].j;
  const int32_t c0 = (int32_t)p.cut[blockIdx.x].c, c1 = (int32_t)p.cut[blockIdx.x + 1].c;
  for (int32_t c = c0; c < c1; ++c) {
    const int64_t je = p.ep[p.colstep[c]];
    kb_add_points(p, vec, j, je);
    j = je;
    __syncthreads();
    uint64_t v[2][4], ex[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {   // entries 4 tid .. 4 tid + 3, and 2,048 further on
      const int32_t i = h * 4 * kRowThreads + 4 * threadIdx.x;
      ex[h] = 0;
      if (h * 4 * kRowThreads >= p.Bs) continue;
#pragma unroll
      for (int k = 0; k < 4; ++k) v[h][k] = i < p.Bs ? vec[i + k] : 0;
      const uint64_t s = v[h][0] + v[h][1] + v[h][2] + v[h][3];
      uint64_t incl = s;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint64_t y = __shfl_up_sync(kAll, incl, o);
        if (lane >= o) incl += y;
      }
      ex[h] = incl - s;
      if (lane == 31) s_sum[c & 1][h][warp] = incl;
    }
    __syncthreads();
    uint64_t run0 = 0;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int32_t i = h * 4 * kRowThreads + 4 * threadIdx.x;
      if (h * 4 * kRowThreads >= p.Bs) continue;
      uint64_t w = lane < kRowThreads / 32 ? s_sum[c & 1][h][lane] : 0;
#pragma unroll
      for (int o = 1; o < kRowThreads / 32; o <<= 1) {
        const uint64_t y = __shfl_up_sync(kAll, w, o);
        if (lane >= o) w += y;
      }
      const uint64_t below = __shfl_sync(kAll, w, warp ? warp - 1 : 0);
      uint64_t a = run0 + (warp ? below : 0) + ex[h];
      run0 += __shfl_sync(kAll, w, kRowThreads / 32 - 1);
      if (i < p.Bs) {
        int64_t* row = p.rows + (size_t)c * p.Bs + i;
        const uint64_t b1 = a + v[h][0], b2 = b1 + v[h][1], b3 = b2 + v[h][2];
        reinterpret_cast<longlong2*>(row)[0] = make_longlong2((int64_t)a, (int64_t)b1);
        reinterpret_cast<longlong2*>(row)[1] = make_longlong2((int64_t)b2, (int64_t)b3);
      }
    }
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
  const int32_t ca = s_c[0], cz = s_c[1];
#pragma unroll 4
  for (int64_t j = j0 + threadIdx.x; j < j1; j += 512) {
    const int32_t c = kb_find_col(p.coltime, ca, cz, (uint32_t)j);
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
  __syncthreads();
  for (int32_t d = threadIdx.x; d < p.B; d += blockDim.x) p.prhist[(int64_t)blockIdx.x * p.B + d] = h[d];
}

// Scatter by key block in rounds of 256 queries (at most 512 probes of a block): rounds
// are in tour order, the probes of one round in any -- the sweep looks one page of 512
// ahead.  acc becomes the part of the answer in whole key blocks.  Bound by the random
// sectors of its stores and row reads (4.2 ms for 200M probes; 5.2 ms with stable ranks
// from __match_any_sync).
// Four CTAs an SM, by their shared memory: the tiles at work write to a sector in every key
// block each, and those of eight CTAs an SM do not stay in the L2 until they are full
// (2,442 key blocks: eight CTAs 12.60 ms for the probes and the sweep, five 12.34, four
// 12.32, two 12.6).
constexpr int kPrThreads = 256;
constexpr size_t kPrSmem = (size_t)56 << 10;
__global__ void __launch_bounds__(kPrThreads) k_kb_probe_scatter(KbParams p) {
  if (*p.status) return;
  extern __shared__ __align__(16) uint32_t next[];
  __shared__ int32_t s_c[2];
  const int64_t j0 = (int64_t)blockIdx.x * kKbPrTile, j1 = imin64(j0 + kKbPrTile, p.Q);
  for (int32_t i = threadIdx.x; i < p.B; i += kPrThreads) next[i] = p.prhist[(int64_t)blockIdx.x * p.B + i];
  kb_col_range(p, j0, j1, s_c);
  const int32_t ca = s_c[0], cz = s_c[1];
  auto load = [&](int64_t j) -> unsigned long long { return j < j1 ? p.acc[j] : 0; };
  // the row entries of a query's bounds, requested a round before they are subtracted
  auto rows = [&](int64_t j, unsigned long long az, int64_t& ra, int64_t& rz) {
    const uint32_t ba = (uint32_t)az / p.m, bz = (uint32_t)(az >> 32) / p.m;
    ra = rz = 0;
    if (ba != bz) {
      const int64_t* row = p.rows + (size_t)kb_find_col(p.coltime, ca, cz, (uint32_t)j) * p.Bs;
      ra = __ldg(row + ba);
      rz = __ldg(row + bz);
    }
  };
  int64_t j = j0 + threadIdx.x, ra, rz;
  unsigned long long az = load(j), n1 = load(j + kPrThreads);
  rows(j, az, ra, rz);
  for (int64_t r0 = j0; r0 < j1; r0 += kPrThreads, j += kPrThreads) {
    const unsigned long long n2 = load(j + 2 * kPrThreads);
    int64_t na, nz;
    rows(j + kPrThreads, n1, na, nz);   // (past the tile: an empty query)
    const uint32_t a = (uint32_t)az, z = (uint32_t)(az >> 32);
    if (a != z) {
      const uint32_t ba = a / p.m, bz = z / p.m, sa = a - ba * p.m, sz = z - bz * p.m;
      if (sa) p.prs[atomicAdd(next + ba, 1u)] = make_uint2((uint32_t)j, sa | 0x80000000u);
      if (sz) p.prs[atomicAdd(next + bz, 1u)] = make_uint2((uint32_t)j, sz);
    }
    if (j < j1) p.acc[j] = (uint64_t)rz - (uint64_t)ra;
    az = n1; n1 = n2; ra = na; rz = nz;
    __syncthreads();
  }
}

// ------------------------------------------------------------------ sweep
// One key block at a time per CTA, or a part of its probes where it has many more than an
// equal share (a key that most queries name, intervals over the whole domain, few key blocks): every part replays
// the block's points from the first on, which costs it the tiles' barriers, so a part is
// 32 probes a slot and more (half the time of its probes).  30,000 states, 1M events over 300,000
// keys, 5M queries: all on one key 21.6 -> 0.84 ms a replay, all over the whole domain 10.2 ->
// 0.80, uniform 1.18 -> 1.12; 100,000 states, 20M events over 10M keys, 50M Zipf point queries 56 ->
// 11.3, uniform 11.9; 300 states, 1,000 events (two key blocks) over 262,145 keys, 3M queries 6.2 -> 0.39.
// (Parts of half an equal share whatever the slots: 10M events, 5M queries, Zipf keys 4.76 -> 5.04.)
//
// The block's points (signed deltas at slots) and probes
// (prefixes over the slots), both in tour order.  The points before the current tile
// of 32 are held as a prefix structure over the slots: T0[s] = sum of the slots below s
// in s's group of 32, T1 = sum of the groups below.  A probe reads one of each and adds
// the tile's own points before it in time and below it by slot (32 broadcast reads,
// four in flight).  After the tile's probes the sixteen warps apply its points without
// atomics: the 32 lanes of the warp that owns the group add to T0's tail of it (an entry
// is always the same lane's), T1 stays in registers, a lane per group, and takes the
// points of lower ranges as one warp sum.
//
// Bound by instruction issue (58 % of the slots) and the two barriers a tile.  On 20M
// events over 10M keys with 100M range queries (1.25M tiles, 200M probes) the sweep takes
// 6.9 ms; with a table of each tile's corrections, built by one or two warps of their own
// while the tile before it was probed, it took 12 to 14.4 ms (the builders' dependent
// chains ran 2,400 cycles and more a tile), with one 32-step loop a probe and a
// seventeenth warp 8.4 ms (17 warps leave 32 registers a thread at three CTAs an SM).
constexpr int kSwWarps = 16, kSwThreads = kSwWarps * 32;
constexpr int kSwRing = 8;                   // tiles of points in shared memory
struct KbSweepSmem {
  uint4 pt[kSwRing][32];                     // by tile mod kSwRing: {time, slot, delta}
  unsigned long long T1[kKbMaxSlots / 32];
  int32_t block;
  uint32_t part;
};
__device__ __forceinline__ void kb_copy16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
// Sum over the warp, modulo 2^64, in three 32-bit reductions (32 values of 24 bits fit).
__device__ __forceinline__ uint64_t kb_warp_sum(uint64_t v) {
  const uint32_t a = __reduce_add_sync(kAll, (uint32_t)v & 0xffffffu);
  const uint32_t b = __reduce_add_sync(kAll, (uint32_t)(v >> 24) & 0xffffffu);
  const uint32_t c = __reduce_add_sync(kAll, (uint32_t)(v >> 48));
  return (uint64_t)a + ((uint64_t)b << 24) + ((uint64_t)c << 48);
}

// v += the point's delta when it lies at or before time tm and below slot r (two
// predicated adds; a select of the 64-bit delta and an add took twice as many).
__device__ __forceinline__ void kb_add_if(uint64_t& v, const uint4& x, uint32_t tm, uint32_t r) {
  uint32_t lo = (uint32_t)v, hi = (uint32_t)(v >> 32);
  asm("{\n\t.reg .pred q;\n\tsetp.le.u32 q, %2, %3;\n\tsetp.lt.and.u32 q, %4, %5, q;\n\t"
      "@q add.cc.u32 %0, %0, %6;\n\t@q addc.u32 %1, %1, %7;\n\t}"
      : "+r"(lo), "+r"(hi)
      : "r"(x.x), "r"(tm), "r"(x.y), "r"(r), "r"(x.z), "r"(x.w));
  v = ((uint64_t)hi << 32) | lo;
}

__global__ void __launch_bounds__(kSwThreads, kSwCtas) k_kb_sweep(KbParams p) {
  if (*p.status) return;
  extern __shared__ __align__(16) unsigned long long T0[];   // m slots
  __shared__ KbSweepSmem sm;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bool copier = warp == kSwWarps - 1;
  const uint32_t g = p.m / kKbSlotStep, span = g * 32, first = warp * span;   // groups, slots, first slot of a warp
  for (;;) {
    __syncthreads();
    if (tid == 0) {
      // the blocks' first parts, then the others
      int32_t b = atomicAdd(p.ticket, 1);
      uint32_t part = 0;
      if (b >= p.B) {
        const uint32_t e = (uint32_t)(b - p.B);
        b = p.B;
        if (e < p.more[p.B]) {
          b = first_after(0, p.B, [&](int32_t x) { return p.more[x + 1] > e; });
          part = 1 + e - p.more[b];
        }
      }
      sm.block = b;
      sm.part = part;
    }
    __syncthreads();
    const int32_t b = sm.block;
    if (b >= p.B) break;
    const uint32_t p0 = p.ptoff[b], p1 = p.ptoff[b + 1];
    uint32_t page = p.proff[b] + sm.part * p.part;
    const uint32_t q1 = min(p.proff[b + 1], page + p.part);   // (probes stay below 2^31, parts below 2^30)
    if (p0 == p1 || page == q1) continue;
    const uint32_t nt = (p1 - p0 + 31) / 32;
    for (uint32_t i = tid; i < p.m / 2; i += kSwThreads) reinterpret_cast<uint4*>(T0)[i] = make_uint4(0, 0, 0, 0);
    for (uint32_t i = tid; i < p.m / 32; i += kSwThreads) sm.T1[i] = 0;
    // a tile's points (a missing one: at a time after every query, above every slot)
    auto copy_points = [&](uint32_t k) {
      const uint32_t i = p0 + 32 * k + lane;
      uint4* at = &sm.pt[k % kSwRing][lane];
      if (k < nt && i < p1) kb_copy16(at, p.pts + i);
      else *at = make_uint4(kNone, kNone, 0u, 0u);
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    if (copier) {
      for (uint32_t k = 0; k < kSwRing - 1; ++k) copy_points(k);
      asm volatile("cp.async.wait_group %0;" ::"n"(kSwRing - 3) : "memory");   // tiles 0 and 1 have landed
    }
    auto load_probe = [&](uint32_t i) -> uint2 { return i < q1 ? __ldg(p.prs + i) : make_uint2(0u, kNone); };
    // this thread's probe of the page, of the next one and of the one after
    uint2 pr = load_probe(page + tid), pn = load_probe(page + kSwThreads + tid),
          pl = load_probe(page + 2 * kSwThreads + tid);
    bool done = pr.y == kNone, donen = pn.y == kNone;   // (slots stay below 2^31 - 1)
    uint64_t t1 = 0;                                    // T1 of the warp's group `lane`
    __syncthreads();
    for (uint32_t k = 0; k < nt; ++k) {
      const uint4* pt = sm.pt[k % kSwRing];
      const uint32_t limit = sm.pt[(k + 1) % kSwRing][0].x;
      bool more = true;
      while (more) {
        // the page's and the next page's probes of the tile (the order is loose within a page)
        auto answer = [&](const uint2& q, bool& fin) {
          const bool in = !fin && q.x < limit;
          if (!__any_sync(kAll, in)) return;
          const uint32_t r = in ? q.y & 0x7fffffffu : 0u, tm = in ? q.x : 0u;
          const uint32_t last = __reduce_max_sync(kAll, tm);
          uint64_t v = sm.T1[r >> 5] + T0[r];
#pragma unroll 1
          for (int i = 0; i < 32; i += 4) {   // four reads in flight, up to the warp's last probe in time
            uint4 x[4];
#pragma unroll
            for (int h = 0; h < 4; ++h) x[h] = pt[i + h];
#pragma unroll
            for (int h = 0; h < 4; ++h) kb_add_if(v, x[h], tm, r);
            if (x[3].x > last) break;
          }
          if (in && v) atomicAdd(p.acc + q.x, (unsigned long long)((q.y >> 31) ? (uint64_t)0 - v : v));
          fin |= in;
        };
        answer(pr, done);
        answer(pn, donen);
        more = __syncthreads_and(done);              // the whole page is answered
        if (more) {
          page += kSwThreads;
          if (page >= q1) break;
          pr = pn;
          done = donen;
          pn = pl;
          donen = pn.y == kNone;
          pl = load_probe(page + 2 * kSwThreads + tid);
        }
      }
      if (more) break;                               // no probes are left
      if (copier) copy_points(k + kSwRing - 1);      // into the place of tile k - 1
      const uint4 mine = pt[lane];
      uint32_t hit = __ballot_sync(kAll, mine.y - first < span);
      t1 += kb_warp_sum(mine.y < first ? ((uint64_t)mine.w << 32) | mine.z : 0);
      while (hit) {
        const uint4 x = pt[__ffs(hit) - 1];
        hit &= hit - 1;
        const uint64_t d = ((uint64_t)x.w << 32) | x.z;
        if (lane > (int)(x.y & 31u)) T0[(x.y & ~31u) + lane] += d;
        if (lane > (int)((x.y - first) >> 5)) t1 += d;
      }
      if (lane < (int)g) sm.T1[warp * g + lane] = t1;
      if (copier) asm volatile("cp.async.wait_group %0;" ::"n"(kSwRing - 3) : "memory");   // tiles k + 1 and k + 2
      __syncthreads();
    }
    if (copier) asm volatile("cp.async.wait_all;" ::: "memory");   // before the ring is used again
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
  k.segs = 3 * s.sms;   // one wave of the row pass (three CTAs an SM)
  k.pt_tiles = (2 * s.E + kKbPtTile - 1) / kKbPtTile;
  k.pr_tiles = (s.Q + kKbPrTile - 1) / kKbPrTile;
  const size_t S = (size_t)s.S, S2 = 2 * S, B = (size_t)k.B;
  const size_t cols = (size_t)std::min<int64_t>(s.S, s.Q);
  const size_t scan_n = std::max(S2, (size_t)s.Cmax + 1);
  size_t o = 0;
  auto take = [&](int i, size_t bytes) { k.off[i] = o; o = al256(o + bytes); };
  take(KB_SOFF, 8); take(KB_TEOFF, 16); take(KB_TQOFF, 16); take(KB_TC, 4); take(KB_TBOFF, 8); take(KB_TBITS, 8);
  take(KB_TCARRY, 8); take(KB_TGSUM, 8); take(KB_LASTQ, 4); take(KB_TTOFF, 8);
  take(KB_MISC, 256);
  take(KB_EOFF, (S + 1) * 8); take(KB_QOFF, (S + 1) * 8);
  take(KB_FORK, S * 4); take(KB_NEXT, S * 4); take(KB_CNT, S * 8); take(KB_EHEAD, S * 4); take(KB_XHEAD, S * 4);
  take(KB_RANK, S2 * 8);
  take(KB_SCAN, scan_tmp_bytes(scan_n));
  take(KB_STEP, S2 * 4); take(KB_W, S2 * 8); take(KB_EP, S2 * 8); take(KB_TIME, S2 * 4);
  take(KB_COLSTATE, cols * 4); take(KB_COLTIME, (cols + 1) * 4); take(KB_COLSTEP, cols * 4);
  take(KB_POS, ((size_t)s.Cmax + 2) * 4);
  take(KB_TOUR, 2 * (size_t)s.E * 16);
  take(KB_PTHIST, B * (size_t)k.pt_tiles * 4);
  take(KB_PTOFF, (B + 1) * 4);
  take(KB_PTS, 2 * (size_t)s.E * 16);
  take(KB_SEG, (size_t)k.segs * B * 8);
  take(KB_CUT, ((size_t)k.segs + 1) * sizeof(KbCut));
  take(KB_ROWS, cols * ((B + 3) & ~(size_t)3) * 8);
  take(KB_PRHIST, B * (size_t)k.pr_tiles * 4);
  take(KB_PROFF, (B + 1) * 4);
  take(KB_MORE, (B + 1) * 4);
  take(KB_PART, kStartChunks * B * 4);
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
      {(const void*)k_kb_point_scatter, kb_scatter_smem(kKbMaxBlocks)},
      {(const void*)k_kb_probe_scatter, kPrSmem},
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
  // Work for one or two state blocks and a domain of few windows: the state-block path has
  // fewer kernels and no pass over the domain; its time goes by the query steps and events of every
  // window (300 states, 1,000 events, 100 queries, us a replay, state blocks / key blocks:
  // 262,145 keys 113 / 229, 1M 156 / 245, 2M 215 / 246, 4M 337 / 235; 71 states, 25 events, 2,558
  // queries, 880,418 keys 480 / 226).
  const int64_t windows = ((int64_t)s.Cmax + kKbMinKeys - 1) / kKbMinKeys;
  if (est_work(s.S, s.E, s.Q) < 2 * kMinWork &&
      windows * (600 + 4 * std::min<int64_t>(s.Q, 100 * (int64_t)s.S) + s.E / 2) < 9000)
    return false;
  k = KbSpec();
  k.S = s.S; k.C = s.Cmax; k.E = s.E; k.Q = s.Q;
  // About four blocks per sweep CTA, larger ones where the rows would
  // not fit.  Never more scratch than twice the state-block pipeline's or 32 MiB, and nothing
  // that fits the allocation-free entry's 32 MiB there may outgrow them here.
  const size_t small = (size_t)32 << 20;
  const size_t limit = general_bytes > small ? 2 * general_bytes : small;
  int64_t steps = std::min<int64_t>(s.E / (4 * kSwCtas * (int64_t)s.sms * kKbSlotStep) + 1, kKbMaxSlots / kKbSlotStep);
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

int kb_enqueue(const KbSpec& k, const PipeSpec& spec, const BwReplayArgs* a, EventSet* timing, int* kernels_out) {
  PipeSpec s = spec;
  s.contract = false;   // columns and points are taken from the states themselves
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
  ta.tt.noff = ta.tt.soff; ta.tt.toff = (int32_t*)at(KB_TTOFF);
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
  p.tour = (uint4*)at(KB_TOUR); p.ptoff = (uint32_t*)at(KB_PTOFF); p.proff = (uint32_t*)at(KB_PROFF);
  p.more = (uint32_t*)at(KB_MORE);
  p.seg = (uint64_t*)at(KB_SEG); p.cut = (KbCut*)at(KB_CUT); p.rows = (int64_t*)at(KB_ROWS); p.prhist = (uint32_t*)at(KB_PRHIST);
  p.prs = (uint2*)at(KB_PRS); p.acc = (unsigned long long*)at(KB_ACC);
  p.status = ta.misc + M_STATUS; p.ticket = ta.misc + M_SWEEP_TICKET;
  p.E = k.E; p.Q = k.Q; p.pt_tiles = k.pt_tiles; p.pr_tiles = k.pr_tiles;
  p.S = k.S; p.B = k.B; p.Bs = (k.B + 3) & ~3; p.segs = k.segs; p.C = k.C; p.m = (uint32_t)k.m;
  const int64_t ctas = (int64_t)kSwCtas * s.sms;
  p.part = (uint32_t)(std::max<int64_t>(32 * k.m, k.Q / ctas) / kSwThreads + 1) * kSwThreads;

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
  uint32_t* part = (uint32_t*)at(KB_PART);
  auto starts = [&](uint32_t* hist, int64_t tiles, uint32_t* off, uint32_t* more) -> int {
    const dim3 g((unsigned)((k.B + 127) / 128), kStartChunks);
    k_kb_start_sum<<<g, 128, 0, st>>>(hist, k.B, tiles, part, p.status);
    if ((rc = chk("k_kb_start_sum"))) return rc;
    k_kb_start_scan<<<1, 1024, 0, st>>>(part, k.B, off, more, p.part, p.status);
    if ((rc = chk("k_kb_start_scan"))) return rc;
    k_kb_start_apply<<<g, 128, 0, st>>>(hist, k.B, tiles, part, p.status);
    return chk("k_kb_start_apply");
  };
  int bits = 1;
  while ((1 << bits) < k.B) ++bits;
  k_kb_points<<<(unsigned)k.pt_tiles, 256, (size_t)k.B * 4, st>>>(p);
  if ((rc = chk("k_kb_points"))) return rc;
  if ((rc = starts(p.pthist, k.pt_tiles, p.ptoff, nullptr))) return rc;
  k_kb_point_scatter<<<(unsigned)k.pt_tiles, kPtWarps * 32, kb_scatter_smem(k.B), st>>>(p, bits);
  if ((rc = chk("k_kb_point_scatter"))) return rc;
  if ((rc = mark(4))) return rc;
  k_kb_seg<<<k.segs, 512, (size_t)k.B * 8, st>>>(p);
  if ((rc = chk("k_kb_seg"))) return rc;
  k_kb_segscan<<<(k.B + 31) / 32, 1024, 0, st>>>(p);
  if ((rc = chk("k_kb_segscan"))) return rc;
  k_kb_rows<<<k.segs, kRowThreads, (size_t)p.Bs * 8, st>>>(p);
  if ((rc = chk("k_kb_rows"))) return rc;
  if ((rc = mark(5))) return rc;
  k_kb_probe_count<<<(unsigned)k.pr_tiles, 512, (size_t)k.B * 4, st>>>(p);
  if ((rc = chk("k_kb_probe_count"))) return rc;
  if ((rc = starts(p.prhist, k.pr_tiles, p.proff, p.more))) return rc;
  static_assert((size_t)kKbMaxBlocks * 4 <= kPrSmem, "probe scatter shared memory");
  k_kb_probe_scatter<<<(unsigned)k.pr_tiles, kPrThreads, kPrSmem, st>>>(p);
  if ((rc = chk("k_kb_probe_scatter"))) return rc;
  k_kb_sweep<<<(unsigned)std::min<int64_t>(k.B + 2 * k.Q / p.part, ctas), kSwThreads, (size_t)k.m * 8, st>>>(p);
  if ((rc = chk("k_kb_sweep"))) return rc;
  k_kb_answers<<<(unsigned)k.pr_tiles, 256, 0, st>>>(p);
  if ((rc = chk("k_kb_answers"))) return rc;
  if ((rc = mark(6))) return rc;
  if (kernels_out) *kernels_out = kernels;
  return 0;
}

}  // namespace bw
