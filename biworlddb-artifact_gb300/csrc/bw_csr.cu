// bw_csr.cu -- sparse-key CSR rank-LUT: device build and lookups.
//
// The reference's CsrBase (sparse_engine.hpp:70-102) ranks a class by a per-64-class
// bitmap word and a cumulative popcount table, and build_csr_base
// (sparse_engine.hpp:287-360) fills it with two row scans over a dense class domain.
// Over a sparse 2^40-key universe a bitmap is not affordable, so here the same rank
// (number of index keys below k) and the same range sum (pre[rank(hi)-1] -
// pre[rank(lo)-1]) come from:
//   build    LSD radix sort of the (key, amount) pairs, 8 bits per pass
//            (bw_sort.cuh); run-length merge of equal keys with the cumulative
//            amounts (the prefix `pre`) in two passes over the pairs; a bucket LUT
//            lut[b] = #keys below b << shift sized to the caller's byte budget,
//            filled by warps that each cover the bucket gaps of 32 keys with
//            coalesced stores; the low `shift` bits of every key as u16 when
//            shift <= 16, so a probe reads 2 LUT words + a few 2-byte entries.
//   lookup   one thread per 2 point keys / per range, 128-bit loads and stores;
//            a bucket's keys are searched by bisection over the low bits.
#include <cuda_runtime.h>
#include <algorithm>
#include <cstdint>
#include <cstdio>

#include "bw_gpu.h"
#include "bw_common.cuh"
#include "bw_sort.cuh"

namespace bw {
namespace {

inline size_t al256(size_t x) { return (x + 255) & ~size_t(255); }

// Sort pass over (key, amount) pairs kept in two arrays.
struct CsrIO {
  const uint64_t* k;
  const int64_t* v;
  uint64_t* ko;
  int64_t* vo;
  int bits;
  static constexpr int kBadStatus = 1;
  __device__ __forceinline__ uint4 load(int64_t i) const {
    const uint64_t a = k[i], b = (uint64_t)v[i];
    return make_uint4((uint32_t)a, (uint32_t)(a >> 32), (uint32_t)b, (uint32_t)(b >> 32));
  }
  __device__ __forceinline__ uint32_t key(int64_t i, int shift) const { return (uint32_t)(k[i] >> shift); }
  __device__ __forceinline__ bool bad(int64_t i) const { return (k[i] >> bits) != 0; }
  static __device__ __forceinline__ uint32_t digits(const uint4& x, int shift) {
    return (uint32_t)((((uint64_t)x.y << 32) | x.x) >> shift);
  }
  __device__ __forceinline__ void store(int64_t at, const uint4& x) const {
    ko[at] = ((uint64_t)x.y << 32) | x.x;
    vo[at] = (int64_t)(((uint64_t)x.w << 32) | x.z);
  }
};

// Run-length merge of the sorted pairs in two passes over them: run ends and amounts
// per tile, then (with the tiles' prefixes) every run's key, cumulative amount and low
// bits at its place.  A warp takes 256 consecutive pairs, two per lane and round.
// (Separate flag, scan and compaction kernels moved 2 GB for 20M pairs and took 290 us; now 66 + 11 + 134.)
constexpr int kRunThreads = 512, kRunRounds = 4;
constexpr int64_t kRunTile = (int64_t)kRunThreads * 2 * kRunRounds;
struct RunPair {
  uint64_t k0, k1, v0, v1;
  bool f0, f1;               // the pair's items end a run
  // items i and i + 1 (i even) of n; every lane of the warp calls it, lanes consecutive
  __device__ __forceinline__ RunPair(const uint64_t* __restrict__ k, const int64_t* __restrict__ v, int64_t i, int64_t n) {
    k0 = k1 = v0 = v1 = 0;
    if (i + 1 < n) {
      const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(k + i);
      const longlong2 b = *reinterpret_cast<const longlong2*>(v + i);
      k0 = a.x; k1 = a.y; v0 = (uint64_t)b.x; v1 = (uint64_t)b.y;
    } else if (i < n) {
      k0 = k[i]; v0 = (uint64_t)v[i];
    }
    uint64_t next = __shfl_down_sync(0xffffffffu, k0, 1);
    if ((threadIdx.x & 31) == 31 && i + 2 < n) next = k[i + 2];
    f0 = i < n && (i + 1 == n || k1 != k0);
    f1 = i + 1 < n && (i + 2 == n || next != k1);
  }
};
__device__ __forceinline__ int64_t run_at(int r) {
  return (int64_t)blockIdx.x * kRunTile + (int64_t)(threadIdx.x >> 5) * (64 * kRunRounds) + r * 64 +
         2 * (int64_t)(threadIdx.x & 31);
}
__global__ void __launch_bounds__(kRunThreads) k_run_sums(const uint64_t* __restrict__ k, const int64_t* __restrict__ v,
                                                          int64_t n, uint64_t* __restrict__ part) {
  uint64_t ends = 0, sum = 0;
#pragma unroll
  for (int r = 0; r < kRunRounds; ++r) {
    const RunPair x(k, v, run_at(r), n);
    ends += (x.f0 ? 1 : 0) + (x.f1 ? 1 : 0);
    sum += x.v0 + x.v1;
  }
  uint64_t te = 0, ts = 0;
  block_exclusive_scan<uint64_t>(ends, &te);
  block_exclusive_scan<uint64_t>(sum, &ts);
  if (threadIdx.x == 0) {
    part[2 * (int64_t)blockIdx.x] = te;
    part[2 * (int64_t)blockIdx.x + 1] = ts;
  }
}
__global__ void __launch_bounds__(1024) k_run_parts(uint64_t* part, int64_t tiles) {
  uint64_t ce = 0, cs = 0;
  for (int64_t t0 = 0; t0 < tiles; t0 += 1024) {
    const int64_t t = t0 + threadIdx.x;
    const uint64_t e = t < tiles ? part[2 * t] : 0, s = t < tiles ? part[2 * t + 1] : 0;
    uint64_t te = 0, ts = 0;
    const uint64_t xe = block_exclusive_scan<uint64_t>(e, &te), xs = block_exclusive_scan<uint64_t>(s, &ts);
    if (t < tiles) {
      part[2 * t] = ce + xe;
      part[2 * t + 1] = cs + xs;
    }
    ce += te;
    cs += ts;
  }
}
__global__ void __launch_bounds__(kRunThreads) k_run_write(const uint64_t* __restrict__ k, const int64_t* __restrict__ v,
                                                           int64_t n, int shift, const uint64_t* __restrict__ part,
                                                           uint64_t* __restrict__ ukeys, int64_t* __restrict__ pre,
                                                           uint16_t* __restrict__ low, int64_t* __restrict__ count) {
  __shared__ uint64_t s_e[kRunThreads / 32], s_s[kRunThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned lt = (1u << lane) - 1u;
  const uint64_t mask = shift >= 64 ? ~0ull : ((1ull << shift) - 1ull);
  uint64_t k0[kRunRounds], k1[kRunRounds], c0[kRunRounds], c1[kRunRounds];   // keys, cumulative amounts in the warp
  uint32_t at[kRunRounds], f[kRunRounds];
  uint32_t ends = 0;
  uint64_t run = 0;
#pragma unroll
  for (int r = 0; r < kRunRounds; ++r) {
    const RunPair x(k, v, run_at(r), n);
    const unsigned m0 = __ballot_sync(0xffffffffu, x.f0), m1 = __ballot_sync(0xffffffffu, x.f1);
    at[r] = ends + __popc(m0 & lt) + __popc(m1 & lt);
    ends += __popc(m0) + __popc(m1);
    f[r] = (x.f0 ? 1u : 0u) | (x.f1 ? 2u : 0u);
    const uint64_t s = x.v0 + x.v1;
    uint64_t incl = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint64_t y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    k0[r] = x.k0;
    k1[r] = x.k1;
    c0[r] = run + incl - x.v1;
    c1[r] = run + incl;
    run += __shfl_sync(0xffffffffu, incl, 31);
  }
  if (lane == 0) {
    s_e[warp] = ends;
    s_s[warp] = run;
  }
  __syncthreads();
  uint64_t be = part[2 * (int64_t)blockIdx.x], bs = part[2 * (int64_t)blockIdx.x + 1];
  for (int w = 0; w < warp; ++w) {
    be += s_e[w];
    bs += s_s[w];
  }
#pragma unroll
  for (int r = 0; r < kRunRounds; ++r) {
    int64_t u = (int64_t)(be + at[r]);
    const int64_t i = run_at(r);
    if (f[r] & 1u) {
      ukeys[u] = k0[r];
      pre[u] = (int64_t)(bs + c0[r]);
      if (low) low[u] = (uint16_t)(k0[r] & mask);
      ++u;
      if (i + 1 == n) *count = u;
    }
    if (f[r] & 2u) {
      ukeys[u] = k1[r];
      pre[u] = (int64_t)(bs + c1[r]);
      if (low) low[u] = (uint16_t)(k1[r] & mask);
      if (i + 2 == n) *count = u + 1;
    }
  }
}

// lut[b] = number of keys whose bucket is below b, for b up to the last key's bucket.
// Warp w handles keys [32w, 32w+32): the buckets (bucket(key[32w-1]), bucket(key[32w+31])]
// get the warp's base index plus the count of its lanes with a lower bucket, found by
// bisection over the lanes' buckets with shuffles.
// Buckets are clamped to [0, nb) so that keys outside the universe (a flagged input
// error) cannot write past the table.
__global__ void k_lut_fill(const uint64_t* __restrict__ ukeys, const int64_t* __restrict__ count, int shift,
                           int64_t nb, uint32_t* __restrict__ lut) {
  const int64_t m = *count;
  const int lane = threadIdx.x & 31;
  const int64_t gw = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t w = gw; w * 32 < m; w += nw) {
    const int64_t u0 = w * 32;
    const int64_t u = u0 + lane;
    const int64_t bu = u < m ? (int64_t)(ukeys[u] >> shift) : INT64_MAX;
    const int64_t bstart = u0 ? imin64((int64_t)(ukeys[u0 - 1] >> shift), nb - 1) + 1 : 0;
    const int64_t ulast = (u0 + 32 < m ? u0 + 32 : m) - 1;
    const int64_t bend = imin64((int64_t)(ukeys[ulast] >> shift), nb - 1);
    for (int64_t b0 = bstart; b0 <= bend; b0 += 32) {
      const int64_t b = b0 + lane;
      int lo = 0;
#pragma unroll
      for (int step = 16; step; step >>= 1) {
        const int64_t x = __shfl_sync(0xffffffffu, bu, lo + step - 1);
        if (x < b) lo += step;
      }
      const int64_t x = __shfl_sync(0xffffffffu, bu, lo);
      if (x < b) ++lo;
      if (b <= bend) lut[b] = (uint32_t)(u0 + lo);
    }
  }
}

// Buckets past the last key's bucket (all of them when there are no keys) hold m.
__global__ void k_lut_tail(const uint64_t* __restrict__ ukeys, const int64_t* __restrict__ count, int shift,
                           int64_t nb, uint32_t* __restrict__ lut) {
  const int64_t m = *count;
  const int64_t first = m ? imin64((int64_t)(ukeys[m - 1] >> shift), nb - 1) + 1 : 0;
  for (int64_t b = first + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; b < nb; b += (int64_t)gridDim.x * blockDim.x)
    lut[b] = (uint32_t)m;
}

// rank(k) = number of index keys below k; *present when k is one of them.  V4: the
// LUT is read as aligned groups of four entries, which hold both ends of a bucket three
// times in four (the lookups are bound by the sectors the L1 and L2 serve; 100M point
// lookups: 1.11 -> 1.04 ms).
template <bool V4>
__device__ __forceinline__ int64_t csr_rank(const BwCsr& x, int64_t m, uint64_t k, bool& present) {
  present = false;
  if (x.key_bits < 64 && (k >> x.key_bits) != 0) return m;
  const int64_t b = (int64_t)(k >> x.shift);
  int64_t lo, hi;
  if constexpr (V4) {
    const uint4 q = __ldg(reinterpret_cast<const uint4*>(x.lut) + (b >> 2));
    const int c = (int)(b & 3);
    lo = c == 0 ? q.x : c == 1 ? q.y : c == 2 ? q.z : q.w;
    hi = c == 0 ? q.y : c == 1 ? q.z : q.w;
    if (c == 3) hi = b + 1 < x.n_buckets ? (int64_t)__ldg(x.lut + b + 1) : m;
  } else {
    lo = __ldg(x.lut + b);
    hi = b + 1 < x.n_buckets ? (int64_t)__ldg(x.lut + b + 1) : m;
  }
  // clamped to [0, m]: an index built from flagged input stays memory-safe
  lo = imin64(lo, m);
  hi = imin64(hi, m);
  const int64_t end = hi;   // the bucket's keys are [lo, end)
  if (x.low) {
    // keys of one bucket share their high bits: compare the low `shift` bits
    const uint16_t t = (uint16_t)(k & ((1ull << x.shift) - 1ull));
    while (lo < hi) {
      const int64_t mid = (lo + hi) >> 1;
      if (__ldg(x.low + mid) < t) lo = mid + 1; else hi = mid;
    }
    present = lo < end && __ldg(x.low + lo) == t;
  } else {
    while (lo < hi) {
      const int64_t mid = (lo + hi) >> 1;
      if (__ldg(x.keys + mid) < k) lo = mid + 1; else hi = mid;
    }
    present = lo < end && __ldg(x.keys + lo) == k;
  }
  return lo;
}

// Lookup inputs and outputs are streamed (evict first, `Once`): they are read or written once,
// and the L2 is left to the index.  Only where they and the LUT are more than kOnceBytes: smaller
// ones come from and go to kernels beside this one through the L2 (3M points, 64 KiB LUT, streamed / not,
// us: 3 keys 19.2 / 17.5, 15,000 keys 22.6 / 21.4, 10M keys 93.3 / 93.1; 64 MiB, 10M keys 39.7 / 41.5).
constexpr int64_t kOnceBytes = (int64_t)64 << 20;
template <bool Once, typename T>
__device__ __forceinline__ T lookup_ld(const T* p) {
  if constexpr (Once) return __ldcs(p);
  else return *p;
}
template <bool Once, typename T>
__device__ __forceinline__ void lookup_st(T* p, const T& v) {
  if constexpr (Once) __stcs(p, v);
  else *p = v;
}

template <bool V4, bool Once>
__device__ __forceinline__ void csr_points(const BwCsr& x, int64_t m, const uint64_t* __restrict__ keys, int64_t n,
                                           int64_t* __restrict__ out) {
  const int64_t npairs = n >> 1;
  const ulonglong2* kv = reinterpret_cast<const ulonglong2*>(keys);
  longlong2* ov = reinterpret_cast<longlong2*>(out);
  for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < npairs; p += (int64_t)gridDim.x * blockDim.x) {
    const ulonglong2 k = lookup_ld<Once>(kv + p);
    bool pa, pb;
    const int64_t ra = csr_rank<V4>(x, m, k.x, pa);
    const int64_t rb = csr_rank<V4>(x, m, k.y, pb);
    lookup_st<Once>(ov + p, make_longlong2(pa ? ra : -ra - 1, pb ? rb : -rb - 1));
  }
  if ((n & 1) && blockIdx.x == 0 && threadIdx.x == 0) {
    bool pr;
    const int64_t r = csr_rank<V4>(x, m, keys[n - 1], pr);
    out[n - 1] = pr ? r : -r - 1;
  }
}
// The fours gain 3 to 8 % from some thousand keys on; below, and where a small LUT stays in the L1,
// the selects cost more than the reads save (7M points, singly / in fours, us: 3 keys, 64 KiB LUT
// 30.2 / 35.7, 4 MiB 33.4 / 37.8; 15,000 keys, 64 KiB 40.7 / 43.9, 4 MiB 57.2 / 51.9; 200,000 keys, 64 KiB
// 85.2 / 79.1).  The count is known on the device only.
template <bool V4, bool Once>
__global__ void k_csr_point(BwCsr x, const uint64_t* __restrict__ keys, int64_t n, int64_t* __restrict__ out) {
  const int64_t m = *x.count;
  if (V4 && m >= (x.n_buckets >= (1 << 18) ? 1 << 12 : 1 << 16)) csr_points<V4, Once>(x, m, keys, n, out);
  else csr_points<false, Once>(x, m, keys, n, out);
}

// Range lookups.  LUT, low bits and prefix sums together (164 MB for 10M keys and a
// 64 MiB LUT) do not stay in the L2; the LUT with the low bits does, and so do the prefix
// sums.  So for large indexes each thread first writes the ranks of all its ranges into
// `out`, then turns them into differences and sums; the grid is resident as a whole, so
// its CTAs do either at about the same time (100M ranges over 10M keys: 5.7 -> 3.1 ms).
// Below kSplitKeys the 32 bytes a range that this writes and reads back cost more than the
// misses (20M ranges, one pass / two, us: 60,000 keys 403 / 436, 1.5M 427 / 483, 3M 513 /
// 494, 6M 803 / 524).  The LUT's entries are read one by one here: groups of four (above)
// cost the large index 5% and gain 2% on the smallest.
//
// Calls of up to kRangeMany ranges are launched with the eight CTAs an SM holds, larger ones with six,
// which leave more of the L1 and the L2 to each other (us, eight / six: 300,000 ranges, 10M keys, 64 MiB
// LUT 20.9 / 23.2, 3M keys, 4 MiB 13.8 / 14.7; 7M ranges, 10M keys, 4 MiB 330 / 315, 1M keys, 64 KiB 286 /
// 261; on indexes of a few keys eight stay faster, 46.8 / 50.4, but the count is known on the device only).
constexpr int kRangeCtas = 8, kRangeFew = 6;        // CTAs of 256 threads, an SM
constexpr int64_t kRangeMany = 1'000'000;
constexpr int64_t kSplitKeys = (int64_t)7 << 19;    // 28 MB of prefix sums
__device__ __forceinline__ longlong2 range_answer(const BwCsr& x, int64_t a, int64_t b) {
  uint64_t sum = 0;
  if (a != b) {
    const uint64_t shi = b ? (uint64_t)__ldg(x.pre + b - 1) : 0;
    const uint64_t slo = a ? (uint64_t)__ldg(x.pre + a - 1) : 0;
    sum = shi - slo;
  }
  return make_longlong2(b - a, (int64_t)sum);
}
template <bool Once>
__global__ void __launch_bounds__(256, kRangeCtas) k_csr_range(BwCsr x, const uint64_t* __restrict__ bounds, int64_t n,
                                                              int64_t* out) {
  const int64_t m = *x.count;
  const bool split = m >= kSplitKeys;
  const ulonglong2* bv = reinterpret_cast<const ulonglong2*>(bounds);
  longlong2* ov = reinterpret_cast<longlong2*>(out);
  const int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, step = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = i0; i < n; i += step) {
    const ulonglong2 q = lookup_ld<Once>(bv + i);
    bool pr;
    const int64_t a = csr_rank<false>(x, m, q.x, pr);
    const int64_t b = csr_rank<false>(x, m, q.y, pr);
    lookup_st<Once>(ov + i, split ? make_longlong2(a, b) : range_answer(x, a, b));
  }
  if (!split) return;
  for (int64_t i = i0; i < n; i += step) {
    const longlong2 r = lookup_ld<Once>(ov + i);
    lookup_st<Once>(ov + i, range_answer(x, r.x, r.y));
  }
}

// Versioned sparse keys (the event model over the index's ranks): event records
// keyed by the rank of their u64 key (a key missing from the index gets rank m, which
// the replay reports as out of range), and query records over rank intervals -- a
// point lookup of a present key is [rank, rank + 1), of an absent one empty; a range
// lookup [lo, hi) over keys is [rank(lo), rank(hi)) over ranks.
template <bool V4>
__global__ void k_csr_events(BwCsr x, const uint32_t* __restrict__ states, const uint64_t* __restrict__ keys,
                             const int64_t* __restrict__ deltas, int64_t n, BwEvent* __restrict__ out) {
  const int64_t m = *x.count;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    bool pr;
    const int64_t r = csr_rank<V4>(x, m, __ldcs(keys + i), pr);
    BwEvent e;
    e.state = __ldcs(states + i);
    e.key = (uint32_t)(pr ? r : m);
    e.delta = __ldcs(deltas + i);
    out[i] = e;
  }
}
template <bool V4>
__global__ void k_csr_queries(BwCsr x, const uint32_t* __restrict__ states, const uint64_t* __restrict__ lo,
                              const uint64_t* __restrict__ hi, int64_t n, BwQuery* __restrict__ out) {
  const int64_t m = *x.count;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    bool pr;
    const int64_t a = csr_rank<V4>(x, m, __ldcs(lo + i), pr);
    BwQuery q;
    q.state = __ldcs(states + i);
    if (!hi) {
      q.lo = pr ? (uint32_t)a : 0u;
      q.hi = pr ? (uint32_t)a + 1u : 0u;
    } else {
      bool pb;
      q.lo = (uint32_t)a;
      q.hi = (uint32_t)csr_rank<V4>(x, m, __ldcs(hi + i), pb);
    }
    __stcs(&out[i].state, q.state);
    __stcs(&out[i].lo, q.lo);
    __stcs(&out[i].hi, q.hi);
  }
}

struct CsrLayout {
  int32_t shift = 0, passes = 0;
  int64_t nb = 0;
  RsLayout rs;
  size_t off_count, off_status, off_keys, off_pre, off_low, off_lut;     // persistent index
  size_t off_ka, off_va, off_kb, off_vb, off_hist, off_part, off_base, off_runs;  // build scratch
  size_t total;
};

int csr_layout(int64_t n, int32_t key_bits, size_t budget, CsrLayout& L) {
  if (n < 0 || n >= ((int64_t)1 << 31) || key_bits < 1 || key_bits > 63 || budget < 4) return BW_EINVAL;
  int lb = 0;  // log2 of the bucket count
  while (lb < key_bits && ((size_t)1 << (lb + 1)) * 4 <= budget) ++lb;
  L.nb = (int64_t)1 << lb;
  L.shift = key_bits - lb;
  L.passes = (key_bits + 7) / 8;
  L.rs = rs_layout(n, L.passes);
  const size_t un = (size_t)(n > 0 ? n : 1);
  size_t o = 0;
  auto take = [&](size_t bytes) { const size_t at = o; o = al256(o + bytes); return at; };
  L.off_count = take(8);
  L.off_status = take(4);
  L.off_keys = take(un * 8);
  L.off_pre = take(un * 8);
  L.off_low = take(L.shift <= 16 ? un * 2 : 0);
  L.off_lut = take((size_t)L.nb * 4);
  L.off_ka = take(un * 8);
  L.off_va = take(un * 8);
  L.off_kb = take(un * 8);
  L.off_vb = take(un * 8);
  L.off_hist = take(L.rs.hist);
  L.off_part = take(L.rs.part);
  L.off_base = take(L.rs.base);
  L.off_runs = take(((un + kRunTile - 1) / kRunTile) * 16);
  L.total = o;
  return 0;
}

int report(cudaError_t e, const char* what) {
  if (e != cudaSuccess) std::fprintf(stderr, "bw_csr: %s failed: %s\n", what, cudaGetErrorString(e));
  return (int)e;
}

int sm_count() {
  int sms = 0, dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    sms = 148;
  return sms;
}

int grid_for(int64_t items, int threads) {
  const int64_t want = (items + threads - 1) / threads;
  const int64_t cap = (int64_t)sm_count() * 16;
  return (int)(want < 1 ? 1 : (want < cap ? want : cap));
}

}  // namespace
}  // namespace bw

using namespace bw;

extern "C" int bw_csr_workspace_size(int64_t n_items, int32_t key_bits, size_t lut_budget_bytes, size_t* bytes) {
  if (!bytes) return BW_EINVAL;
  CsrLayout L;
  if (csr_layout(n_items, key_bits, lut_budget_bytes, L)) return BW_EINVAL;
  *bytes = L.total;
  return 0;
}

extern "C" int bw_csr_build(const uint64_t* keys, const int64_t* amounts, int64_t n_items, int32_t key_bits,
                            size_t lut_budget_bytes, void* workspace, size_t workspace_bytes, void* stream,
                            BwCsr* out) {
  CsrLayout L;
  if (!out || !workspace || csr_layout(n_items, key_bits, lut_budget_bytes, L)) return BW_EINVAL;
  if (n_items > 0 && (!keys || !amounts)) return BW_EINVAL;
  if ((reinterpret_cast<uintptr_t>(workspace) & 255) != 0) return BW_EINVAL;
  if (workspace_bytes < L.total) {
    std::fprintf(stderr, "bw_csr_build: workspace %zu < required %zu bytes\n", workspace_bytes, L.total);
    return BW_EINVAL;
  }
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  char* ws = static_cast<char*>(workspace);
  int64_t* count = reinterpret_cast<int64_t*>(ws + L.off_count);
  int32_t* status = reinterpret_cast<int32_t*>(ws + L.off_status);
  uint64_t* ukeys = reinterpret_cast<uint64_t*>(ws + L.off_keys);
  int64_t* pre = reinterpret_cast<int64_t*>(ws + L.off_pre);
  uint16_t* low = L.shift <= 16 ? reinterpret_cast<uint16_t*>(ws + L.off_low) : nullptr;
  uint32_t* lut = reinterpret_cast<uint32_t*>(ws + L.off_lut);
  uint64_t* ka = reinterpret_cast<uint64_t*>(ws + L.off_ka);
  int64_t* va = reinterpret_cast<int64_t*>(ws + L.off_va);
  uint64_t* kb = reinterpret_cast<uint64_t*>(ws + L.off_kb);
  int64_t* vb = reinterpret_cast<int64_t*>(ws + L.off_vb);
  uint32_t* hist = reinterpret_cast<uint32_t*>(ws + L.off_hist);
  uint32_t* part = reinterpret_cast<uint32_t*>(ws + L.off_part);
  uint64_t* base = reinterpret_cast<uint64_t*>(ws + L.off_base);
  uint64_t* runs = reinterpret_cast<uint64_t*>(ws + L.off_runs);
  int rc;
  if ((rc = report(cudaMemsetAsync(count, 0, 8, st), "memset"))) return rc;
  if ((rc = report(cudaMemsetAsync(status, 0, 4, st), "memset"))) return rc;
  const int64_t n = n_items;
  if (n > 0) {
    // ---- LSD radix sort, 8 bits per pass; pass p reads (k, v) and writes (ko, vo)
    if ((rc = report(cudaMemsetAsync(part, 0, L.rs.part, st), "memset"))) return rc;
    CsrIO io{keys, amounts, ka, va, key_bits};
    for (int p = 0; p < L.passes; ++p) {
      if ((rc = report((cudaError_t)rs_pass(io, n, 8 * p, L.rs, hist, part + (size_t)p * L.rs.chunks * kRsDigits, base,
                                            p == 0, status, st), "sort pass")))
        return rc;
      io.k = io.ko;
      io.v = io.vo;
      io.ko = io.k == ka ? kb : ka;
      io.vo = io.v == va ? vb : va;
    }
    const uint64_t* ksorted = io.k;
    const int64_t* vsorted = io.v;
    // ---- run-length merge
    const int64_t tiles = (n + kRunTile - 1) / kRunTile;
    k_run_sums<<<(unsigned)tiles, kRunThreads, 0, st>>>(ksorted, vsorted, n, runs);
    if ((rc = report(cudaGetLastError(), "k_run_sums"))) return rc;
    k_run_parts<<<1, 1024, 0, st>>>(runs, tiles);
    if ((rc = report(cudaGetLastError(), "k_run_parts"))) return rc;
    k_run_write<<<(unsigned)tiles, kRunThreads, 0, st>>>(ksorted, vsorted, n, L.shift, runs, ukeys, pre, low, count);
    if ((rc = report(cudaGetLastError(), "k_run_write"))) return rc;
    k_lut_fill<<<grid_for(n, 256), 256, 0, st>>>(ukeys, count, L.shift, L.nb, lut);
    if ((rc = report(cudaGetLastError(), "k_lut_fill"))) return rc;
  }
  k_lut_tail<<<grid_for(L.nb, 256), 256, 0, st>>>(ukeys, count, L.shift, L.nb, lut);
  if ((rc = report(cudaGetLastError(), "k_lut_tail"))) return rc;
  out->key_bits = key_bits;
  out->shift = L.shift;
  out->n_buckets = L.nb;
  out->count = count;
  out->status = status;
  out->keys = ukeys;
  out->pre = pre;
  out->lut = lut;
  out->low = low;
  return 0;
}

// Whether the LUT is read as groups of four entries: where it can be, and stays in the L2
// (20M points, 60,000 keys, singly / in fours: 64 MiB LUT 150 / 145 us, 256 MiB 252 / 275).
static bool lut4(const BwCsr* x) {
  return (reinterpret_cast<uintptr_t>(x->lut) & 15) == 0 && x->n_buckets >= 4 && x->n_buckets <= ((int64_t)1 << 25);
}

static int check_index(const BwCsr* x) {
  if (!x || !x->count || !x->status || !x->lut || !x->keys || !x->pre || x->key_bits < 1 || x->key_bits > 63 || x->shift < 0 ||
      x->shift > x->key_bits || x->n_buckets != ((int64_t)1 << (x->key_bits - x->shift)) || (x->low && x->shift > 16))
    return BW_EINVAL;
  return 0;
}

extern "C" int bw_csr_point(const BwCsr* idx, const uint64_t* keys, int64_t n, int64_t* out, void* stream) {
  if (check_index(idx) || n < 0 || (n > 0 && (!keys || !out))) return BW_EINVAL;
  if (n == 0) return 0;
  if ((reinterpret_cast<uintptr_t>(keys) & 15) || (reinterpret_cast<uintptr_t>(out) & 15)) return BW_EINVAL;
  const bool once = n * 16 + idx->n_buckets * 4 > kOnceBytes;
  (lut4(idx) ? once ? k_csr_point<true, true> : k_csr_point<true, false>
             : once ? k_csr_point<false, true> : k_csr_point<false, false>)<<<
      grid_for((n + 1) / 2, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(*idx, keys, n, out);
  return report(cudaGetLastError(), "k_csr_point");
}

extern "C" int bw_csr_range(const BwCsr* idx, const uint64_t* bounds, int64_t n, int64_t* out, void* stream) {
  if (check_index(idx) || n < 0 || (n > 0 && (!bounds || !out))) return BW_EINVAL;
  if (n == 0) return 0;
  if ((reinterpret_cast<uintptr_t>(bounds) & 15) || (reinterpret_cast<uintptr_t>(out) & 15)) return BW_EINVAL;
  const cudaStream_t st = static_cast<cudaStream_t>(stream);
  const bool once = n * 32 + idx->n_buckets * 4 > kOnceBytes;
  // no more CTAs than are resident at once
  (once ? k_csr_range<true> : k_csr_range<false>)<<<
      std::min(grid_for(n, 256), sm_count() * (n <= kRangeMany ? kRangeCtas : kRangeFew)), 256, 0, st>>>(*idx, bounds, n, out);
  return report(cudaGetLastError(), "k_csr_range");
}

extern "C" int bw_csr_status(const BwCsr* idx, int32_t* status) {
  if (check_index(idx) || !status) return BW_EINVAL;
  int rc = report(cudaDeviceSynchronize(), "synchronise");
  if (rc) return rc;
  return report(cudaMemcpy(status, idx->status, 4, cudaMemcpyDeviceToHost), "status read");
}

extern "C" int bw_csr_events(const BwCsr* idx, const uint32_t* states, const uint64_t* keys, const int64_t* deltas,
                             int64_t n, BwEvent* out, void* stream) {
  if (check_index(idx) || n < 0 || (n > 0 && (!states || !keys || !deltas || !out))) return BW_EINVAL;
  if (n == 0) return 0;
  (lut4(idx) ? k_csr_events<true> : k_csr_events<false>)<<<grid_for(n, 256), 256, 0,
                                                           static_cast<cudaStream_t>(stream)>>>(*idx, states, keys,
                                                                                                deltas, n, out);
  return report(cudaGetLastError(), "k_csr_events");
}

extern "C" int bw_csr_queries(const BwCsr* idx, const uint32_t* states, const uint64_t* lo, const uint64_t* hi,
                              int64_t n, BwQuery* out, void* stream) {
  if (check_index(idx) || n < 0 || (n > 0 && (!states || !lo || !out))) return BW_EINVAL;
  if (n == 0) return 0;
  (lut4(idx) ? k_csr_queries<true> : k_csr_queries<false>)<<<grid_for(n, 256), 256, 0,
                                                             static_cast<cudaStream_t>(stream)>>>(*idx, states, lo, hi,
                                                                                                  n, out);
  return report(cudaGetLastError(), "k_csr_queries");
}
