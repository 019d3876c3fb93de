// bw_qsweep.cu -- query-step sweep of the general (tree) pipeline, for trees whose
// states are asked many queries each (tile 7).
//
// A block's Euler steps are replayed one at a time by all 512 threads: thread i applies
// event i of the step; at a step with queries threads 2i and 2i + 1 take the lower and
// upper bound of query i (further ones, past 256, four at a time).  The window over the block's
// key ranks (shared memory) holds Fenwick nodes inside groups of 16 ranks and the groups' totals
// (an update is up to five no-return atomics) and, rebuilt by a warp a run before a query step that
// follows updates, the prefixes of the totals inside every run of 2,048 ranks; a warp scans the
// totals of the runs itself.  A probe is one prefix, one shuffle and up to four nodes -- per
// thread, so a step's queries cost a few hundred cycles together, however many they are up to 256.
//
// The carried part of every answer is written beforehand by k_qcarry, a block's queries
// side by side over its carry row (random reads of one 512 KB row at a time stay in the
// L2; inside the sweep 304 rows were read at once); the sweep adds the window's part with
// a no-return atomic.  A thread's event and bound of a step are copied into shared-memory
// slots of its own three steps ahead, two with int64 windows (cp.async: register loads four steps
// ahead shared their scoreboards with the step's own shared-memory reads and cost a memory latency a
// step), the step descriptors through a ring.
//
// Bound by the latency of the three barriers of a query step, two CTAs an SM to overlap
// them.  With k_qcarry, against the tiles of 256 threads: trip-log tree of 300,000 states, 40M
// events and 50M queries 4.56 -> 2.29 ms, 30,000 states, 4M events and 5M queries 0.48 -> 0.33.
#include <cuda_runtime.h>
#include <cstdint>

#include "bw_gpu.h"
#include "bw_common.cuh"
#include "bw_pipeline.cuh"

namespace bw {
namespace {

constexpr int kQsThreads = 512, kQsWarps = kQsThreads / 32;
constexpr uint32_t kQsGroup = 16, kQsRunGroups = 128, kQsSuper = kQsGroup * kQsRunGroups;   // ranks of a total, of a run
constexpr uint32_t kQsMaxRuns = 16;                  // one warp each
constexpr int kQsRing = 128;                         // step descriptors
constexpr int kQsMore = 4;                           // queries a thread pair reads at a time past its first
constexpr int kQsSlots = 9;                          // slot arrays of a word per thread
constexpr uint32_t kFull = 0xffffffffu;
static_assert(kQsRunGroups == 4 * 32, "a warp scans the totals of one run, four a lane");

struct QsSmem {
  size_t rl, leaf, gsum, gpre, stot, ring, slots, bytes;
};
__host__ __device__ inline size_t qs_al(size_t x) { return (x + 15) & ~size_t(15); }
// `supers` runs of 2,048 int32 ranks (half as many int64 ones in the same bytes).
__host__ __device__ inline QsSmem qs_smem(int32_t ww, uint32_t supers) {
  QsSmem L;
  size_t o = qs_al((size_t)ww * 8);
  L.rl = o;    o = qs_al(o + ((size_t)ww + 2) * 2);
  L.leaf = o;  o = qs_al(o + (size_t)supers * kQsSuper * 4);
  L.gsum = o;  o = qs_al(o + (size_t)supers * kQsRunGroups * 4);
  L.gpre = o;  o = qs_al(o + (size_t)supers * kQsRunGroups * 4);
  L.stot = o;  o = qs_al(o + (size_t)supers * 4);
  L.ring = o;  o = qs_al(o + (size_t)kQsRing * 16);
  L.slots = o; o = qs_al(o + (size_t)kQsSlots * kQsThreads * 4);
  L.bytes = o;
  return L;
}

__device__ __forceinline__ void qs_copy16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}

__device__ __forceinline__ void qs_copy4(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}

template <typename Node>
__device__ __forceinline__ Node qs_scan(Node v, int lane) {   // inclusive, over the warp
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const Node y = __shfl_up_sync(kFull, v, o);
    if (lane >= o) v += y;
  }
  return v;
}

// Prefix of i < 16 ranks inside a group: Fenwick nodes 1 .. 15 of the group at g (node n
// at g[n - 1]; the sixteenth word is unused), four independent reads.
template <typename Node>
__device__ __forceinline__ Node qs_partial(const Node* g, uint32_t i) {
  Node s = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    if (i) s += g[i - 1];
    i &= i - 1;
  }
  return s;
}
// Four consecutive totals of a lane: loaded, scanned over the warp's 128, exclusive
// prefixes stored; returns the run's total in lane 31.
__device__ __forceinline__ uint32_t qs_run(const uint32_t* in, uint32_t* out, int lane) {
  const uint4 v = reinterpret_cast<const uint4*>(in)[lane];
  const uint32_t s1 = v.x + v.y, s2 = s1 + v.z, s3 = s2 + v.w, incl = qs_scan(s3, lane), ex = incl - s3;
  reinterpret_cast<uint4*>(out)[lane] = make_uint4(ex, ex + v.x, ex + s1, ex + s2);
  return incl;
}
__device__ __forceinline__ unsigned long long qs_run(const unsigned long long* in, unsigned long long* out, int lane) {
  const ulonglong2 a = reinterpret_cast<const ulonglong2*>(in)[2 * lane], b = reinterpret_cast<const ulonglong2*>(in)[2 * lane + 1];
  const unsigned long long s1 = a.x + a.y, s2 = s1 + b.x, s3 = s2 + b.y, incl = qs_scan(s3, lane), ex = incl - s3;
  reinterpret_cast<ulonglong2*>(out)[2 * lane] = make_ulonglong2(ex, ex + a.x);
  reinterpret_cast<ulonglong2*>(out)[2 * lane + 1] = make_ulonglong2(ex + s1, ex + s2);
  return incl;
}

template <typename Node>
__device__ __forceinline__ void qs_block(const EsParams& p, int32_t ww, uint32_t supers, unsigned char* sm, int32_t b) {
  const BlockTab bt = p.blocks[b];
  const int32_t t0 = bt.t0, t1 = bt.t1;
  if (t0 >= t1) return;
  const QsSmem L = qs_smem(ww, supers);
  uint64_t* bits = reinterpret_cast<uint64_t*>(sm);
  uint16_t* rl = reinterpret_cast<uint16_t*>(sm + L.rl);
  Node* leaf = reinterpret_cast<Node*>(sm + L.leaf);
  Node* gsum = reinterpret_cast<Node*>(sm + L.gsum);
  Node* gpre = reinterpret_cast<Node*>(sm + L.gpre);
  Node* stot = reinterpret_cast<Node*>(sm + L.stot);
  uint4* ring = reinterpret_cast<uint4*>(sm + L.ring);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  uint32_t* slots = reinterpret_cast<uint32_t*>(sm + L.slots) + threadIdx.x;   // word w of this thread: slots[w * 512]
  constexpr int kDepth = sizeof(Node) == 4 ? 3 : 2;   // steps copied ahead
  constexpr int kWords = sizeof(Node) == 4 ? 2 : 3;   // key and delta words; the bounds follow
  const int32_t nsl = p.nslices[b];
  const Slice* bsl = p.slices + (size_t)b * p.max_slices;
  for (int32_t si = 0; si < nsl; ++si) {
    const Slice s = bsl[si];
    if (s.n == 0) continue;   // no keys: no part of any answer
    const uint32_t klo = (uint32_t)s.word_lo << 6;
    const uint32_t khi = (uint32_t)min((uint64_t)s.word_hi << 6, (uint64_t)bt.C);
    const uint32_t nsup = s.n / kQsSuper + 1;   // rank s.n lies in the last run
    {
      const uint64_t* gbits = p.bits + bt.bits_off + s.word_lo;
      const uint32_t* grl = p.rlut + bt.bits_off + b + s.word_lo;
      const int32_t nwd = s.word_hi - s.word_lo;
      for (int32_t i = tid; i < nwd; i += kQsThreads) {
        bits[i] = gbits[i];
        rl[i] = (uint16_t)(grl[i] - s.rank_lo);
      }
      uint4* z = reinterpret_cast<uint4*>(leaf);
      for (uint32_t i = tid; i < nsup * kQsSuper * sizeof(Node) / 16; i += kQsThreads) z[i] = make_uint4(0, 0, 0, 0);
      for (uint32_t i = tid; i < nsup * kQsRunGroups; i += kQsThreads) gsum[i] = gpre[i] = 0;
      for (uint32_t i = tid; i < nsup; i += kQsThreads) stot[i] = 0;
    }
    // descriptors: step t at ring[t % kQsRing]; half a ring is requested at the start of
    // the other half and has landed by its middle
    const uint4 none = make_uint4(0, 0, 0, 0);
    auto request = [&](int32_t from) {
      if (tid < kQsRing / 2) {
        const int32_t t = from + tid;
        if (t < t1) qs_copy16(ring + (t & (kQsRing - 1)), p.desc + t);
        else ring[t & (kQsRing - 1)] = none;
      }
    };
    const int32_t a0 = t0 & ~(kQsRing / 2 - 1);   // halves are aligned
    request(a0);
    request(a0 + kQsRing / 2);
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    auto key_rank = [&](uint32_t k) -> uint32_t {   // slice rank of a bound
      if (k <= klo) return 0u;
      if (k >= khi) return s.n;
      const uint32_t x = k - klo, w = x >> 6;
      return (uint32_t)rl[w] + (uint32_t)__popcll(bits[w] & ((1ull << (x & 63)) - 1ull));
    };
    auto apply = [&](const uint4& e, bool neg) {
      const uint32_t x = e.y - klo;
      if (x >= khi - klo) return;
      const uint32_t w = x >> 6, r = (uint32_t)rl[w] + (uint32_t)__popcll(bits[w] & ((1ull << (x & 63)) - 1ull));
      Node* g = leaf + (r & ~(kQsGroup - 1));
      uint32_t n = (r & (kQsGroup - 1)) + 1;
      uint64_t d = ((uint64_t)e.w << 32) | e.z;
      if (neg) d = (uint64_t)0 - d;
      auto add = [&](Node* at) {
        if constexpr (sizeof(Node) == 4) atomicAdd(at, (uint32_t)d);
        else shared_add_u64(at, d);
      };
      add(gsum + r / kQsGroup);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (n < kQsGroup) add(g + n - 1);
        n += n & (0u - n);
      }
    };
    auto bound_at = [&](uint32_t q) -> uint32_t {   // this thread's bound of query q
      const uint32_t* x = reinterpret_cast<const uint32_t*>(p.qs + q);
      return __ldg(x + 1 + (tid & 1));
    };
    // step t's event and bound of this thread into stage t % kDepth
    auto copy = [&](int32_t t, int stage) {
      if (t < t1) {
        const uint4 d = ring[t & (kQsRing - 1)];
        if (tid < (int32_t)d.z) {
          const uint32_t* e = reinterpret_cast<const uint32_t*>(p.ev + d.x + tid) + 1;
#pragma unroll
          for (int w = 0; w < kWords; ++w) qs_copy4(slots + (stage * kWords + w) * kQsThreads, e + w);
        }
        if ((tid >> 1) < (int32_t)d.w)
          qs_copy4(slots + (kDepth * kWords + stage) * kQsThreads,
                   reinterpret_cast<const uint32_t*>(p.qs + (d.y + (tid >> 1))) + 1 + (tid & 1));
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // the window's part of the pair's query: prefix at hi - prefix at lo
    auto answer = [&](bool in, uint32_t q, uint32_t x, uint32_t r, Node spre) {
      Node v = gpre[r / kQsGroup] + qs_partial(leaf + (r & ~(kQsGroup - 1)), r & (kQsGroup - 1));
      v += __shfl_sync(kFull, spre, (int)(r / kQsSuper));
      v = __shfl_down_sync(kFull, v, 1) - v;
      const uint32_t xh = __shfl_down_sync(kFull, x, 1);
      if (in && !(tid & 1) && xh > x) {
        const uint64_t a = sizeof(Node) == 4 ? (uint64_t)(int64_t)(int32_t)v : (uint64_t)v;
        if (a) atomicAdd(reinterpret_cast<unsigned long long*>(p.answers + q), (unsigned long long)a);
      }
    };
    bool dirty = false;   // (the same in every thread) updates since the prefixes were built
    int stage = 0;        // t % kDepth, from t0
#pragma unroll
    for (int k = 0; k < kDepth; ++k) copy(t0 + k, k);
    for (int32_t t = t0; t < t1; ++t) {
      const int32_t half = t & (kQsRing / 2 - 1);
      if (half == 0 && t > t0) {
        __syncthreads();                       // every thread is past the half before
        request(t + kQsRing / 2);
      } else if (half == kQsRing / 4) {
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
      }
      asm volatile("cp.async.wait_group %0;" ::"n"(kDepth - 1) : "memory");   // this thread's copies of step t
      const uint4 d = ring[t & (kQsRing - 1)];
      const int32_t ne = (int32_t)d.z, nq = (int32_t)d.w;
      if (tid < ne) {
        uint4 e;
        e.y = slots[stage * kWords * kQsThreads];
        e.z = slots[(stage * kWords + 1) * kQsThreads];
        e.w = kWords == 3 ? slots[(stage * kWords + 2) * kQsThreads] : 0u;
        apply(e, nq < 0);
        for (int32_t i = kQsThreads + tid; i < ne; i += kQsThreads) apply(__ldg(p.ev + (size_t)d.x + i), nq < 0);
      }
      dirty |= ne > 0;
      if (nq > 0) {
        const bool mine = (tid >> 1) < nq, active = warp * 16 < nq;
        const uint32_t x0 = mine ? slots[(kDepth * kWords + stage) * kQsThreads] : 0u, r0 = mine ? key_rank(x0) : 0u;
        if (dirty) {
          __syncthreads();                     // the updates of every step so far
          if (warp < (int)nsup) {
            const Node total = qs_run(gsum + warp * kQsRunGroups, gpre + warp * kQsRunGroups, lane);
            if (lane == 31) stot[warp] = total;
          }
          __syncthreads();
        }
        if (active) {
          const Node own = lane < (int)nsup ? stot[lane] : (Node)0;
          Node spre = own;                     // totals of the runs below run `lane`
#pragma unroll
          for (int o = 1; o < (int)kQsMaxRuns; o <<= 1) {
            const Node y = __shfl_up_sync(kFull, spre, o);
            if (lane >= o) spre += y;
          }
          spre -= own;
          answer(mine, d.y + (tid >> 1), x0, r0, spre);
          for (int32_t q0 = kQsThreads / 2; q0 + warp * 16 < nq; q0 += kQsMore * kQsThreads / 2) {   // more than 256 queries
            uint32_t x[kQsMore];   // (read together: a memory latency for every 256 queries else)
#pragma unroll
            for (int u = 0; u < kQsMore; ++u) {
              const int32_t q = q0 + u * (kQsThreads / 2) + (tid >> 1);
              x[u] = q < nq ? bound_at(d.y + q) : 0u;
            }
#pragma unroll
            for (int u = 0; u < kQsMore; ++u) {
              const int32_t q = q0 + u * (kQsThreads / 2) + (tid >> 1);
              if (q - (tid >> 1) + warp * 16 < nq) answer(q < nq, d.y + q, x[u], q < nq ? key_rank(x[u]) : 0u, spre);
            }
          }
        }
        __syncthreads();                       // probes done before the next updates
        dirty = false;
      }
      copy(t + kDepth, stage);
      stage = stage + 1 == kDepth ? 0 : stage + 1;
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
  }
}

// The carried part of every query's answer (0 where the block starts its tree).  A CTA
// per part of a block: a warp takes eight consecutive steps at a time and their queries,
// flattened.  The parts of a block run side by side, so that some eighty carry rows are
// read at a time and stay in the L2.  (One grid dimension for both: a caller may ask for
// more blocks than the second one takes.)
// A group of steps with more than kQcHeavy queries is left for the end, when the CTA's
// warps share it: a state asked much more than the others kept a single warp busy (a replay of
// 30,000 states and 1M queries, half of them on one state, 13.0 -> 1.8 ms; one state, 2.8M queries
// 70 -> 7.9; queries spread evenly unchanged).  Lists in device memory would let all parts share
// a group, but the sweep, which takes such a step with one CTA, needs as long as one CTA here.
constexpr int kQcParts = 16, kQcSteps = 8, kQcWarps = 8;
constexpr int kQcBatch = 4;                 // queries a lane reads at a time
constexpr uint32_t kQcHeavy = 1024;
constexpr int kQcList = 32;                 // groups left for the end; further ones are done where they occur
__global__ void __launch_bounds__(32 * kQcWarps) k_qcarry(EsParams p) {
  if (*p.status) return;
  __shared__ int32_t s_heavy[kQcList], s_nheavy;
  const BlockTab bt = p.blocks[blockIdx.x / kQcParts];
  const int64_t* crow = bt.carry_in >= 0 ? p.carry + bt.carry_in : nullptr;
  const int lane = threadIdx.x & 31, own = threadIdx.x >> 5, warp = (blockIdx.x % kQcParts) * kQcWarps + own;
  if (threadIdx.x == 0) s_nheavy = 0;
  __syncthreads();
  uint32_t n, incl, first;   // of this lane's step: queries, those up to it, the first one
  auto decode = [&](int32_t c) -> uint32_t {
    const uint4 d = lane < kQcSteps && c + lane < bt.t1 ? __ldg(reinterpret_cast<const uint4*>(p.desc) + c + lane)
                                                        : make_uint4(0, 0, 0, 0);
    n = (int32_t)d.w > 0 ? d.w : 0u;
    first = d.y;
    incl = n;
#pragma unroll
    for (int o = 1; o < kQcSteps; o <<= 1) {
      const uint32_t y = __shfl_up_sync(kFull, incl, o);
      if (lane >= o) incl += y;
    }
    return __shfl_sync(kFull, incl, kQcSteps - 1);
  };
  auto answer = [&](uint32_t from, uint32_t total, uint32_t stride) {
    for (uint64_t g0 = from; g0 < total; g0 += stride) {
      uint32_t q[kQcBatch], a[kQcBatch], z[kQcBatch];
#pragma unroll
      for (int u = 0; u < kQcBatch; ++u) {
        const uint32_t g = (uint32_t)g0 + 32 * u + lane;
        int lo = 0, hi = kQcSteps - 1;   // first step whose inclusive count exceeds g
#pragma unroll
        for (int it = 0; it < 3; ++it) {
          const int mid = (lo + hi) >> 1;
          if (__shfl_sync(kFull, incl, mid) > g) hi = mid; else lo = mid + 1;
        }
        const uint32_t before = __shfl_sync(kFull, incl - n, lo), q0 = __shfl_sync(kFull, first, lo);
        q[u] = q0 + (g - before);
        a[u] = z[u] = 0;
        if (g < total && crow) {
          a[u] = __ldg(&p.qs[q[u]].lo);
          z[u] = __ldg(&p.qs[q[u]].hi);
        }
      }
      int64_t ra[kQcBatch], rz[kQcBatch];
#pragma unroll
      for (int u = 0; u < kQcBatch; ++u) {
        ra[u] = rz[u] = 0;
        if (a[u] < z[u]) {
          ra[u] = __ldg(crow + a[u]);
          rz[u] = __ldg(crow + z[u]);
        }
      }
#pragma unroll
      for (int u = 0; u < kQcBatch; ++u)
        if ((uint32_t)g0 + 32 * u + lane < total) p.answers[q[u]] = (int64_t)((uint64_t)rz[u] - (uint64_t)ra[u]);
    }
  };
  for (int32_t c = bt.t0 + kQcSteps * warp; c < bt.t1; c += kQcSteps * kQcWarps * kQcParts) {
    const uint32_t total = decode(c);
    if (total > kQcHeavy) {
      int32_t i = 0;
      if (lane == 0) i = atomicAdd(&s_nheavy, 1);
      i = __shfl_sync(kFull, i, 0);
      if (i < kQcList) {
        if (lane == 0) s_heavy[i] = c;
        continue;
      }
    }
    answer(0, total, 32 * kQcBatch);
  }
  __syncthreads();
  const int32_t nh = min(s_nheavy, kQcList);
  for (int32_t h = 0; h < nh; ++h) answer(own * 32 * kQcBatch, decode(s_heavy[h]), kQcWarps * 32 * kQcBatch);
}

__global__ void __launch_bounds__(kQsThreads, 2) k_qsweep(EsParams p, int32_t ww, uint32_t supers) {
  extern __shared__ __align__(16) unsigned char sm[];
  __shared__ int32_t s_ticket;
  if (*p.status) return;   // never index with descriptors of rejected input
  for (;;) {
    __syncthreads();
    if (threadIdx.x == 0) s_ticket = atomicAdd(p.ticket, 1);
    __syncthreads();
    const int32_t i = s_ticket;
    if (i >= p.B) break;
    const int32_t b = p.order ? p.order[i] : i;
    if (p.bmode[b] & kMode32) qs_block<uint32_t>(p, ww, supers, sm, b);
    else qs_block<unsigned long long>(p, ww, supers, sm, b);
  }
}

}  // namespace

// Rank capacities for domains of `nwords` bitmap words (two CTAs an SM): as many runs of
// 2,048 as fit, the last rank kept for bounds past the last key.
QsLayout qsweep_layout(int32_t nwords) {
  QsLayout q;
  q.ww = nwords < kWinWords ? nwords : kWinWords;
  const size_t budget = (size_t)kSmemPerSM / 2 - 1024 - 256;
  uint32_t n = 2;
  while (n < kQsMaxRuns && qs_smem(q.ww, n + 1).bytes <= budget) ++n;
  q.supers = n;
  q.cap32 = n * kQsSuper - 1;
  q.cap64 = (n / 2) * kQsSuper - 1;
  q.bytes = qs_smem(q.ww, n).bytes;
  return q;
}

int qsweep_attrs() {
  return (int)cudaFuncSetAttribute(k_qsweep, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemPerSM / 2 - 1024);
}

int qsweep_launch(const EsParams& p, const QsLayout& q, int grid, cudaStream_t st) {
  k_qcarry<<<(unsigned)(p.B * kQcParts), 256, 0, st>>>(p);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return (int)e;   // (the sweep adds to what k_qcarry writes)
  k_qsweep<<<grid, kQsThreads, q.bytes, st>>>(p, q.ww, q.supers);
  return (int)cudaGetLastError();
}

}  // namespace bw
