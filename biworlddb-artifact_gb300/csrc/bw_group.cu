// bw_group.cu -- grouping ungrouped event and query arrays by state on the device
// (bw_group_events, bw_group_queries; include/bw_gpu.h).
//
// The replay takes events and queries grouped by state.  A caller whose records
// arrive in another order (an event stream, a log merged from several writers)
// groups them here: a stable LSD radix sort of 16-byte records by their u32 state,
// 8 bits per pass over the bits the state count needs (three passes up to 16.7M
// states; the passes are those of bw_sort.cuh).  Queries travel as 16-byte records
// (state, lo, hi, input index) so the caller gets, beside the grouped queries, the
// input position of each one (bw_scatter_answers puts the answers back in input
// order); the first pass packs them and the last one writes the two arrays, so they
// cost no pass of their own.  The first pass also checks every state against the state
// count (BW_STATUS_STATE_RANGE in the status word).
#include <cuda_runtime.h>
#include <cstdint>
#include <cstdio>

#include "bw_gpu.h"
#include "bw_common.cuh"
#include "bw_sort.cuh"

namespace bw {
namespace {

inline size_t al256(size_t x) { return (x + 255) & ~size_t(255); }

// Sort pass over records by their first word.  QIN: the pass reads 12-byte queries and
// carries each one's input index as the record's last word; QOUT: it writes the queries
// and the indexes apart.
template <bool QIN, bool QOUT>
struct GrpIO {
  const void* in;
  void* out;
  int64_t* order;
  uint32_t n_states;
  static constexpr int kBadStatus = BW_STATUS_STATE_RANGE;
  __device__ __forceinline__ uint4 load(int64_t i) const {
    if constexpr (QIN) {
      const BwQuery q = static_cast<const BwQuery*>(in)[i];
      return make_uint4(q.state, q.lo, q.hi, (uint32_t)i);
    } else {
      return static_cast<const uint4*>(in)[i];
    }
  }
  __device__ __forceinline__ uint32_t state(int64_t i) const {
    if constexpr (QIN) return static_cast<const BwQuery*>(in)[i].state;
    else return static_cast<const uint4*>(in)[i].x;
  }
  __device__ __forceinline__ uint32_t key(int64_t i, int shift) const { return state(i) >> shift; }
  __device__ __forceinline__ bool bad(int64_t i) const { return state(i) >= n_states; }
  static __device__ __forceinline__ uint32_t digits(const uint4& x, int shift) { return x.x >> shift; }
  __device__ __forceinline__ void store(int64_t at, const uint4& x) const {
    if constexpr (QOUT) {
      static_cast<BwQuery*>(out)[at] = BwQuery{x.x, x.y, x.z};
      if (order) order[at] = (int64_t)x.w;
    } else {
      static_cast<uint4*>(out)[at] = x;
    }
  }
};

int grp_passes(int32_t n_states) {
  int bits = 0;
  while (bits < 32 && ((uint64_t)1 << bits) < (uint64_t)(n_states > 1 ? n_states : 1)) ++bits;
  return bits == 0 ? 1 : (bits + 7) / 8;
}

struct GrpLayout {
  RsLayout rs;
  size_t status, hist, part, base, rec_a, rec_b, total;
};
GrpLayout grp_layout(int64_t n, bool queries) {
  GrpLayout L;
  L.rs = rs_layout(n, 4);   // (the state count is not known here: at most four passes)
  size_t o = 0;
  L.status = o;  o = al256(o + 4);
  L.hist = o;    o = al256(o + L.rs.hist);
  L.part = o;    o = al256(o + L.rs.part);
  L.base = o;    o = al256(o + L.rs.base);
  L.rec_a = o;   o = al256(o + (size_t)n * 16);
  L.rec_b = o;   o = al256(o + (queries ? (size_t)n * 16 : 0));
  L.total = o;
  return L;
}

int grp_report(cudaError_t e, const char* what) {
  if (e == cudaSuccess) return 0;
  std::fprintf(stderr, "bw_group: %s: %s\n", what, cudaGetErrorString(e));
  return (int)e;
}

// The passes of a grouping share the counters in `ws`.
struct GrpSort {
  const GrpLayout& L;
  char* ws;
  int64_t n;
  uint32_t n_states;
  cudaStream_t st;
  int begin() const {
    const int rc = grp_report(cudaMemsetAsync(ws + L.status, 0, 4, st), "status reset");
    return rc ? rc : grp_report(cudaMemsetAsync(ws + L.part, 0, L.rs.part, st), "counter reset");
  }
  template <bool QIN, bool QOUT>
  int pass(int p, const void* in, void* out, int64_t* order = nullptr) const {
    const GrpIO<QIN, QOUT> io{in, out, order, n_states};
    return grp_report((cudaError_t)rs_pass(io, n, 8 * p, L.rs, reinterpret_cast<uint32_t*>(ws + L.hist),
                                           reinterpret_cast<uint32_t*>(ws + L.part) + (size_t)p * L.rs.chunks * kRsDigits,
                                           reinterpret_cast<uint64_t*>(ws + L.base), p == 0,
                                           reinterpret_cast<int32_t*>(ws + L.status), st), "sort pass");
  }
};

}  // namespace
}  // namespace bw

using namespace bw;

extern "C" int bw_group_workspace_size(int64_t n, int32_t queries, size_t* bytes) {
  if (n < 0 || !bytes) return BW_EINVAL;
  *bytes = grp_layout(n, queries != 0).total;
  return 0;
}

extern "C" int bw_group_events(const BwEvent* in, int64_t n, int32_t n_states, BwEvent* out, void* workspace,
                               size_t workspace_bytes, void* stream) {
  if (n < 0 || n_states < 1 || (n && (!in || !out || (const void*)in == (const void*)out))) return BW_EINVAL;
  const GrpLayout L = grp_layout(n, false);
  if (!workspace || workspace_bytes < L.total) return BW_EINVAL;
  if ((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out)) & 15) return BW_EINVAL;
  if (n == 0) return 0;
  char* ws = static_cast<char*>(workspace);
  const GrpSort g{L, ws, n, (uint32_t)n_states, static_cast<cudaStream_t>(stream)};
  const int passes = grp_passes(n_states);
  int rc = g.begin();
  const void* src = in;
  for (int p = 0; p < passes && !rc; ++p) {
    void* dst = ((passes - p) % 2 == 1) ? static_cast<void*>(out) : ws + L.rec_a;   // the last pass lands in out
    rc = g.pass<false, false>(p, src, dst);
    src = dst;
  }
  return rc;
}

extern "C" int bw_group_queries(const BwQuery* in, int64_t n, int32_t n_states, BwQuery* out, int64_t* order,
                                void* workspace, size_t workspace_bytes, void* stream) {
  if (n < 0 || n_states < 1 || n >= ((int64_t)1 << 32) || (n && (!in || !out))) return BW_EINVAL;
  const GrpLayout L = grp_layout(n, true);
  if (!workspace || workspace_bytes < L.total) return BW_EINVAL;
  if (n == 0) return 0;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  char* ws = static_cast<char*>(workspace);
  const GrpSort g{L, ws, n, (uint32_t)n_states, st};
  const int passes = grp_passes(n_states);
  int rc = g.begin();
  if (rc) return rc;
  if (passes == 1) {
    const void* src = in;
    if (in == out) {   // a single pass reads while it writes
      if ((rc = grp_report(cudaMemcpyAsync(ws + L.rec_a, in, (size_t)n * sizeof(BwQuery), cudaMemcpyDeviceToDevice, st),
                           "query copy")))
        return rc;
      src = ws + L.rec_a;
    }
    return g.pass<true, true>(0, src, out, order);
  }
  // records of 16 bytes between the first pass and the last
  char* rec[2] = {ws + L.rec_a, ws + L.rec_b};
  rc = g.pass<true, false>(0, in, rec[0]);
  for (int p = 1; p + 1 < passes && !rc; ++p) rc = g.pass<false, false>(p, rec[(p - 1) & 1], rec[p & 1]);
  return rc ? rc : g.pass<false, true>(passes - 1, rec[(passes - 2) & 1], out, order);
}

extern "C" int bw_group_status(const void* workspace, int32_t* status) {
  if (!workspace || !status) return BW_EINVAL;
  return grp_report(cudaMemcpy(status, workspace, 4, cudaMemcpyDeviceToHost), "status read");
}
