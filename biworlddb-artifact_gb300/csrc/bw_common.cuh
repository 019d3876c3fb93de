// bw_common.cuh -- device helpers shared by the GB300 kernels.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>

#if defined(__CUDA_ARCH__)
#define BW_ARCH_TAG (__CUDA_ARCH__)
#else
#define BW_ARCH_TAG 1030
#endif

namespace bw {

__host__ __device__ __forceinline__ int64_t imin64(int64_t a, int64_t b) { return a < b ? a : b; }

// ------------------------------------------------------------------ rank LUT
// Rank of key offset x inside a slice: popcount rank table + bitmap word, the
// CSR rank-LUT probe of sparse_engine.hpp:77-86 (rlut + popcount(word & mask)).
__device__ __forceinline__ uint32_t local_rank(const uint64_t* bits, const uint32_t* rl, uint32_t x) {
  const uint32_t wi = x >> 6;
  const uint64_t m = (1ull << (x & 63)) - 1ull;
  return rl[wi] + (uint32_t)__popcll(bits[wi] & m);
}

// Exact 64-bit add into a shared-memory word with two 32-bit atomics.  The low
// word's atomic returns its old value; its unsigned overflow is the carry into the
// high word.  Any interleaving of such adds leaves (hi:lo) equal to the sum modulo
// 2^64 once all of them have completed (readers wait at a barrier).  On sm_103 a
// contended 64-bit shared atomicAdd is one to two orders of magnitude slower than
// this pair (measured: 22.6 ms vs 0.53 ms for 512k adds per SM on one address).
__device__ __forceinline__ void shared_add_u64(unsigned long long* addr, uint64_t v) {
  unsigned* w = reinterpret_cast<unsigned*>(addr);
  const unsigned lo = (unsigned)v;
  const unsigned old = atomicAdd(w, lo);
  const unsigned hi = (unsigned)(v >> 32) + ((old + lo) < old ? 1u : 0u);
  if (hi) atomicAdd(w + 1, hi);
}

// Set bit b of a shared-memory bitmap of 64-bit words with a 32-bit atomic.
__device__ __forceinline__ void shared_set_bit(uint64_t* words, uint32_t b) {
  atomicOr(reinterpret_cast<unsigned*>(words) + (b >> 5), 1u << (b & 31));
}

// Fenwick point update at 1-based index i over n nodes (one thread).
__device__ __forceinline__ void fenwick_add(unsigned long long* fen, uint32_t n, uint32_t i, uint64_t d) {
  for (; i <= n; i += i & (0u - i)) shared_add_u64(fen + i, d);
}

__device__ __forceinline__ uint64_t fenwick_prefix(const unsigned long long* fen, uint32_t r) {
  uint64_t s = 0;
  for (uint32_t i = r; i; i &= i - 1) s += fen[i];
  return s;
}

// Prefix (keys < k) of the current slice's contribution: 0 below the slice, the
// slice total above it, the Fenwick prefix at the key's rank inside it.
__device__ __forceinline__ uint64_t slice_prefix(const unsigned long long* fen, uint32_t n, const uint64_t* bits,
                                                 const uint32_t* rl, uint32_t klo, uint32_t khi, uint32_t k) {
  if (k <= klo) return 0;
  if (k >= khi) return fenwick_prefix(fen, n);
  return fenwick_prefix(fen, local_rank(bits, rl, k - klo));
}

// ------------------------------------------------------------------ block scans
// Block-wide exclusive scan of a per-thread value; returns the block total.
template <typename T>
__device__ __forceinline__ T block_exclusive_scan(T v, T* total_out = nullptr) {
  __shared__ T s_warp[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  T x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const T y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) s_warp[warp] = x;
  __syncthreads();
  if (warp == 0) {
    T w = lane < nw ? s_warp[lane] : (T)0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const T y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    s_warp[lane] = w;  // inclusive warp totals
  }
  __syncthreads();
  const T before = (warp ? s_warp[warp - 1] : (T)0) + x - v;
  const T total = s_warp[nw - 1];
  __syncthreads();
  if (total_out) *total_out = total;
  return before;
}

// out[i] = sum_{j<i} popcount(bits[j]) for i in [0, n]; returns the total.
__device__ __forceinline__ uint32_t block_exclusive_scan_popc(const uint64_t* bits, uint32_t* out, int n) {
  const int per = (n + blockDim.x - 1) / blockDim.x;
  const int lo = threadIdx.x * per, hi = min(n, lo + per);
  uint32_t local = 0;
  for (int i = lo; i < hi; ++i) local += (uint32_t)__popcll(bits[i]);
  uint32_t total = 0;
  uint32_t run = block_exclusive_scan<uint32_t>(local, &total);
  for (int i = lo; i < hi; ++i) {
    out[i] = run;
    run += (uint32_t)__popcll(bits[i]);
  }
  if (threadIdx.x == 0) out[n] = total;
  __syncthreads();
  return total;
}

// In-place exclusive scan of a[0..n) (uint64, wrapping).
__device__ __forceinline__ void block_exclusive_scan_u64(unsigned long long* a, uint32_t n) {
  const uint32_t per = (n + blockDim.x - 1) / blockDim.x;
  const uint32_t lo = threadIdx.x * per, hi = min(n, lo + per);
  uint64_t local = 0;
  for (uint32_t i = lo; i < hi; ++i) local += a[i];
  uint64_t run = block_exclusive_scan<uint64_t>(local);
  for (uint32_t i = lo; i < hi; ++i) {
    const uint64_t v = a[i];
    a[i] = run;
    run += v;
  }
  __syncthreads();
}

// ------------------------------------------------------------------ chained launches
// A chain of short kernels, each launched while the one before still runs: a kernel that
// is launched by launch_chained() calls chain_wait() first, which lets its successor's CTAs
// come onto the GPU and then waits until everything before it is done and visible.  Only
// what the kernels of a chain hand on matters here, so that must not be read through the
// non-coherent path (__ldg, const __restrict__), whose loads may move ahead of the wait.
// Saves 1.5 to 2 us a launch (building the tours of 46 trees, 24 kernels: 111 -> 67 us).
// Long kernels (`early` false) are launched the ordinary way: successors that wait for them
// take places on the SMs unevenly (4,096 trees, 27M states: 1.33 -> 1.46 ms).
__device__ __forceinline__ void chain_wait() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
}
constexpr int64_t kChainedStates = (int64_t)1 << 24;   // tours of fewer states are chained (7M: 375 -> 326 us)
template <typename... P, typename... A>
inline cudaError_t launch_chained(bool early, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                                  A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at = {};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = early ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

// ------------------------------------------------------------------ device scan
// Kernels below have internal linkage: every translation unit that includes this
// header gets its own copy.
namespace {
constexpr int kScanThreads = 512;
constexpr int kScanPer = 8;
constexpr int64_t kScanTile = (int64_t)kScanThreads * kScanPer;

inline size_t scan_tmp_bytes(size_t n) { return ((n + kScanTile - 1) / kScanTile + 1) * 8; }

// T: int64_t or uint32_t (sums wrap).  A warp takes 256 consecutive elements in rounds
// of one 16-byte vector per lane, so every access is coalesced (eight consecutive
// elements per thread touched each sector in eight separate loads).  x is 16-byte aligned.
template <typename T>
struct ScanItems {
  static constexpr int V = 16 / sizeof(T), R = kScanPer / V;
  alignas(16) T v[R][V];
  __device__ __forceinline__ static int64_t at(int r) {
    return (int64_t)blockIdx.x * kScanTile + (int64_t)(threadIdx.x >> 5) * (32 * kScanPer) +
           (int64_t)r * (32 * V) + (int64_t)(threadIdx.x & 31) * V;
  }
  __device__ __forceinline__ void load(const T* x, int64_t n) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int64_t i = at(r);
      if (i + V <= n) {
        *reinterpret_cast<uint4*>(v[r]) = *reinterpret_cast<const uint4*>(x + i);
      } else {
#pragma unroll
        for (int j = 0; j < V; ++j) v[r][j] = i + j < n ? x[i + j] : (T)0;
      }
    }
  }
};
template <typename T>
__global__ void __launch_bounds__(kScanThreads) k_scan_reduce(const T* x, int64_t n, T* part, const int32_t* n_dev) {
  chain_wait();
  if (n_dev) n = imin64(n, *n_dev);
  if ((int64_t)blockIdx.x * kScanTile >= n) return;
  ScanItems<T> it;
  it.load(x, n);
  uint64_t s = 0;
#pragma unroll
  for (int r = 0; r < it.R; ++r)
#pragma unroll
    for (int j = 0; j < it.V; ++j) s += (uint64_t)it.v[r][j];
  uint64_t total = 0;
  block_exclusive_scan<uint64_t>(s, &total);
  if (threadIdx.x == 0) part[blockIdx.x] = (T)total;
}
// Exclusive scan of the tile totals in place, where they are too many for every tile's CTA
// to sum the totals before its own (kScanSelf).
constexpr int64_t kScanSelf = 2048;
template <typename T>
__global__ void k_scan_parts(T* part, int64_t n, const int32_t* n_dev) {
  chain_wait();
  // single CTA: exclusive scan of the tile totals in place
  if (n_dev) n = imin64(n, *n_dev);
  const int64_t np = (n + kScanTile - 1) / kScanTile;
  uint64_t carry = 0;
  for (int64_t c0 = 0; c0 < np; c0 += blockDim.x) {
    const int64_t i = c0 + threadIdx.x;
    const uint64_t v = i < np ? (uint64_t)part[i] : 0;
    uint64_t total = 0;
    const uint64_t ex = block_exclusive_scan<uint64_t>(v, &total);
    if (i < np) part[i] = (T)(carry + ex);
    carry += total;
  }
}
template <typename T>
__global__ void __launch_bounds__(kScanThreads) k_scan_apply(T* x, int64_t n, const T* part, int self,
                                                             const int32_t* n_dev) {
  chain_wait();
  if (n_dev) n = imin64(n, *n_dev);
  if ((int64_t)blockIdx.x * kScanTile >= n) return;
  __shared__ uint64_t s_warp[kScanThreads / 32], s_part[kScanThreads / 32];
  using I = ScanItems<T>;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  I it;
  it.load(x, n);
  uint64_t ahead = 0;   // (self) the totals of the tiles before this one
  if (self) {
#pragma unroll
    for (int j = 0; j < kScanSelf / kScanThreads; ++j) {
      const int t = j * kScanThreads + threadIdx.x;
      ahead += t < (int)blockIdx.x ? (uint64_t)part[t] : 0;
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) ahead += __shfl_xor_sync(0xffffffffu, ahead, o);
  }
  uint64_t before[I::R], run = 0;   // sum of the warp's elements before this lane's vector of round r
#pragma unroll
  for (int r = 0; r < I::R; ++r) {
    uint64_t s = 0;
#pragma unroll
    for (int j = 0; j < I::V; ++j) s += (uint64_t)it.v[r][j];
    uint64_t incl = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint64_t y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    before[r] = run + incl - s;
    run += __shfl_sync(0xffffffffu, incl, 31);
  }
  if (lane == 0) {
    s_warp[warp] = run;
    s_part[warp] = ahead;
  }
  __syncthreads();
  uint64_t base = self ? 0 : (uint64_t)part[blockIdx.x];
  if (self)
    for (int w = 0; w < kScanThreads / 32; ++w) base += s_part[w];
  for (int w = 0; w < warp; ++w) base += s_warp[w];
#pragma unroll
  for (int r = 0; r < I::R; ++r) {
    uint64_t acc = base + before[r];
#pragma unroll
    for (int j = 0; j < I::V; ++j) {
      acc += (uint64_t)it.v[r][j];
      it.v[r][j] = (T)acc;
    }
    const int64_t i = I::at(r);
    if (i + I::V <= n) {
      *reinterpret_cast<uint4*>(x + i) = *reinterpret_cast<const uint4*>(it.v[r]);
    } else {
#pragma unroll
      for (int j = 0; j < I::V; ++j)
        if (i + j < n) x[i + j] = it.v[r][j];
    }
  }
}

// Inclusive scan of x[0..n) in place (two launches, three above 8M elements, counted into
// `kernels`); tmp holds scan_tmp_bytes(n).  n_dev: the count on the device, n its upper bound.
template <typename T>
inline int device_inclusive_scan(T* x, int64_t n, void* tmp, cudaStream_t st, int& kernels,
                                 const int32_t* n_dev = nullptr) {
  if (n <= 0) return 0;
  const int64_t np = (n + kScanTile - 1) / kScanTile;
  const bool self = np <= kScanSelf, early = n < 2 * kChainedStates;
  cudaError_t e = launch_chained(early, k_scan_reduce<T>, (unsigned)np, kScanThreads, 0, st, x, n, static_cast<T*>(tmp), n_dev);
  if (e == cudaSuccess && !self) e = launch_chained(early, k_scan_parts<T>, 1, 1024, 0, st, static_cast<T*>(tmp), n, n_dev);
  if (e == cudaSuccess)
    e = launch_chained(early, k_scan_apply<T>, (unsigned)np, kScanThreads, 0, st, x, n, static_cast<const T*>(tmp),
                       self ? 1 : 0, n_dev);
  kernels += self ? 2 : 3;
  return (int)e;
}
inline int device_inclusive_scan_i64(int64_t* x, int64_t n, int64_t* tmp, cudaStream_t st, int& kernels) {
  return device_inclusive_scan<int64_t>(x, n, tmp, st, kernels);
}

}  // namespace
}  // namespace bw
