// bw_search.cuh -- bisection shared by device code and by host programs that check it.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define BW_HD __host__ __device__ __forceinline__
#else
#define BW_HD inline
#endif

namespace bw {

// First x in [lo, hi] with after(x), true from some x on and taken as true at hi.  Bounds
// up to 2^31 - 1: lo + hi may not fit 32 bits (a tour has up to 2^31 - 2 steps).
template <typename F>
BW_HD int32_t first_after(int32_t lo, int32_t hi, F&& after) {
  while (lo < hi) {
    const int32_t mid = lo + ((hi - lo) >> 1);
    if (after(mid)) hi = mid; else lo = mid + 1;
  }
  return lo;
}

}  // namespace bw
