// bw_sort.cuh -- stable radix partition of 16-byte items, 8 bits a pass, shared by the
// sparse-key index build and the grouping by state.
//
// A pass is three kernels: k_rs_hist counts the digits of every 2,048-item tile
// (tile-major, so every access runs along the digits) and adds them to its chunk of
// tiles; k_rs_start turns the counts into starts (digit totals and earlier chunks are
// summed by every chunk's CTA, then a prefix down its tiles); k_rs_scatter ranks a tile
// and writes it digit by digit.  Ranks inside a warp come from eight ballots a round: with
// 32 distinct digits __match_any_sync took some 400 cycles.  The tile is put in digit order
// in shared memory first, so that a warp's store covers four or five runs of
// consecutive addresses instead of 32.  Tiles of 256 threads and eight items, four CTAs an
// SM: longer runs cost more in occupancy than they save (index build of 20M pairs: 4,096 items
// 1,392 us, 2,048 1,344 to 1,362, 1,536 1,415, 2,560 1,360, 8,192 1,540).
// Measured on 20M 16-byte pairs, before and after with tiles of 4,096: scatter 455 -> 158 us a
// pass (4.1 TB/s), counts 46 -> 32; with 2,048 scatter 142.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>

#include "bw_common.cuh"

namespace bw {
namespace {

constexpr int kRsThreads = 256, kRsWarps = kRsThreads / 32, kRsItems = 8;
constexpr int kRsTile = kRsThreads * kRsItems;
constexpr int kRsDigits = 256;
constexpr int kRsChunks = 128;            // chunks of tiles (at most; a multiple of 64)
constexpr size_t kRsSmem = (size_t)kRsTile * 16;

struct RsLayout {
  int64_t tiles = 0;
  int32_t chunks = 0, passes = 0;
  // sizes of the workspace arrays: counts per tile, counts per chunk (one table a
  // pass, zeroed together), starts per chunk
  size_t hist = 0, part = 0, base = 0;
};
inline RsLayout rs_layout(int64_t n, int passes) {
  RsLayout L;
  L.tiles = (n + kRsTile - 1) / kRsTile;
  if (L.tiles < 1) L.tiles = 1;
  L.chunks = (int32_t)(L.tiles < kRsChunks ? L.tiles : kRsChunks);
  L.passes = passes;
  L.hist = (size_t)L.tiles * kRsDigits * 4;
  L.part = (size_t)passes * L.chunks * kRsDigits * 4;
  L.base = (size_t)L.chunks * kRsDigits * 8;
  return L;
}
__host__ __device__ inline int64_t rs_chunk_start(int64_t tiles, int32_t chunks, int32_t c) {
  return tiles * c / chunks;
}

// IO: digit source and item moves of a pass.
//   uint4 load(int64_t i); uint32_t key(int64_t i, int shift): (the item's key >> shift);
//   static uint32_t digits(uint4, int shift); void store(int64_t at, uint4);
//   bool bad(int64_t i): the first pass's input check.
template <typename IO>
__global__ void __launch_bounds__(kRsThreads) k_rs_hist(IO io, int64_t n, int shift, int64_t tiles, int32_t chunks,
                                                        uint32_t* hist, uint32_t* part, int check, int32_t* status) {
  chain_wait();
  __shared__ uint32_t cnt[kRsDigits];
  if (threadIdx.x < kRsDigits) cnt[threadIdx.x] = 0;
  __syncthreads();
  const int64_t base = (int64_t)blockIdx.x * kRsTile;
  uint32_t d[kRsItems];
  bool bad = false;
#pragma unroll
  for (int j = 0; j < kRsItems; ++j) {
    const int64_t i = base + j * kRsThreads + threadIdx.x;
    d[j] = kRsDigits;
    if (i < n) {
      d[j] = io.key(i, shift) & (kRsDigits - 1);
      if (check) bad |= io.bad(i);
    }
  }
#pragma unroll
  for (int j = 0; j < kRsItems; ++j)
    if (d[j] < kRsDigits) atomicAdd(cnt + d[j], 1u);
  if (bad) atomicCAS(status, 0, IO::kBadStatus);
  __syncthreads();
  if (threadIdx.x < kRsDigits) {
    const uint32_t c = cnt[threadIdx.x];
    hist[(int64_t)blockIdx.x * kRsDigits + threadIdx.x] = c;
    // the chunk of this tile: the last one that starts at or before it
    int32_t k = (int32_t)((int64_t)blockIdx.x * chunks / tiles);
    while (k + 1 < chunks && rs_chunk_start(tiles, chunks, k + 1) <= blockIdx.x) ++k;
    if (c) atomicAdd(part + (int64_t)k * kRsDigits + threadIdx.x, c);
  }
}

// Counts -> starts: base[chunk][d] = items of smaller digits + those of earlier chunks,
// hist[tile][d] = those of the chunk's earlier tiles.  Every chunk's CTA sums all chunks,
// four groups of threads a quarter each (one group took 27 us for twice as many chunks), and the
// groups take a quarter of the chunk's tiles each (one group took 21 us for 38 tiles a chunk,
// four 9.5, and 12.5 for 76).
__global__ void __launch_bounds__(4 * kRsDigits) k_rs_start(uint32_t* hist, const uint32_t* part, int64_t tiles,
                                                            int32_t chunks, uint64_t* base) {
  chain_wait();
  __shared__ uint64_t s_total[4][kRsDigits], s_before[4][kRsDigits];
  __shared__ uint32_t s_tiles[4][kRsDigits];
  const int d = threadIdx.x & (kRsDigits - 1), g = threadIdx.x / kRsDigits;
  // this group's tiles of the chunk: the first 16 stay in registers
  const int64_t t0 = rs_chunk_start(tiles, chunks, blockIdx.x), t1 = rs_chunk_start(tiles, chunks, blockIdx.x + 1);
  const int64_t q0 = t0 + (t1 - t0) * g / 4, q1 = t0 + (t1 - t0) * (g + 1) / 4;
  uint32_t first[16], sum = 0;
#pragma unroll
  for (int i = 0; i < 16; ++i) first[i] = q0 + i < q1 ? hist[(q0 + i) * kRsDigits + d] : 0u;
  uint64_t total = 0, before = 0;
  for (int32_t c0 = 0; c0 < kRsChunks / 4; c0 += 16) {
    uint32_t x[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const int32_t c = 4 * (c0 + i) + g;
      x[i] = c < chunks ? part[(int64_t)c * kRsDigits + d] : 0u;
    }
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      total += x[i];
      before += 4 * (c0 + i) + g < (int32_t)blockIdx.x ? x[i] : 0u;
    }
  }
#pragma unroll
  for (int i = 0; i < 16; ++i) sum += first[i];
  for (int64_t t = q0 + 16; t < q1; ++t) sum += hist[t * kRsDigits + d];
  s_total[g][d] = total;
  s_before[g][d] = before;
  s_tiles[g][d] = sum;
  __syncthreads();
  total = g == 0 ? s_total[0][d] + s_total[1][d] + s_total[2][d] + s_total[3][d] : 0;
  const uint64_t start = block_exclusive_scan<uint64_t>(total);
  if (g == 0)
    base[(int64_t)blockIdx.x * kRsDigits + d] =
        start + s_before[0][d] + s_before[1][d] + s_before[2][d] + s_before[3][d];
  uint32_t run = 0;
  for (int h = 0; h < g; ++h) run += s_tiles[h][d];
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    if (q0 + i < q1) hist[(q0 + i) * kRsDigits + d] = run;
    run += first[i];
  }
  for (int64_t t = q0 + 16; t < q1; t += 16) {   // in place: a batch is read before it is written
    uint32_t x[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) x[i] = t + i < q1 ? hist[(t + i) * kRsDigits + d] : 0u;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      if (t + i < q1) hist[(t + i) * kRsDigits + d] = run;
      run += x[i];
    }
  }
}

template <typename IO>
__global__ void __launch_bounds__(kRsThreads, 4) k_rs_scatter(IO io, int64_t n, int shift, int64_t tiles,
                                                              int32_t chunks, const uint32_t* hist,
                                                              const uint64_t* base) {
  chain_wait();
  extern __shared__ __align__(16) uint4 stage[];          // kRsTile
  __shared__ uint16_t wcnt[kRsWarps][kRsDigits];
  __shared__ uint64_t gbase[kRsDigits];                    // output position of local position 0 of the digit
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  for (int i = tid; i < kRsWarps * kRsDigits / 8; i += kRsThreads)
    reinterpret_cast<uint4*>(&wcnt[0][0])[i] = make_uint4(0, 0, 0, 0);
  const int64_t t0 = (int64_t)blockIdx.x * kRsTile;
  const int count = (int)imin64(kRsTile, n - t0);
  uint4 it[kRsItems];
#pragma unroll
  for (int j = 0; j < kRsItems; ++j) {
    const int i = (warp * kRsItems + j) * 32 + lane;
    it[j] = i < count ? io.load(t0 + i) : make_uint4(0, 0, 0, 0);
  }
  __syncthreads();
  const unsigned lt = (1u << lane) - 1u;
  uint16_t* wc = wcnt[warp];
  uint16_t r[kRsItems];
#pragma unroll
  for (int j = 0; j < kRsItems; ++j) {
    const bool in = (warp * kRsItems + j) * 32 + lane < count;
    const uint32_t d = IO::digits(it[j], shift) & (kRsDigits - 1);
    unsigned peers = __ballot_sync(0xffffffffu, in);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const bool one = (d >> k) & 1u;
      const unsigned m = __ballot_sync(0xffffffffu, one);
      peers &= one ? m : ~m;
    }
    const uint32_t old = wc[d];
    __syncwarp();
    r[j] = (uint16_t)(old + __popc(peers & lt));
    if (in && (peers & lt) == 0) wc[d] = (uint16_t)(old + __popc(peers));
    __syncwarp();
  }
  __syncthreads();
  uint32_t total = 0;
  if (tid < kRsDigits) {
#pragma unroll
    for (int w = 0; w < kRsWarps; ++w) {
      const uint32_t c = wcnt[w][tid];
      wcnt[w][tid] = (uint16_t)total;
      total += c;
    }
  }
  const uint32_t start = block_exclusive_scan<uint32_t>(total);   // (every thread: a CTA-wide scan)
  if (tid < kRsDigits) {
#pragma unroll
    for (int w = 0; w < kRsWarps; ++w) wcnt[w][tid] = (uint16_t)(wcnt[w][tid] + start);
    int32_t k = (int32_t)((int64_t)blockIdx.x * chunks / tiles);
    while (k + 1 < chunks && rs_chunk_start(tiles, chunks, k + 1) <= blockIdx.x) ++k;
    gbase[tid] = base[(int64_t)k * kRsDigits + tid] + hist[(int64_t)blockIdx.x * kRsDigits + tid] - start;
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kRsItems; ++j)
    if ((warp * kRsItems + j) * 32 + lane < count)
      stage[wc[IO::digits(it[j], shift) & (kRsDigits - 1)] + r[j]] = it[j];
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kRsItems; ++j) {
    const int i = j * kRsThreads + tid;
    if (i < count) {
      const uint4 x = stage[i];
      io.store((int64_t)(gbase[IO::digits(x, shift) & (kRsDigits - 1)] + i), x);
    }
  }
}

// One pass; `part` is this pass's zeroed chunk table.
template <typename IO>
inline int rs_pass(const IO& io, int64_t n, int shift, const RsLayout& L, uint32_t* hist, uint32_t* part,
                   uint64_t* base, bool check, int32_t* status, cudaStream_t st) {
  const cudaError_t attr = cudaFuncSetAttribute(k_rs_scatter<IO>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                (int)kRsSmem);   // (of the current device)
  if (attr != cudaSuccess) return (int)attr;
  // (chained launches: 20M pairs, five passes 1,433 -> 1,396 us an index build, 1.3M 323 -> 291)
  cudaError_t e = launch_chained(true, k_rs_hist<IO>, (unsigned)L.tiles, kRsThreads, 0, st, io, n, shift, L.tiles,
                                 L.chunks, hist, part, check ? 1 : 0, status);
  if (e == cudaSuccess)
    e = launch_chained(true, k_rs_start, L.chunks, 4 * kRsDigits, 0, st, hist, part, L.tiles, L.chunks, base);
  if (e == cudaSuccess)
    e = launch_chained(true, k_rs_scatter<IO>, (unsigned)L.tiles, kRsThreads, kRsSmem, st, io, n, shift, L.tiles,
                       L.chunks, hist, base);
  return (int)e;
}

}  // namespace
}  // namespace bw
