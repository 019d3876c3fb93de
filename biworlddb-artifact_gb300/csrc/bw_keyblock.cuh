// bw_keyblock.cuh -- one-tree replay over large key domains (bw_keyblock.cu).
#pragma once
#include <cuda_runtime.h>
#include <cstdint>

#include "bw_gpu.h"
#include "bw_pipeline.cuh"

namespace bw {

constexpr int kKbMaxBlocks = 4096;            // key blocks (partition digits held in shared memory)
constexpr int kKbSlotStep = 512;              // slots per block: a multiple of 16 warps x 32 lanes ...
constexpr int kKbMaxSlots = 16 * kKbSlotStep; // ... and at most 8,192 (64 KB of int64: three CTAs per SM)
constexpr int kSwCtas = 3;                    // sweep CTAs per SM
constexpr int kKbPtTile = 4096;               // points per partition tile
constexpr int kKbPrTile = 4096;               // queries per partition tile (two probes each)
// Domains up to kKbMinKeys (one window of the state-block path) stay with the state-block
// pipeline.  Around the line the two
// paths are close where there is work for both: 30,000 states, state blocks / key blocks, us, 262,145
// keys: 1M events, 1M queries 939 / 952, 10M events, 10,000 queries 1,492 / 2,832; 600,000 keys 1,984 /
// 956 and 2,518 / 2,840; 300 states, 262,145 keys 880 / 585 and 3,350 / 2,796.
constexpr uint32_t kKbMinKeys = 1u << kWinBits;

enum {
  KB_SOFF, KB_TEOFF, KB_TQOFF, KB_TC, KB_TBOFF, KB_TBITS, KB_TCARRY, KB_TGSUM, KB_LASTQ, KB_TTOFF, KB_MISC, KB_EOFF, KB_QOFF,
  KB_FORK, KB_NEXT, KB_CNT, KB_EHEAD, KB_XHEAD, KB_RANK, KB_SCAN, KB_STEP, KB_W, KB_EP, KB_TIME, KB_COLSTATE,
  KB_COLTIME, KB_COLSTEP, KB_POS, KB_TOUR, KB_PTHIST, KB_PTOFF, KB_PTS, KB_SEG, KB_CUT, KB_ROWS, KB_PRHIST,
  KB_PROFF, KB_MORE, KB_PART, KB_PRS, KB_ACC, KB_COUNT
};

struct KbSpec {
  int32_t S = 0;
  uint32_t C = 0;
  int64_t E = 0, Q = 0;
  int32_t m = 0;           // event slots per key block
  int32_t B = 0;           // key blocks
  int32_t segs = 0;        // tour segments of the row pass
  int64_t pt_tiles = 0, pr_tiles = 0;
  size_t off[KB_COUNT];
  size_t total = 0;
};

// Whether a replay that would take the general pipeline (spec `s`, workspace
// `general_bytes`) is replayed by key blocks instead; fills `k` when it is.
bool kb_select(const BwReplayArgs* a, const PipeSpec& s, size_t general_bytes, KbSpec& k);
int kb_enqueue(const KbSpec& k, const PipeSpec& s, const BwReplayArgs* a, EventSet* timing, int* kernels);
const int32_t* kb_status_word(const KbSpec& k, const void* workspace);

}  // namespace bw
