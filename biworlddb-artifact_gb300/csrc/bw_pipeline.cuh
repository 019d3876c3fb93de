// bw_pipeline.cuh -- the version-forest replay pipeline shared by the plain entry
// (bw_replay_*, one tree) and the batched entry (bw_forest_*, many trees).
//
// A forest is a concatenation of independent version trees.  Tree t owns global
// states [s0, s0 + ns), events [e0, e0 + ne), queries [q0, q0 + nq) and a key
// domain [0, C); its parent array, event states and query states are local to the
// tree (parent[local 0] = -1, parent[l] < l).  The pipeline lays every tree's
// Euler tour out at steps [2 s0, 2 s0 + 2 ns), cuts each tree into nb equal-work
// state blocks that never span trees, and replays all blocks of all trees with
// persistent CTAs that take blocks from a shared queue (largest first).
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include <vector>

#include "bw_gpu.h"

namespace bw {

// ------------------------------------------------------------------ constants
constexpr int kPrepThreads = 512;             // CTA width of the prepare kernel (two per SM)
constexpr int kWinBits = 18;                  // rank window: 2^18 keys per smem bitmap
constexpr int kWinWords = 1 << (kWinBits - 6);
constexpr int kMaxSlices = 256;               // key slices per block (single trees: see finish_spec)
constexpr int kSmemLimit = 232448;            // 227 KiB dynamic smem per CTA on sm_100/103
constexpr int kSmemPerSM = 233472;            // 228 KiB shared memory per SM
constexpr int kCarryGroup = 16;               // rows per group of the carry scan
constexpr int kCarryChunk = 256;              // columns per carry unit
constexpr int64_t kStepCost = 4;              // fixed cost of an Euler step, in event units
constexpr int64_t kQueryStepCost = 64;        // extra cost of a step with queries (two CTA barriers)
constexpr int64_t kQueryCost = 2;             // a query is two prefix probes
// Smallest block of a tree that does not fill the GPU (two blocks an SM), in est_work
// units.  At 65,536 a tree of 12,000 states and 200,000 events had 25 blocks and its sweep
// took 752 us, at 25,000 (64 blocks) 269 us; 50,000 states and 1M events 702 and 288 us.  The larger value stays for callers whose scratch the
// smaller blocks would outgrow.
constexpr int64_t kMinWork = 16384, kMinWorkCoarse = 65536;
// Above the coarse count and two events per unit of the block work, the blocks of one tree are
// at most sqrt(kRowWork work / (C + 1)): a block more shortens the longest one by work / B^2
// and adds a carry row of C + 1 words to write, scan and read.  300 states, 1,000 events, 1M
// queries: over 262,144 keys 30 / 68 / 123 blocks 322 / 376 / 774 us, over 16,000 keys 123 blocks
// 161 (30: 294 with the sweep of before); 300,000 states, 1,000 events, 5,000 queries over 262,144
// keys 41 / 79 / 166 blocks 327 / 379 / 544.  With events the longest block weighs more: 228
// states, 2.8M events, 51,613 queries over 259,872 keys 87 blocks 2,204, 304 blocks 794.  (With 300 in the
// place of 600: 51,240 states, 1,623 events, 1.6M queries, 51,174 keys 444, else 420.)
constexpr int64_t kRowWork = 600;
// A tour is contracted when at most one state in kContract has a query (see k_ct_nodes).
constexpr int64_t kContract = 2;
// Single trees take the query-step sweep where a state is asked kQueryDense queries and more
// and, below kQueryStates states (whose blocks' chains of steps leave the GPU part empty),
// where a step has work besides; else the Euler-tile sweep.  Query steps / Euler tiles, us a
// replay: 100,000 states, 5M events, 2M queries 745 / 905, 100,000 states, 4M events, 1.7M queries
// 710 / 684; 44,000 states, 1.7M events, 490,000 queries 502 / 395; 5,000 states, 60,000 events,
// 250,000 queries 365 / 274, 500,000 queries 217 / 311; 10,000 states, 2.5M events, 180,000
// queries 212 / 248.  (k_sweep, which trees with a query for every eight events took before,
// needs 829, 779 and 302 us where the Euler tiles need 684, 395 and 182.)
constexpr int64_t kQueryDense = 18;
constexpr int64_t kQueryStates = 20'000;
inline bool query_steps(int64_t S, int64_t E, int64_t Q) {
  return Q >= kQueryDense * S && (S >= kQueryStates || E / 4 + Q >= 60 * S);
}

// Estimated sweep work of a tree (or a whole forest) from its sizes: every event is
// applied on enter and on exit, every state is entered and left, and at most
// min(S, Q) steps carry queries.
__host__ __device__ inline int64_t est_work(int64_t S, int64_t E, int64_t Q) {
  return 2 * E + kQueryCost * Q + 2 * kStepCost * S + kQueryStepCost * (S < Q ? S : Q);
}

// Sweep geometry (see bw_pipeline.cu).
constexpr int kChunk = 256;
constexpr int kChunkBits = 8;
constexpr int kChunkLevels = 8;
constexpr int kChunkStride = 257;
constexpr int kMaxChunks = 128;
constexpr int kRebuildPer = 5;
constexpr int64_t kOfflinePairs = 32768;      // tile (queries x events) below which probes are batched
constexpr int kOfflineQ = 128;                // and at most this many queries (their sums live in smem)

// Sweep tile geometry: THREADS per CTA, EV events and QP queries staged per thread
// per tile, at most STEPS steps per tile, a ring of RING step descriptors refilled
// RING - 3 * STEPS (rounded down to whole warps) at a time: a refill during a tile's
// probes keeps the slots of that tile and the next two.
// COOP: the tile is staged cooperatively and made visible by a barrier (suits many
// small steps); otherwise every thread stages the items it will apply and probe
// itself and waits for its own copies only (suits few large, query-heavy steps).
// FLAT: the rank structure keeps plain values per rank with chunk totals (two
// atomics per update, probes summed by a warp: suits few queries per many events);
// otherwise a Fenwick tree inside every chunk (<= 9 atomics per update, probes by one
// thread: suits many queries).
// SPEC: warp-specialised: the last warp cuts and stages tiles (ring, tile cut,
// cp.async of events and queries) two tiles ahead into three buffers while the
// other warps replay, synchronised by one CTA barrier per tile and a consumer-only
// named barrier (flat chunks only).
template <int EV, int QP, int STEPS, int RING, int THREADS, bool COOP, bool FLAT, bool SPEC = false>
struct TileCfg {
  static constexpr bool kCoop = COOP, kFlat = FLAT, kSpec = SPEC;
  static constexpr int kBufs = SPEC ? 3 : 2;
  static constexpr int kEvPer = EV, kQPer = QP, kTileSteps = STEPS, kRing = RING,
                       kRingFill = (RING - 3 * STEPS) / 32 * 32;
  static constexpr int kThreads = THREADS, kWarps = THREADS / 32, kMinBlocks = THREADS >= 512 ? 1 : 2;
  static constexpr int kTileEv = EV * THREADS, kTileQ = QP * THREADS;
  static_assert((RING & (RING - 1)) == 0 && kRingFill >= STEPS && STEPS <= 128 && STEPS % 32 == 0,
                "tile ring too small");
  static_assert(!SPEC || (FLAT && !COOP && THREADS >= 128), "specialised tiles are flat, own staging");
};
using TileNarrow = TileCfg<2, 2, 32, 128, 256, false, false>;      // query-heavy steps: small staging, Fenwick
using TileWide = TileCfg<4, 1, 64, 256, 256, true, true>;          // event-heavy steps: deep staging, flat
using TileNarrow512 = TileCfg<2, 1, 128, 512, 512, false, true>;   // 16 warps (one CTA per SM), own staging, flat
using TileWide512 = TileCfg<2, 1, 64, 256, 512, true, true>;
using TileSpec512 = TileCfg<1, 1, 64, 512, 512, false, true, true>;   // 15 replay warps + 1 staging warp
// kTileQueryId: the query-step sweep of bw_qsweep.cu (a step at a time, a thread per
// event and per query bound; two CTAs per SM).
// kTileEulerId: the Euler-tile sweep of bw_esweep.cu (bulk-copied signed event tiles,
// flat window, a producer warp; one CTA per SM) instead of k_sweep.
enum { kTileAuto = 0, kTileNarrowId = 1, kTileWideId = 2, kTileNarrow512Id = 3, kTileWide512Id = 4, kTileSpec512Id = 5,
       kTileEulerId = 6, kTileQueryId = 7 };
constexpr int kTileMaxId = kTileEulerId;   // largest that a forest's tuning may name; the next is chosen only
// Window capacity of the Euler-tile sweep: int32 entries, or int64 ones in the same
// bytes (the prepare pass cuts its rank slices with the k_sweep window's capacities,
// 27,904 and 13,824 entries, which both fit).
constexpr uint32_t kEsCap32 = 27904;
constexpr uint32_t kEsCap64 = 13952;

// A step asked kHotQueries and more makes its block hot: the Euler-tile sweep leaves such blocks to a
// second kernel, launched where a forest or tree has kHotMin queries and more.
constexpr int kHotQueries = 316;
constexpr int64_t kHotMin = 2048;
enum { kMode32 = 1, kModeHot = 2 };   // of a block: int32 sums are exact; for the second kernel

// ------------------------------------------------------------------ records
struct StepDesc {        // one Euler step, 16 bytes
  uint32_t e0;           // first event of the node (global index)
  uint32_t q0;           // first query of the node (enter steps)
  int32_t ne;            // event count
  int32_t nq;            // query count on enter, -1 on exit
};

struct Slice {           // contiguous key range with <= cap distinct block keys
  int32_t word_lo, word_hi;  // bitmap words [word_lo, word_hi)
  uint32_t rank_lo;          // block-local rank of the first key of the slice
  uint32_t n;                // distinct keys in the slice
};

struct BlockTab {        // one state block, written on the device per launch
  int32_t tree, idx;     // tree and block index inside the tree
  int32_t t0, t1;        // steps [t0, t1)
  uint32_t C;            // key domain of the tree
  int32_t nwords;        // bitmap words of the domain
  int64_t bits_off;      // first bitmap word (rank table: bits_off + block index)
  int64_t carry_in;      // carry row read by the sweep (-1: the block starts its tree)
  int64_t carry_out;     // net-delta row written by prepare (-1: last block of its tree)
};

struct CarryUnit {       // 256 columns of one row group of one tree's carry rows
  int32_t tree, group, chunk, pad;
};

// Device-side tree tables (in the workspace).
struct TreeTabs {
  int32_t* soff;         // T+1 first global state
  int64_t* eoff;         // T+1 first event
  int64_t* qoff;         // T+1 first query
  uint32_t* C;           // T   key domain
  int32_t* boff;         // T+1 first block
  int64_t* bits;         // T   first bitmap word of the tree's blocks
  int64_t* carry;        // T   first carry word of the tree's rows
  int64_t* gsum;         // T   first group-sum word
  int32_t* last_q;       // T   last step answering a query + 1 (0: none)
  int32_t* noff;         // T+1 first tour node (states: soff; contracted: written per launch)
  int32_t* toff;         // T+1 first tour step
};

// Shared-memory layout of the sweep for a rank-table window of `ww` words.
struct SweepLayout {
  int32_t ww;
  int32_t nch32, nch64;
  uint32_t cap32, cap64;
  size_t off_rl, off_fine, off_T, off_P, off_ring, off_pdesc, off_epre, off_qpre, off_ev, off_emeta, off_q, off_qmeta,
      off_corr, off_tiles, bytes;
};
template <typename Cfg>
__host__ __device__ inline SweepLayout sweep_layout(int32_t nwords, size_t budget) {
  SweepLayout L;
  L.ww = nwords < kWinWords ? nwords : kWinWords;
  auto al = [](size_t x) { return (x + 15) & ~size_t(15); };
  const size_t staging = sizeof(StepDesc) * (Cfg::kRing + Cfg::kRingFill) + 2 * 8 * (size_t)Cfg::kRing +
                         Cfg::kBufs * (size_t)Cfg::kTileEv * 16 + al(Cfg::kBufs * (size_t)Cfg::kTileEv) +
                         al(Cfg::kBufs * (size_t)Cfg::kTileQ * 12) + al(Cfg::kBufs * (size_t)Cfg::kTileQ) +
                         (size_t)kOfflineQ * 8 + 3 * 32;
  // per-warp copies of the chunk-total prefix: Fenwick chunks only (flat chunks
  // probe the chunk totals directly)
  const size_t pcopies = Cfg::kFlat ? 0 : (size_t)Cfg::kWarps * (kMaxChunks + 1) * 8;
  const size_t fixed = al((size_t)L.ww * 8) + al(((size_t)L.ww + 2) * 4) + staging + pcopies + 128;
  const size_t per32 = (size_t)kChunkStride * 4 + 8;  // int32 nodes + chunk total
  int32_t n32 = budget > fixed ? (int32_t)((budget - fixed) / per32) : 0;
  if (n32 > kMaxChunks) n32 = kMaxChunks;
  L.nch32 = n32;
  L.nch64 = (int32_t)(((size_t)n32 * kChunkStride * 4) / ((size_t)kChunkStride * 8));
  L.cap32 = (uint32_t)L.nch32 * kChunk;
  L.cap64 = (uint32_t)L.nch64 * kChunk;
  size_t o = al((size_t)L.ww * 8);
  L.off_rl = o;   o = al(o + ((size_t)L.ww + 2) * 4);
  L.off_fine = o; o = al(o + (size_t)n32 * kChunkStride * 4);
  L.off_T = o;    o = al(o + (size_t)n32 * 8);
  L.off_P = o;    o = al(o + pcopies);
  L.off_ring = o; o = al(o + sizeof(StepDesc) * Cfg::kRing);
  L.off_pdesc = o; o = al(o + sizeof(StepDesc) * Cfg::kRingFill);
  L.off_epre = o; o = al(o + 8 * (size_t)Cfg::kRing);
  L.off_qpre = o; o = al(o + 8 * (size_t)Cfg::kRing);
  L.off_ev = o;   o = al(o + Cfg::kBufs * (size_t)Cfg::kTileEv * 16);
  L.off_emeta = o; o = al(o + Cfg::kBufs * (size_t)Cfg::kTileEv);
  L.off_q = o;    o = al(o + Cfg::kBufs * (size_t)Cfg::kTileQ * 12);
  L.off_qmeta = o; o = al(o + Cfg::kBufs * (size_t)Cfg::kTileQ);
  L.off_corr = o; o = al(o + (size_t)kOfflineQ * 8);
  L.off_tiles = o; o = al(o + 3 * 32);
  L.bytes = o;
  return L;
}

// Window of the query-step sweep (bw_qsweep.cu): runs of 2,048 int32 ranks that fit beside a
// rank table of `ww` words, and the rank capacities the prepare pass cuts slices with.
struct QsLayout {
  int32_t ww = 0;
  uint32_t supers = 0, cap32 = 0, cap64 = 0;
  size_t bytes = 0;
};
QsLayout qsweep_layout(int32_t nwords);

// ------------------------------------------------------------------ host plan
// Tunable knobs of a pipeline (picked by the caller or the forest autotuner).
struct Tuning {
  int64_t block_work = 0;   // target work per state block (est_work units); 0 = auto
  int32_t ctas_per_sm = 0;  // persistent sweep CTAs per SM (1 or 2); 0 = auto
  int32_t slice_ranks = 0;  // cap on the ranks of one LUT slice (0 = all that fit shared memory)
  int32_t contract = -1;    // 1 / 0: contracted tour or not (-1: by the queries per state)
  int32_t tile = 0;         // sweep tile geometry: kTileNarrowId .. kTileEulerId, 0 = the default (finish_spec)
};

// Everything the enqueue needs that does not depend on the data.  Built on the
// host from the tree shapes (for one tree: from the scalar arguments).
struct PipeSpec {
  int32_t T = 1;
  int32_t S = 0;                // total states
  int64_t E = 0, Q = 0;
  uint32_t Cmax = 1;
  int32_t Smax = 1;             // largest tree (bounds the list-ranking rounds)
  int32_t B = 1;                // total blocks
  int64_t bits_words = 0;       // sum over blocks of bitmap words
  int64_t carry_words = 0;      // sum over trees of (nb - 1) * (C + 1)
  int64_t gsum_words = 0;       // sum over trees with > kCarryGroup rows of groups * (C + 1)
  int32_t n_units = 0;          // carry units
  bool group_pass = false;      // some tree has more than one row group
  int32_t ctas_per_sm = 2;
  int32_t tile = kTileNarrowId;
  int32_t sms = 0;
  SweepLayout SL{};
  QsLayout QL{};                // tile 7
  int32_t max_slices = kMaxSlices;   // slices a block may have
  bool chain_hint = false;
  bool contract = false;        // the tour runs over contracted nodes, without those no query needs
  // one-tree scalars (T == 1): tables are written by a kernel at each launch
  int32_t nb1 = 1;
  // forest host tables, uploaded once by bind (empty for the plain one-tree spec)
  std::vector<int32_t> h_soff, h_boff;
  std::vector<int64_t> h_eoff, h_qoff, h_bits, h_carry, h_gsum;
  std::vector<uint32_t> h_C;
  std::vector<CarryUnit> h_units;
  std::vector<int32_t> h_order;
};

struct Layout {
  size_t off[48];
  size_t total;
};

enum {
  W_TSOFF, W_TEOFF, W_TQOFF, W_TC, W_TBOFF, W_TBITS, W_TCARRY, W_TGSUM, W_LASTQ, W_UNITS, W_ORDER,
  W_MISC, W_EOFF, W_QOFF, W_GPAR, W_FORK, W_NEXT, W_CNT, W_EHEAD, W_XHEAD, W_RANKA, W_RANKB,
  W_STEPS, W_DESC, W_TIN, W_TOUT, W_WORK, W_SCAN, W_BLOCKS, W_BMODE, W_BITS, W_RLUT, W_SLICES,
  W_NSLICES, W_CARRY, W_GSUM, W_TNOFF, W_TTOFF, W_NEOFF, W_NQOFF, W_NPAR, W_COUNT
};

// misc words
enum { M_STATUS = 0, M_PREP_TICKET = 1, M_SWEEP_TICKET = 2, M_CHAIN = 3, M_PREPB_TICKET = 4, M_NODES = 5, M_STEPS = 6,
       M_HOT = 7, M_HOT_TICKET = 8,
       M_ROUNDS = 32 };  // 64 words

// Stage timing events of one launch: stage i runs from ev[i] to ev[i + 1]; a chain
// launch (chain = 1) records the sweep from ev[BW_STAGE_SWEEP] to ev[BW_STAGE_SWEEP+1]
// and the carry that follows it up to ev[BW_STAGE_COUNT + 1].
struct EventSet {
  cudaEvent_t ev[BW_STAGE_COUNT + 2];
  int chain = 0;
};

// Build the spec of a forest (tree shapes on the host).  Returns 0 or BW_EINVAL.
int pipe_spec_forest(int32_t T, const int64_t* soff, const int64_t* eoff, const int64_t* qoff,
                     const uint32_t* C, const Tuning& tune, int sms, PipeSpec& spec);
// Spec of one tree (the plain replay).
int pipe_spec_one(int32_t S, uint32_t C, int64_t E, int64_t Q, int32_t blocks, bool chain, const Tuning& tune,
                  int sms, PipeSpec& spec, int64_t min_work = kMinWork);
void pipe_layout(const PipeSpec& spec, Layout& L);
// Upload the forest tables into the workspace (no-op for one tree).  Synchronous.
int pipe_bind(const PipeSpec& spec, void* workspace, cudaStream_t st);
// Enqueue the whole pipeline (kernels and memsets only: capturable in a CUDA graph).
int pipe_enqueue(const PipeSpec& spec, void* workspace, const int32_t* parent, const BwEvent* events,
                 const BwQuery* queries, int64_t* answers, cudaStream_t st, EventSet* timing, int* kernels);
// Arrays of the ingest and linearise stages; `rank` holds (next, distance to the end of
// the tour) per segment once pipe_tour's kernels have run.
struct TourArrays {
  TreeTabs tt;
  int32_t* misc;
  int64_t *eoff, *qoff;      // S + 1 each
  int32_t* gpar;             // forests: global parents (one tree: NULL)
  int32_t *fork_head, *next_sib;
  int64_t* cnt;
  int32_t *ehead, *xhead;
  uint64_t* rank;            // 2 S
  int64_t* scan_tmp;
  // contracted tours: event and query offsets and parents of the nodes; S words of scratch
  // for the node numbers and S bytes for the fork marks
  int64_t *neoff, *nqoff;
  int32_t* npar;
  uint32_t* ends;
  uint8_t* forked;
};
int pipe_tour(const PipeSpec& spec, bool forest, const TourArrays& w, const int32_t* parent, const BwEvent* events,
              const BwQuery* queries, cudaStream_t st, EventSet* timing, int& kernels);

// Euler-tile sweep (bw_esweep.cu): the inputs of k_sweep, the rank capacities the
// prepare pass cut the slices with, events as 16-byte records (16-byte aligned).
struct EsParams {
  const uint4* ev;
  const BwQuery* qs;
  const StepDesc* desc;
  const BlockTab* blocks;
  const int32_t* order;   // queue order (NULL: identity)
  int32_t B;
  uint32_t cap32, cap64;
  const uint64_t* bits;
  const uint32_t* rlut;
  const Slice* slices;    // max_slices a block
  int32_t max_slices;
  const int32_t* nslices;
  const int64_t* carry;
  int64_t* answers;
  int32_t* status;
  const int32_t* bmode;   // kMode32 | kModeHot
  int32_t* ticket;
  int32_t* hot;           // Euler tiles: whether there is a second kernel's work, and its ticket (NULL: all in one)
};
int esweep_attrs();   // one-time shared-memory opt-in (cudaError_t as int)
int esweep_launch(const EsParams& p, int grid, cudaStream_t st);
int qsweep_attrs();
int qsweep_launch(const EsParams& p, const QsLayout& q, int grid, cudaStream_t st);

// Device address of the status word inside a workspace laid out for `spec`.
const int32_t* pipe_status_word(const PipeSpec& spec, const void* workspace);
int report(cudaError_t e, const char* what);

}  // namespace bw
