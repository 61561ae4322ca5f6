// Hand-written sm_100a kernel for fused graphs WITH a reduce-by-row: persistent CTAs walk merge-path tiles, a
// contiguous run each, or (whole rows, below) short runs in turn; each tile's row-end offsets, index arrays and
// (two-phase graphs) per-edge tensors are staged into shared memory by 1-D bulk async copies (TMA, mbarrier
// complete_tx) that a producer warp issues STAGES tiles ahead.
//   Two-phase graphs (plain SpMV and every graph whose map needs no per-row data): phase 1, lanes on
//   consecutive edges -- each thread copies IPT edges from the stage to registers, hands the stage back,
//   gathers, runs the generated map and writes the products to shared memory; phase 2, one thread per
//   row sums its products and stores the row; rows longer than kShortRowMax are summed by whole warps.
//   Row-mode graphs (a selector equals the row id: spring-mass, fluxes): in tiles without long rows one
//   thread per row loads the row's own record once, gathers and maps its edges in register batches and
//   stores the row; in tiles with a long row whole warps take the rows one at a time (lanes 32 edges
//   apart, shuffle tree).  Nothing of a row-mode graph passes through a shared-memory product buffer.
//   Whole rows (either kind of graph, when the plan found a matrix of short rows whose tiles can all hold whole rows, and
//   that one lane per row suits): no carries at all, so no barriers either -- every warp takes 32 rows of a staged tile, one per lane,
//   and keeps everything in registers.  The other two loops run on such tiles too, without carries between CTAs.  No carry ties a
//   CTA to consecutive tiles either: where the gathered vectors are large, runs of kTileRun tiles go round the CTAs (kRounds); and a
//   small launch of short rows takes them without tiles and stages, a row per thread straight from global memory (kSmall).
// The carry of a row that spans tiles travels inside the CTA in shared memory; the only cross-CTA state
// is one carry per CTA, folded in by the last CTA to finish (ticket counter), in CTA order.  No atomics
// on the output, no pre-zeroed output, run-to-run deterministic.
//
// Replaces (reference, paths inside the FlexSpmv project): SpmvKernel
// include/merged_spmv_kernels.cuh:110-128 and AgentFlexSpmv::ConsumeTile / reduce<>
// cuda_template/reducer/merged_agent_spmv_template.cuh:180-445 (CUB BlockScan + per-row atomicAdd).
#pragma once
#include "flex_common.cuh"
#include "flex_tensor.cuh"
#include <type_traits>

namespace flex {

struct NoOwn {};       // what finish_row reads of a row itself in graphs without an epilogue

template <int BLOCK_, int IPT_, int STAGES_, int MIN_CTAS_, int BATCH_ = 8, bool PIPELINE_ = false, int ROW_BATCH_ = BATCH_>
struct TileCfg {
  // software pipelining across tiles (gathers of tile k in flight while tile k-1 is reduced); measured
  // slower than the plain loop on B200 (58% against 68% of the HBM peak on the 7-point fp64 SpMV: one
  // CTA less per SM for the second s_prod / s_rel buffer), so it is off by default
  static constexpr bool kPipeline = PIPELINE_;
  static constexpr int kBlock = BLOCK_;
  static constexpr int kIpt = IPT_;
  static constexpr int kStages = STAGES_;
  static constexpr int kMinCtas = MIN_CTAS_;
  static constexpr int kTile = BLOCK_ * IPT_;
  static constexpr int kWarps = BLOCK_ / 32;
  static constexpr int kBatch = BATCH_;   // edges of one row whose gathers are in flight together (short-row tiles)
  static constexpr int kRowBatch = ROW_BATCH_;   // the same in the loop over whole rows
  // consecutive tiles of a CTA where whole rows go round the CTAs (TileKernelArgs::rounds); large tiles go round one by one: 1024^2
  // shallow-water step (one model replayed) 333 us, in runs of two 336, of four 353; Rusanov 74.0, 76.6, 77.7
  static constexpr bool kLarge = kTile >= 2560;
  static constexpr int kTileRun = kLarge ? 1 : 4;
};

// Whether the plan may move all tile boundaries of the graph to row starts, and the kernel has the loop over whole rows, one
// row per lane: staged graphs that write nothing per edge (a thread that walks a row would store its edges' outputs a row
// length apart).
template <class G, class Cfg, bool WIN>
struct WholeRows {
  static constexpr bool value = !WIN && !G::kDirectLoads && !Cfg::kPipeline && !G::kStoresPerEdge;
};

constexpr int kMaxCtas = 2048;            // capacity of the per-CTA carry arrays in the workspace
#ifndef FLEX_SHORT_ROW_MAX
#define FLEX_SHORT_ROW_MAX 64
#endif
constexpr int kShortRowMax = FLEX_SHORT_ROW_MAX;              // tiles whose rows are all at most this long reduce one thread per row
constexpr uint64_t kWaitPolls = 1000000000ull;  // bound on every mbarrier wait: one second of %globaltimer

template <class G>
struct SmemTile {
  const char* base[G::kNumStreams > 0 ? G::kNumStreams : 1];
  __device__ __forceinline__ void advance(int records) {
    static_for<G::kNumStreams>([&](auto I) { base[I.value] += (size_t)records * G::template stream_bytes<I.value>(); });
  }
  template <int I, class T>
  __device__ __forceinline__ fx::Staged<T> stream(int le) const {
    return fx::Staged<T>{reinterpret_cast<const T*>(base[I] + (size_t)le * G::template stream_bytes<I>())};
  }
};

// Direct mode: the per-edge arrays are read straight from global memory with coalesced loads (lanes on
// consecutive edges); `le` is relative to the tile's first edge.
template <class G>
struct DirectTile {
  const typename G::Params* p;
  long long nz0;
  __device__ __forceinline__ void advance(int records) { nz0 += records; }
  template <int I, class T>
  __device__ __forceinline__ const T* stream(long long le) const {
    return reinterpret_cast<const T*>(G::template stream_ptr<I>(*p) + (size_t)(nz0 + le) * G::template stream_bytes<I>());
  }
};

// The per-edge arrays read straight from global memory through the read-only path; `e` counts from the array's front.
template <typename T>
struct LdgRef {
  const T* ptr;
  __device__ __forceinline__ T operator*() const { return __ldg(ptr); }
  __device__ __forceinline__ T operator[](int i) const { return __ldg(ptr + i); }
};
template <class G>
struct LdgTile {
  const typename G::Params* p;
  template <int I, class T>
  __device__ __forceinline__ LdgRef<T> stream(long long e) const {
    return LdgRef<T>{reinterpret_cast<const T*>(G::template stream_ptr<I>(*p) + (size_t)e * G::template stream_bytes<I>())};
  }
};

template <class G, bool WIN> struct WinBytesOf { static constexpr int value = 0; };
template <class G> struct WinBytesOf<G, true> { static constexpr int value = G::kWinBytes; };

template <class G, typename OffsetT, class Cfg, bool WIN = false>
struct TileSmemLayout {
  using V = typename G::V;
  static constexpr int kAcc = G::kAccDim;
  static constexpr int kBytesPerEdge = G::kStreamBytesPerEdge;
  static constexpr int kPerItem = (int(sizeof(OffsetT)) > kBytesPerEdge) ? int(sizeof(OffsetT)) : kBytesPerEdge;
  // a tile's records: kTile merge items, and the edges in front of its first row end when the plan moves the tile's
  // front boundary back to the start of that row (the gather-window variant may meet such a plan too)
  static constexpr bool kTilesMove = WholeRows<G, Cfg, false>::value;
  static constexpr int kRecordBytes = Cfg::kTile * kPerItem + (kTilesMove ? kWholeRowMax * kBytesPerEdge : 0);
  // each staged window may grow by < 32 bytes from aligning both ends to 16
  static constexpr int kStreamBytes =
      G::kDirectLoads ? 0 : int(align_up(uint64_t(kRecordBytes) + 32u * (G::kNumStreams + 1) + 16, 128));
  // gather windows (WIN): the segments of the gathered vector follow the streams in every stage
  static constexpr int kWinBytes = int(align_up(uint64_t(WinBytesOf<G, WIN>::value), 128));
  static constexpr int kStageBytes = kStreamBytes + kWinBytes;
  struct alignas(16) Ctl {   // read by every consumer thread of every tile: whole 16-byte words (see acquire)
    long long row0, nz0;
    int nrows, nnz;
    int win;            // the tile gathers from the window area and its index stream holds 16-bit positions
    uint32_t roff_off;
    uint32_t stream_off[G::kNumStreams > 0 ? G::kNumStreams : 1];
  };
  // Offsets with `stages` barriers and control blocks.  The shared memory a kernel does not claim stays L1 cache, and the
  // number of gather misses an SM can have in flight grows with that cache (measured on B200: 63 / 130 / 183 / 225 / 265 G
  // random 4-byte gathers per second at 228 / 196 / 164 / 132 / <= 32 KB of shared memory per SM).  The steps are coarse: with
  // 4 CTAs an SM, 128 bytes more than 49152 take the next one (ops_zoo in fp64: 208 -> 214 us), so nothing is reserved here
  // that the graph's loops do not use.
  static constexpr int off_ctl(int stages) { return int(align_up(16 * stages, 16)); }
  static constexpr int off_xs(int stages) { return int(align_up(off_ctl(stages) + sizeof(Ctl) * stages, 16)); }
  static constexpr int off_wkey(int stages) { return int(align_up(off_xs(stages) + 4 * (Cfg::kBlock + 1), 16)); }
  static constexpr int off_wval(int stages) { return int(align_up(off_wkey(stages) + 4 * Cfg::kWarps, 16)); }
  static constexpr int off_carry(int stages) { return int(align_up(off_wval(stages) + sizeof(V) * kAcc * Cfg::kWarps, 16)); }
  static constexpr int off_flag(int stages) { return int(align_up(off_carry(stages) + sizeof(V) * kAcc * 2, 16)); }
  // rows longer than kShortRowMax inside the current tile: [0..1] counters by tile parity, [2..] local rows
  static constexpr int kMaxLong = Cfg::kTile / (kShortRowMax + 1) + 2;
  static constexpr int off_long(int stages) { return int(align_up(off_flag(stages) + 16, 16)); }
  static constexpr int kBuffers = (!G::kGatherNeedsRow && Cfg::kPipeline) ? 2 : 1;   // s_rel / s_prod / long-row list double-buffered when tiles are pipelined
  static constexpr int off_rel(int stages) { return int(align_up(off_long(stages) + 4 * (4 + kMaxLong * kBuffers), 16)); }
  // Row-mode graphs (a selector equals the row id) reduce in registers in every tile: no product buffer.
  static constexpr int off_prod(int stages) { return int(align_up(off_rel(stages) + 4 * (Cfg::kTile + 1) * kBuffers, 16)); }
  static constexpr int off_stages(int stages) {
    return int(align_up(off_prod(stages) + (G::kGatherNeedsRow ? 0 : sizeof(V) * kAcc * Cfg::kTile * kBuffers), 128));
  }
  static constexpr int two_phase(int stages) { return off_stages(stages) + kStageBytes * Cfg::kStages; }
  // The loop over whole rows needs neither row ends nor products in shared memory: its stages begin where those would,
  // and as many fit as the other loop's total allows, one more where that costs at most 2 KB.
  static constexpr bool kWhole = WholeRows<G, Cfg, WIN>::value;
  static constexpr int off_row_stages(int stages) { return int(align_up(off_long(stages), 128)); }
  static constexpr bool kMore = G::kGatherNeedsRow || G::kLightMap;      // (maps that divide run this loop on the shortest rows only)
  static constexpr int row_stages() {
    int n = kWhole ? Cfg::kStages : 0;
    while (kWhole && kMore && n < 4 && off_row_stages(n + 1) + kStageBytes * (n + 1) <= two_phase(n + 1) + 2048) ++n;
    return n;
  }
  static constexpr int kRowStages = row_stages();
  static constexpr int kMaxStages = kRowStages > Cfg::kStages ? kRowStages : Cfg::kStages;
  static constexpr int kOffBars = 0;
  static constexpr int kOffCtl = off_ctl(kMaxStages), kOffXs = off_xs(kMaxStages), kOffWKey = off_wkey(kMaxStages);
  static constexpr int kOffWVal = off_wval(kMaxStages), kOffCarry = off_carry(kMaxStages), kOffFlag = off_flag(kMaxStages);
  static constexpr int kOffLong = off_long(kMaxStages), kOffRel = off_rel(kMaxStages), kOffProd = off_prod(kMaxStages);
  static constexpr int kOffStages = off_stages(kMaxStages), kOffRowStages = off_row_stages(kMaxStages);
  static constexpr int kTwoPhase = two_phase(kMaxStages);
  static constexpr int kRowLoop = kOffRowStages + kStageBytes * kRowStages;
  static constexpr int kTotal = (kWhole && kRowLoop > kTwoPhase) ? kRowLoop : kTwoPhase;
};

struct TileKernelArgs {
  const void* row_offsets;  // leading 0 included
  const void* coords;       // (num_tiles + 1) pairs of OffsetT
  WorkspaceHeader* header;
  long long* carry_row;     // [kMaxCtas]
  void* carry_val;          // [kMaxCtas][kAcc] of V
  long long num_rows;
  long long num_edges;
  long long num_tiles;
  int rounds;               // kRounds: how often every CTA takes kTileRun tiles in turn before the rest is split
  const int* win_table;                // gather windows (WIN kernels): per-tile segment table,
  const unsigned short* win_index;     // per-edge positions inside the window area,
  long long num_vertices;              // rows of the gathered array
};

// One staged window: `count` elements of `eb` bytes starting at element `first` of an array of
// `total` elements at `gbase` (16-byte aligned).  The bulk copy covers whole 16-byte chunks that lie
// inside the array; a ragged tail (the array's last < 16 bytes) is fetched with plain loads.
struct Window {
  const char* src;     // 16-byte aligned start of the bulk part
  uint32_t bulk_bytes; // multiple of 16 (may be 0)
  uint32_t lead;       // bytes between src and the first wanted element
  uint32_t span;       // smem bytes reserved (multiple of 16)
  const char* tail_src;
  uint32_t tail_bytes; // multiple of the element size
};
__device__ __forceinline__ Window make_window(const void* gbase, uint32_t eb, long long first, long long count,
                                              long long total) {
  Window w;
  const uintptr_t addr0 = (uintptr_t)gbase + (uintptr_t)first * eb;
  const uintptr_t addr1 = addr0 + (uintptr_t)count * eb;
  const uintptr_t a0 = addr0 & ~(uintptr_t)15;
  const uintptr_t a1 = (addr1 + 15) & ~(uintptr_t)15;
  const uintptr_t arr_floor = ((uintptr_t)gbase + (uintptr_t)total * eb) & ~(uintptr_t)15;
  uintptr_t bulk_end = a1 < arr_floor ? a1 : arr_floor;
  if (bulk_end < a0) bulk_end = a0;
  w.src = (const char*)a0;
  w.lead = (uint32_t)(addr0 - a0);
  w.span = count > 0 ? (uint32_t)(a1 - a0) : 0u;
  w.bulk_bytes = count > 0 ? (uint32_t)(bulk_end - a0) : 0u;
  const uintptr_t t0 = bulk_end > addr0 ? bulk_end : addr0;
  w.tail_src = (const char*)t0;
  w.tail_bytes = (count > 0 && addr1 > t0) ? (uint32_t)(addr1 - t0) : 0u;
  return w;
}

// Instantiations of the kernel, picked by the size of a launch (GraphApi::launch_tiles).  They differ in what they do with a plan of
// whole rows; other plans run the same loops in all of them.  One kernel for all three costs the plain one 2 % (145^3 fp32 42.3
// -> 43.1 us, spring-mass 500^2 fp64 20.7 -> 21.1).
constexpr int kPlain = 0;
constexpr int kSmall = 1;       // few tiles a CTA: whole rows are read straight from global memory
constexpr int kRounds = 2;      // tiles of whole rows go round the CTAs

template <class G, typename OffsetT, class Cfg, bool WIN = false, int MODE = kPlain>
__global__ void __launch_bounds__(Cfg::kBlock + (G::kDirectLoads ? 0 : 32), Cfg::kMinCtas)
flex_tile_kernel(const typename G::Params p, const TileKernelArgs a) {
  using V = typename G::V;
  using L = TileSmemLayout<G, OffsetT, Cfg, WIN>;
  static_assert(!WIN || (!G::kDirectLoads && !G::kGatherNeedsRow && !Cfg::kPipeline), "gather windows: staged two-phase loop only");
  using Ctl = typename L::Ctl;
  constexpr int kAcc = G::kAccDim;
  constexpr int NS = G::kNumStreams;
  constexpr int BLOCK = Cfg::kBlock, IPT = Cfg::kIpt, S = Cfg::kStages;
  constexpr bool DIRECT = G::kDirectLoads;   // narrow per-edge records: coalesced loads, no staging, no producer warp

  extern __shared__ __align__(128) unsigned char smem[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::kOffBars);    // "full": a stage's copies have landed
  uint64_t* empty = bars + L::kMaxStages;                              // "empty": the consumers released a stage
  Ctl* ctls = reinterpret_cast<Ctl*>(smem + L::kOffCtl);
  int* s_wkey = reinterpret_cast<int*>(smem + L::kOffWKey);
  V* s_wval = reinterpret_cast<V*>(smem + L::kOffWVal);
  V* s_carry = reinterpret_cast<V*>(smem + L::kOffCarry);
  int* s_flag = reinterpret_cast<int*>(smem + L::kOffFlag);
  int* s_nlong = reinterpret_cast<int*>(smem + L::kOffLong);
  int* s_long = s_nlong + 4;
  int* s_rel = reinterpret_cast<int*>(smem + L::kOffRel);
  V* s_prod = reinterpret_cast<V*>(smem + L::kOffProd);
  unsigned char* s_stage = smem + L::kOffStages;
  constexpr bool WHOLE = L::kWhole;

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const OffsetT* row_offsets = static_cast<const OffsetT*>(a.row_offsets);
  const OffsetT* coords = static_cast<const OffsetT*>(a.coords);

  // With a programmatic dependent launch the CTA may have been placed while the kernel before this one on the stream
  // was still draining: wait for its results (and for this workspace's ticket) before the first global access.
  pdl_wait();
  pdl_launch_dependents();

  // contiguous run of tiles of this CTA
  const long long q = a.num_tiles / gridDim.x, rem = a.num_tiles % gridDim.x;
  const long long t_begin = (long long)blockIdx.x * q + ((long long)blockIdx.x < rem ? blockIdx.x : rem);
  const int count = (int)(q + ((long long)blockIdx.x < rem ? 1 : 0));

  // Tile k of the CTA where whole rows go round the CTAs: no carry ties a CTA to consecutive tiles, so in each round it takes
  // kTileRun of them, and what is left behind the last full round is split like above (the same number of tiles a CTA).  The
  // CTAs then walk the matrix as one front.  In a run of its own a CTA meets the columns a plane (or a line) away at a time of its own,
  // unless a plane is a whole number of runs: the three places where a vector record is gathered lie up to half the matrix of traffic
  // apart.  DRAM reads of the 7-point fp64 SpMV, own runs / rounds: 360^3 (a plane is 1.64 runs) 5.45 / 4.71 GB, the vector's 0.37 GB three times / once;
  // 240^3 (2.47) 1.51 / 1.39, twice / once; 300^3 (1.97) 2.72 / 2.72, once in either.  There, and on 192^3 (0.72 / 0.71 GB, 129 / 122 us cold), the front
  // is the faster order at the same traffic: 592 CTAs read one stretch of each array, not 592.  us, own runs / rounds of 4, 8, 16, 32, 64 tiles:
  // 512^3 2529 / 2133, 2146, 2161, 2214, 2328; 300^3 480 / 422, 429, 434, 443, 464; 400^3 fp32 905 / 821, 827, 835, 839, 846; 5-point 3000^2 128 / 118, 122, 123,
  // 125, 126.
  constexpr int kTileRun = Cfg::kTileRun;
  auto round_tile = [&](int k) -> long long {
    if (k < a.rounds * kTileRun) return ((long long)(k / kTileRun) * gridDim.x + blockIdx.x) * kTileRun + k % kTileRun;
    return t_begin + (long long)a.rounds * kTileRun * (gridDim.x - 1 - blockIdx.x) + k;
  };

  // The producer warp asks for its first coordinates together with the header (two round trips become one).  The
  // words lie inside the workspace whether it was planned or not; nothing is done with them before the check below.
  OffsetT first_coords[4] = {0, 0, 0, 0}, first_of_round[4] = {0, 0, 0, 0};
  if constexpr (!DIRECT) {
    if (warp == Cfg::kWarps && count) {
#pragma unroll
      for (int i = 0; i < 4; ++i) first_coords[i] = coords[2 * t_begin + i];
      if constexpr (MODE == kRounds) {
#pragma unroll
        for (int i = 0; i < 4; ++i) first_of_round[i] = coords[2ll * kTileRun * blockIdx.x + i];
      }
    }
  }

  // So do the threads of a small launch with the ends of their first rows.
  OffsetT row_from = 0, row_to = 0;
  long long small_row = 0, small_end = 0;
  if constexpr (MODE == kSmall) {
    const long long share = rows_a_cta(a.num_rows, gridDim.x);
    small_row = blockIdx.x * share + tid;
    small_end = (blockIdx.x + 1) * share < a.num_rows ? (blockIdx.x + 1) * share : a.num_rows;
    // (the first row begins at edge 0 whatever row_offsets[0] says)
    if (small_row < small_end) { row_from = small_row ? row_offsets[small_row] : OffsetT(0); row_to = row_offsets[small_row + 1]; }
  }

  // All that the header says, requested before the first branch: one round trip.
  const uint32_t h_magic = a.header->magic;
  const int h_bits = a.header->offset_bits;
  const long long h_rows = a.header->num_rows, h_edges = a.header->num_edges, h_tiles = a.header->num_tiles;
  const int h_snapped = a.header->snapped_grid, h_whole = a.header->whole_rows, h_row_loop = a.header->row_loop;
  const bool h_stages = MODE == kSmall && a.header->uneven_shares != 0;
  // a workspace that was never planned for this problem holds no usable coordinates: every CTA
  // sees the same header, so all of them leave here and the ticket stays untouched
  if (h_magic != kMagic || h_tiles != a.num_tiles || h_rows != a.num_rows || h_edges != a.num_edges || h_bits != (int)(8 * sizeof(OffsetT))) {
    if (tid == 0 && blockIdx.x == 0) raise_not_planned(a.header);
    return;
  }
  // An epilogue needs a row's whole sum: a matrix that was not planned with whole rows is refused here, where every CTA
  // leaves before its producer warp has issued a copy (one still in flight would write into shared memory that a later CTA
  // owns).  So is a plan with moved boundaries (another graph's) where the stages have no room for them.
  if ((G::kEpilogue && h_whole != 1) || (!L::kTilesMove && !DIRECT && h_whole == 1)) {
    if (tid == 0 && blockIdx.x == 0) raise_status(a.header, FLEXSPMV_ERR_NOT_PLANNED);
    return;
  }
  // the loop over whole rows has its own stages, in its own places
  const bool whole = WHOLE && (G::kEpilogue || h_row_loop == 1);
  if constexpr (MODE == kSmall) {
    if (whole && !h_stages) {
      // ---- whole rows of a small launch: one row per thread, everything straight from global memory ----------------------
      // Bound by round trips: the row's ends (asked for with the header), then the edges and the gathers of every kRowBatch edges, so
      // 1 + 2 ceil(n / kRowBatch) of them for a row of n edges (5 for a 5-point row in fp64, 7 for a cell of three edges), without the barriers,
      // bulk copies and producer's coordinates in front of a stage, whose rows need one copy and ceil(n / kRowBatch) gathers.  Which
      // launches come here: GraphApi::small_launch.  Sums run left to right as in the loop below: the same bits.  512^2 5-point fp64 7.1 -> 5.1 us.
      LdgTile<G> tile{&p};
      constexpr int RB = Cfg::kRowBatch;
      for (; small_row < small_end; small_row += BLOCK + 32) {
        const long long e_from = (long long)row_from;
        const int n = (int)(row_to - row_from);
        if constexpr (G::kEpilogue) G::prefetch_row(p, small_row);
        V sum[kAcc];
#pragma unroll
        for (int j = 0; j < kAcc; ++j) sum[j] = V(0);
        typename G::GRow grow;
        if constexpr (G::kGatherNeedsRow) { if (n > 0) G::gather_row(p, small_row, grow); }
        for (int e0 = 0; e0 < n; e0 += RB) {
          typename G::EReg er[RB];
          typename G::GEdge ge[RB];
#pragma unroll
          for (int b = 0; b < RB; ++b)
            if (e0 + b < n) G::load_edge(p, tile, e_from + e0 + b, e_from + e0 + b, er[b]);
#pragma unroll
          for (int b = 0; b < RB; ++b)
            if (e0 + b < n) G::gather_edge(p, er[b], ge[b]);
#pragma unroll
          for (int b = 0; b < RB; ++b)
            if (e0 + b < n) G::map(p, er[b], e_from + e0 + b, grow, ge[b], sum);
        }
        if (small_row + BLOCK + 32 < small_end) { row_from = row_offsets[small_row + BLOCK + 32]; row_to = row_offsets[small_row + BLOCK + 33]; }
        typename G::GOwn own;
        G::load_own(p, small_row, own);
        G::finish_row(p, small_row, sum, own);
      }
      return;
    }
  }
  const int nstages = WHOLE ? (whole ? L::kRowStages : S) : S;
  unsigned char* const stage_base = (WHOLE && whole) ? smem + L::kOffRowStages : s_stage;

  const bool win_ready = WIN && a.header->win_ready == 1;   // until the window plan has run every tile gathers globally
  (void)win_ready;

  // ---- producer ------------------------------------------------------------------------------------------
  // Table entry of a tile's gather windows, one piece per lane: the segment count in every lane, segment j in
  // lane 16 + j (read one tile ahead, like the coordinates).
  struct WinEnt { int nseg, first, len; };
  auto load_win_entry = [&](long long tile_id) -> WinEnt {
    WinEnt e{0, 0, 0};
    if constexpr (WIN) {
      static_assert(NS + 1 <= 16 && kWinMaxSegs <= 16, "lanes 0..NS stage the streams, lanes 16.. the window segments");
      if (win_ready) {
        const int* ent = a.win_table + tile_id * kWinEntryInts;
        e.nseg = ent[0];
        if (lane >= 16 && lane - 16 < kWinMaxSegs) { e.first = ent[2 + 2 * (lane - 16)]; e.len = ent[3 + 2 * (lane - 16)]; }
      }
    }
    (void)tile_id;
    return e;
  };
  // Stages one tile; executed by the whole producer warp: lane i prepares window i (lane 0: row-end offsets,
  // lane 1+I: stream I, lane 16+j: gather-window segment j), a shuffle prefix sum places the windows in the
  // stage, lane 0 posts the byte count, then every lane issues its own bulk copy.
  auto issue = [&](long long row0, long long nz0, long long row1, long long nz1, int s, const WinEnt& we) {
    unsigned char* dst = stage_base + (size_t)s * L::kStageBytes;
    Window w;
    w.src = nullptr; w.bulk_bytes = 0; w.lead = 0; w.span = 0; w.tail_src = nullptr; w.tail_bytes = 0;
    const int nseg = we.nseg;
    if constexpr (WIN) {
      if (lane >= 16 && lane - 16 < nseg) w = make_window(G::gather_base(p), G::kGatherRecBytes, we.first, we.len, a.num_vertices);
    }
    if (lane == 0) w = make_window(row_offsets, sizeof(OffsetT), row0 + 1, row1 - row0, a.num_rows + 1);
    static_for<NS>([&](auto I) {
      if (lane == I.value + 1) {
        bool local = false;
        if constexpr (WIN) local = (I.value == G::kIdxStream) && nseg > 0;
        if (local) w = make_window(a.win_index, 2, nz0, nz1 - nz0, a.num_edges);
        else w = make_window(G::template stream_ptr<I.value>(p), G::template stream_bytes<I.value>(), nz0, nz1 - nz0, a.num_edges);
      }
    });
    uint32_t off = w.span;   // exclusive prefix sum of the spans over lanes 0..NS (streams) and 16.. (segments)
#pragma unroll
    for (int d = 1; d <= (WIN ? 8 : NS); d <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, off, d);
      if ((lane & 15) >= d) off += t;
    }
    off -= w.span;
    if constexpr (WIN) { if (lane >= 16) off += L::kStreamBytes; }
    uint32_t total = w.bulk_bytes;
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) total += __shfl_xor_sync(0xffffffffu, total, d);
    Ctl& c = ctls[s];
    if (lane == 0) { c.row0 = row0; c.nz0 = nz0; c.nrows = (int)(row1 - row0); c.nnz = (int)(nz1 - nz0); c.roff_off = off + w.lead; c.win = nseg > 0; }
    static_for<NS>([&](auto I) { if (lane == I.value + 1) c.stream_off[I.value] = off + w.lead; });
    // the ragged tail (last < 16 bytes of an array) is fetched with plain loads BEFORE the arrive below,
    // whose release (after the warp barrier) makes it and the control block visible to the consumers
    if (w.tail_bytes) {
      const uint32_t so = off + (uint32_t)(w.tail_src - w.src);
      if (((uint32_t)reinterpret_cast<uintptr_t>(w.tail_src) | w.tail_bytes) & 3u) {   // 2-byte elements (window positions)
        for (uint32_t b = 0; b < w.tail_bytes; b += 2)
          *reinterpret_cast<uint16_t*>(dst + so + b) = *reinterpret_cast<const uint16_t*>(w.tail_src + b);
      } else {
        for (uint32_t b = 0; b < w.tail_bytes; b += 4)
          *reinterpret_cast<uint32_t*>(dst + so + b) = *reinterpret_cast<const uint32_t*>(w.tail_src + b);
      }
    }
    fence_proxy_async_smem();   // earlier generic accesses to this stage are ordered before the bulk copies
    __syncwarp();
    if (lane == 0) mbar_expect_tx(&bars[s], total);
    __syncwarp();
    if (w.bulk_bytes) bulk_g2s(dst + off, w.src, w.bulk_bytes, &bars[s]);
    // what an epilogue reads per row comes from L2 then, not from DRAM, when the tile's rows get there
    if constexpr (G::kEpilogue) G::prefetch_rows(p, row0, row1, lane);
#ifdef FLEX_PREFETCH_DIRECT
    if constexpr (G::kHasDirectEdgeTensors) G::prefetch_direct(p, nz0, nz1, lane);
#endif
  };

  if constexpr (!DIRECT) {
    if (tid == 0) {
#pragma unroll
      for (int s = 0; s < L::kMaxStages; ++s) { mbar_init(&bars[s], 1); mbar_init(&empty[s], Cfg::kWarps); }   // empty: one arrive per consumer warp
      mbar_fence_init();
    }
  }
  if (tid < 2 * kAcc) s_carry[tid] = V(0);
  if (tid < 4) s_nlong[tid] = 0;
  // no row spans two CTAs of this launch
  if (tid == 0) s_flag[1] = (h_whole == 1 || h_snapped == (int)gridDim.x) ? 1 : 0;
  __syncthreads();   // the only barrier that includes the producer warp

  // ---- producer warp: runs up to S tiles ahead of the consumers, off their critical path -----------
  if (!DIRECT && warp == Cfg::kWarps) {
    {
      int issued = 0;
      bool pfail = false;
      // coordinates are read one tile ahead, so their load latency overlaps the wait for a free stage
      long long c_row = (long long)first_coords[0], c_nz = (long long)first_coords[1];
      long long n_row = (long long)first_coords[2], n_nz = (long long)first_coords[3];
      long long t = 0;            // kRounds: tile k, and the tiles until the CTA's next one is not the one behind
      int run = 0x7fffffff;
      if constexpr (MODE == kRounds) t = t_begin;
      if (MODE == kRounds && whole) {
        c_row = (long long)first_of_round[0]; c_nz = (long long)first_of_round[1];
        n_row = (long long)first_of_round[2]; n_nz = (long long)first_of_round[3];
        t = (long long)kTileRun * blockIdx.x;
        run = kTileRun;
      }
      WinEnt c_we = count ? load_win_entry(t_begin) : WinEnt{0, 0, 0};
      // testing aid (flexspmv_debug_withhold_stage): the stage of tile `withhold - 1` and of every later tile is
      // never filled, so that the consumers' bounded wait runs out and the error path can be exercised
      const unsigned long long withhold = a.header->debug[7];
      int s = 0;                  // stage of tile k; round: how often the stages have been filled before
      uint32_t round = 0;
      for (int k = 0; k < count; ++k) {
        if (withhold && (unsigned long long)(MODE == kRounds ? t : t_begin + k) + 1ull >= withhold) break;
        long long nn_row = 0, nn_nz = 0;
        [[maybe_unused]] long long nf_row = 0, nf_nz = 0;      // kRounds: front of the next tile
        if constexpr (MODE == kRounds) {
          nf_row = n_row; nf_nz = n_nz;
          ++t;
          if (k + 1 < count) {
            if (--run == 0) {
              t = round_tile(k + 1);
              run = k + 1 < a.rounds * kTileRun ? kTileRun : 0x7fffffff;
              nf_row = (long long)coords[2 * t]; nf_nz = (long long)coords[2 * t + 1];
            }
            nn_row = (long long)coords[2 * t + 2]; nn_nz = (long long)coords[2 * t + 3];
          }
        } else {
          if (k + 1 < count) { nn_row = (long long)coords[2 * (t_begin + k + 2)]; nn_nz = (long long)coords[2 * (t_begin + k + 2) + 1]; }
        }
        const WinEnt n_we = (k + 1 < count) ? load_win_entry(t_begin + k + 1) : WinEnt{0, 0, 0};
        if (round > 0) {
          const bool ok = mbar_wait_bounded(&empty[s], (round - 1) & 1u, kWaitPolls);
          if (!__all_sync(0xffffffffu, ok)) { pfail = true; break; }
        }
        issue(c_row, c_nz, n_row, n_nz, s, c_we);
        if constexpr (MODE == kRounds) { c_row = nf_row; c_nz = nf_nz; }
        else { c_row = n_row; c_nz = n_nz; }
        n_row = nn_row; n_nz = nn_nz; c_we = n_we;
        issued = k + 1;
        if (++s == nstages) { s = 0; ++round; }
      }
      if (pfail && lane == 0) {   // the consumers never released a stage: flag it, let copies in flight land, leave
        raise_status(a.header, FLEXSPMV_ERR_TIMEOUT);
        a.header->debug[4] = (uint32_t)issued; a.header->debug[5] = blockIdx.x;
        for (int j = issued > nstages ? issued - nstages : 0; j < issued; ++j)
          mbar_wait_bounded(&bars[j % nstages], (uint32_t)(j / nstages) & 1u, kWaitPolls);
      }
    }
    return;
  }

  // ---- consumers (threads 0 .. BLOCK-1); their barriers are the named barrier 1 ---------------------
  using TileT = std::conditional_t<DIRECT, DirectTile<G>, SmemTile<G>>;
  struct TileRef { long long row0, nz0; int nrows, nnz; int win; };
  const unsigned char* xwin = nullptr;   // WIN: the current tile's window area
  bool failed = false;
  long long last_row1 = 0;

  // direct mode: tile coordinates are read one tile ahead into registers
  long long d_row = 0, d_nz = 0, d_row1 = 0, d_nz1 = 0;
  if constexpr (DIRECT) {
    if (count) {
      d_row = (long long)coords[2 * t_begin]; d_nz = (long long)coords[2 * t_begin + 1];
      d_row1 = (long long)coords[2 * t_begin + 2]; d_nz1 = (long long)coords[2 * t_begin + 3];
    }
  }

  // Makes tile k available: waits (bounded) for its stage, or takes its coordinates in direct mode.
  auto acquire = [&](int k, TileRef& t, TileT& tile, const OffsetT*& rend) -> bool {
    if constexpr (DIRECT) {
      t.row0 = d_row; t.nz0 = d_nz; t.nrows = (int)(d_row1 - d_row); t.nnz = (int)(d_nz1 - d_nz); t.win = 0;
      d_row = d_row1; d_nz = d_nz1;
      if (k + 1 < count) { d_row1 = (long long)coords[2 * (t_begin + k + 2)]; d_nz1 = (long long)coords[2 * (t_begin + k + 2) + 1]; }
      tile.p = &p; tile.nz0 = t.nz0;
      rend = row_offsets + t.row0 + 1;
      named_bar_sync(1, BLOCK);   // the previous tile's readers of the shared arrays are done
      return true;
    } else {
      const int s = k % S;
      const bool ok = named_bar_and(1, BLOCK, mbar_wait_bounded(&bars[s], (uint32_t)(k / S) & 1u, kWaitPolls));
      if (!ok) {
        if (tid == 0) {
          raise_status(a.header, FLEXSPMV_ERR_TIMEOUT);
          a.header->debug[0] = (uint32_t)(t_begin + k); a.header->debug[1] = (uint32_t)s; a.header->debug[2] = blockIdx.x;
        }
        return false;
      }
      // one 16-byte shared load per 16 bytes of the control block instead of one load per field: the kernel
      // is bound by shared-memory wavefronts, and every thread of every tile reads this
      Ctl c;
      {
        constexpr int kWords = int(sizeof(Ctl) / 16);
        const int4* src = reinterpret_cast<const int4*>(&ctls[s]);
        int4* dst16 = reinterpret_cast<int4*>(&c);
#pragma unroll
        for (int i = 0; i < kWords; ++i) dst16[i] = src[i];
      }
      t.row0 = c.row0; t.nz0 = c.nz0; t.nrows = c.nrows; t.nnz = c.nnz; t.win = c.win;
      const unsigned char* stage = s_stage + (size_t)s * L::kStageBytes;
      xwin = stage + L::kStreamBytes;
      rend = reinterpret_cast<const OffsetT*>(stage + c.roff_off);
      static_for<NS>([&](auto I) { tile.base[I.value] = reinterpret_cast<const char*>(stage + c.stream_off[I.value]); });
      return true;
    }
  };
  // This warp needs nothing more from stage s: the producer refills it once every warp has said so.
  auto release = [&](int k) {
    if constexpr (!DIRECT) {
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty[k % S]);
    }
  };
  // Row ends as 32-bit edge indices relative to the tile, with a sentinel behind the last row.  Returns
  // whether this thread saw a long row (or a long trailing partial row).
  // With list >= 0 the long rows are also appended (in any order) to buffer lbuf of s_long, counted in
  // s_nlong[list].
  auto convert = [&](const TileRef& t, const OffsetT* rend, int* srel, int list, int lbuf = 0) -> bool {
    int* rows_long = s_long + lbuf * L::kMaxLong;
    bool my_long = false;
    for (int r = tid; r < t.nrows; r += BLOCK) {
      const long long end_r = (long long)rend[r];
      const long long beg_r = r ? (long long)rend[r - 1] : t.nz0;
      srel[r] = (int)(end_r - t.nz0);
      if ((end_r - beg_r) > kShortRowMax) {
        my_long = true;
        if (list >= 0) rows_long[atomicAdd(&s_nlong[list], 1)] = r;
      }
    }
    if (tid == 0) {
      srel[t.nrows] = 0x7fffffff;
      const long long beg_t = t.nrows ? (long long)rend[t.nrows - 1] : t.nz0;
      if ((t.nz0 + t.nnz - beg_t) > kShortRowMax) {
        my_long = true;
        if (list >= 0) rows_long[atomicAdd(&s_nlong[list], 1)] = t.nrows;
      }
    }
    return my_long;
  };
  auto store_row = [&](long long row, const V* v) {
    static_for<G::kNumReducers>([&](auto R) {
      constexpr int d = G::template red_dim<R.value>();
      constexpr int o = G::template red_off<R.value>();
      V* dst = G::template red_out<R.value>(p) + (size_t)row * d;
#pragma unroll
      for (int j = 0; j < d; ++j) dst[j] = v[o + j];
    });
  };

  if constexpr (WHOLE) {
    if (whole) {
      // ---- tiles of whole, short rows: warps work alone, no barrier, no carry, no products in shared memory ----------
      // A warp takes 32 rows of a tile, one per lane: it reads the rows' column indices from the stage, has the gathers
      // of kRowBatch edges per row in flight together -- lane r and lane r + 1 gather neighbours on a stencil, so a warp
      // gather touches 2-3 cache lines instead of the 8-9 of 32 consecutive edges -- and reads the values only when the
      // gathers are back.  Groups of rows go round the warps across tiles (`turn`), so a tile need not hold a multiple of
      // the CTA's rows.  Sums run left to right over the row, as in the two-phase loop.
      // What the two-phase loop is bound by on short rows is the shared-memory / L1 data pipe (75 - 80 % busy at 55 % of
      // DRAM) and two CTA barriers a tile; this one moves no product through shared memory and a third of the gather lines
      // (41 % of the pipe at 70 % of DRAM), and is bound by the latency of the gathers at the registers of 4 CTAs per SM: 10 of
      // 16 stall cycles per issue are long_scoreboard (row-mode graphs, and longer rows in large launches: GraphApi::use_big).  us a launch, two-phase / this loop with a run of tiles a CTA: 7-point fp64
      // SpMV 512^3 3205 / 2564 (in rounds 2133); 145^3 fp32 54.1 / 42.6; 5-point 512^2 fp64 9.1 / 7.1 (without stages 5.1); 27 columns a row
      // fp64, 300 007 rows 26.2 / 23.9; spring-mass 1024^2 fp32 44.5 / 38.4; Rusanov 1024^2 fp64 92 / 83.5.
      constexpr int RB = Cfg::kRowBatch;
      constexpr bool GROUPS = G::kGroup > 1 && Cfg::kLarge;
      [[maybe_unused]] bool groups_wide = false;
      if constexpr (GROUPS) groups_wide = G::groups_aligned(p);
      int s = 0, turn = 0;
      uint32_t parity = 0;
      for (int k = 0; k < count; ++k) {
        const bool ok = mbar_wait_bounded(&bars[s], parity, kWaitPolls);
        if (!__all_sync(0xffffffffu, ok)) {
          if (lane == 0) {
            raise_status(a.header, FLEXSPMV_ERR_TIMEOUT);
            a.header->debug[0] = (uint32_t)(MODE == kRounds ? round_tile(k) : t_begin + k); a.header->debug[1] = (uint32_t)s; a.header->debug[2] = blockIdx.x;
          }
          return;
        }
        Ctl c;
        {
          const int4* src = reinterpret_cast<const int4*>(&ctls[s]);
          int4* dst16 = reinterpret_cast<int4*>(&c);
#pragma unroll
          for (int i = 0; i < int(sizeof(Ctl) / 16); ++i) dst16[i] = src[i];
        }
        const unsigned char* stage = smem + L::kOffRowStages + (size_t)s * L::kStageBytes;
        const OffsetT* rend = reinterpret_cast<const OffsetT*>(stage + c.roff_off);
        SmemTile<G> tile;
        static_for<NS>([&](auto I) { tile.base[I.value] = reinterpret_cast<const char*>(stage + c.stream_off[I.value]); });
        const int groups = (c.nrows + 31) >> 5;
        int g = warp - turn;
        if (g < 0) g += Cfg::kWarps;
        if (g >= groups) {                                         // no rows for this warp
          __syncwarp();
          if (lane == 0) mbar_arrive(&empty[s]);
        }
        for (; g < groups; g += Cfg::kWarps) {
          const int r = (g << 5) + lane;
          int lo = 0, hi = 0;
          if (r < c.nrows) {
            // unsigned: the ends may lie on either side of edge 2^31, and the difference is right modulo 2^32
            hi = (int)((unsigned)rend[r] - (unsigned)c.nz0);
            if (r) lo = (int)((unsigned)rend[r - 1] - (unsigned)c.nz0);
          }
          V sum[kAcc];
#pragma unroll
          for (int j = 0; j < kAcc; ++j) sum[j] = V(0);
          typename G::GRow grow;
          if constexpr (G::kGatherNeedsRow) { if (lo < hi) G::gather_row(p, c.row0 + r, grow); }
          if constexpr (GROUPS) {
            // Four edges' records a word of every array, from a multiple of four on: lanes a row of eight edges apart meet in four banks with
            // single indices (8-way), and read a line each for every edge tensor.  Lattices fp32 600^2 15.3 -> 14.8 us, 1024^2 36.4 -> 35.9, 1500^2 70.6 -> 65.9.  In the
            // smaller configuration, where four edges more in registers spill, no gain: 38.3 -> 38.4, 430^2 9.8 -> 10.0; neither for pairs
            // of 8-byte values, 600^2 26.1 -> 28.5.
            constexpr int N = G::kGroup;
            const int lead = (int)((unsigned)c.nz0 % (unsigned)N);
            for (int e0 = lo - (lo + lead) % N; e0 < hi; e0 += N) {
              typename G::EReg er[N];
              typename G::GEdge ge[N];
              G::load_group(p, tile, e0, c.nz0 + e0, a.num_edges, groups_wide && c.nz0 + e0 + N <= a.num_edges, er);
#pragma unroll
              for (int b = 0; b < N; ++b)
                if (e0 + b >= lo && e0 + b < hi) G::gather_edge(p, er[b], ge[b]);
#pragma unroll
              for (int b = 0; b < N; ++b)
                if (e0 + b >= lo && e0 + b < hi) G::map(p, er[b], c.nz0 + e0 + b, grow, ge[b], sum);
            }
          } else
          for (int e0 = lo; e0 < hi; e0 += RB) {
            typename G::EReg er[RB];
            typename G::GEdge ge[RB];
#pragma unroll
            for (int b = 0; b < RB; ++b)
              if (e0 + b < hi) G::load_edge_idx(tile, e0 + b, er[b]);
#pragma unroll
            for (int b = 0; b < RB; ++b)
              if (e0 + b < hi) {
                if constexpr (!G::kValuesStaged) G::load_edge_vals(p, tile, e0 + b, c.nz0 + e0 + b, er[b]);
                G::gather_edge(p, er[b], ge[b]);
              }
#pragma unroll
            for (int b = 0; b < RB; ++b)
              if (e0 + b < hi) {
                if constexpr (G::kValuesStaged) G::load_edge_vals(p, tile, e0 + b, c.nz0 + e0 + b, er[b]);
                G::map(p, er[b], c.nz0 + e0 + b, grow, ge[b], sum);
              }
          }
          // the warp's last rows of this tile: nothing more is read from the stage
          if (g + Cfg::kWarps >= groups) {
            __syncwarp();
            if (lane == 0) mbar_arrive(&empty[s]);
          }
          if (r < c.nrows) {
            typename G::GOwn own;
            G::load_own(p, c.row0 + r, own);
            G::finish_row(p, c.row0 + r, sum, own);
          }
        }
        turn = (turn + groups) % Cfg::kWarps;
        if (++s == L::kRowStages) { s = 0; parity ^= 1u; }
      }
      return;
    }
  }

  if constexpr (G::kEpilogue) return;     // has the loop above only

  // ---- phase 1 pieces: lanes on consecutive edges ------------------------------------------------------
  auto map_load = [&](const TileRef& t, const TileT& tile, typename G::EReg (&er)[IPT]) {
    auto ttile = tile;
    ttile.advance(tid);   // element `tid` at offset 0: the unrolled accesses are base + constant
#pragma unroll
    for (int i = 0; i < IPT; ++i)
      if (i * BLOCK + tid < t.nnz) G::load_edge(p, ttile, i * BLOCK, t.nz0 + (i * BLOCK + tid), er[i]);
  };
  auto map_gather = [&](const TileRef& t, const typename G::EReg (&er)[IPT], typename G::GEdge (&ge)[IPT],
                        typename G::GRow (&gr)[G::kGatherNeedsRow ? IPT : 1]) {
#pragma unroll
    for (int i = 0; i < IPT; ++i) {
      if (i * BLOCK + tid < t.nnz) {
#ifndef FLEX_EXP_SKIP_GATHER
        G::gather_edge(p, er[i], ge[i]);
#else
        memset(&ge[i], 0, sizeof(ge[i]));
#endif
      }
    }
  };
  auto map_products = [&](const TileRef& t, const typename G::EReg (&er)[IPT], const typename G::GEdge (&ge)[IPT],
                          const typename G::GRow (&gr)[G::kGatherNeedsRow ? IPT : 1], V* sprod) {
    V* tprod = sprod + tid;
#pragma unroll
    for (int i = 0; i < IPT; ++i) {
      if (i * BLOCK + tid < t.nnz) {
        V prod[kAcc];
#pragma unroll
        for (int j = 0; j < kAcc; ++j) prod[j] = V(0);
        G::map(p, er[i], t.nz0 + (i * BLOCK + tid), gr[G::kGatherNeedsRow ? i : 0], ge[i], prod);
#pragma unroll
        for (int j = 0; j < kAcc; ++j) tprod[j * Cfg::kTile + i * BLOCK] = prod[j];
      }
    }
  };

  // ---- phase 1 of a tile with gather windows: 16-bit positions instead of column indices, gathers from the
  //      window area of the stage (so the stage goes back to the producer after the gathers, not before) ----
  auto map_load_gather_win = [&](const TileRef& t, const TileT& tile, typename G::EReg (&er)[IPT], typename G::GEdge (&ge)[IPT]) {
    if constexpr (WIN) {
      auto ttile = tile;
      ttile.advance(tid);
      unsigned short pos[IPT];
#pragma unroll
      for (int i = 0; i < IPT; ++i)
        if (i * BLOCK + tid < t.nnz) {
          G::load_edge_vals(p, ttile, i * BLOCK, t.nz0 + (i * BLOCK + tid), er[i]);   // the index stream holds 16-bit positions here
          pos[i] = reinterpret_cast<const unsigned short*>(tile.base[G::kIdxStream])[i * BLOCK + tid];
        }
#pragma unroll
      for (int i = 0; i < IPT; ++i)
        if (i * BLOCK + tid < t.nnz) G::gather_edge_win(xwin, pos[i], ge[i]);
    }
  };

  // ---- phase 2, short rows: one thread per row sums its products left to right and stores the row
  //      (coalesced); local row 0 continues the CTA's carry (buffer kpar), the trailing partial row
  //      (local row `nrows`) becomes the next carry ---------------------------------------------------------
  //      With list >= 0 the rows in s_long (longer than kShortRowMax) are left to whole warps: lanes sum
  //      strided, a shuffle tree combines them.
  auto reduce_short = [&](const TileRef& t, int kpar, const V* sprod, const int* srel, int list, int lbuf = 0) {
    const int* rows_long = s_long + lbuf * L::kMaxLong;
#ifdef FLEX_EXP_SKIP_REDUCE
    return;
#endif
    if (list >= 0) {
      const int n_long = s_nlong[list];
      for (int i = warp; i < n_long; i += Cfg::kWarps) {
        const int r = rows_long[i];
        const int lo = r ? srel[r - 1] : 0;
        const int hi = r < t.nrows ? srel[r] : t.nnz;
        V sum[kAcc];
#pragma unroll
        for (int j = 0; j < kAcc; ++j) sum[j] = V(0);
        for (int e = lo + lane; e < hi; e += 32) {
#pragma unroll
          for (int j = 0; j < kAcc; ++j) sum[j] += sprod[j * Cfg::kTile + e];
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
#pragma unroll
          for (int j = 0; j < kAcc; ++j) sum[j] += shfl_down_any(sum[j], off);
        }
        if (lane == 0) {
          if (r == 0) {
#pragma unroll
            for (int j = 0; j < kAcc; ++j) sum[j] = s_carry[kpar * kAcc + j] + sum[j];
          }
          if (r < t.nrows) {
            store_row(t.row0 + r, sum);
          } else {
#pragma unroll
            for (int j = 0; j < kAcc; ++j) s_carry[(kpar ^ 1) * kAcc + j] = sum[j];
          }
        }
      }
    }
    for (int r = tid; r <= t.nrows; r += BLOCK) {
      const int lo = r ? srel[r - 1] : 0;
      const int hi = r < t.nrows ? srel[r] : t.nnz;
      int n = hi - lo;
      if (list >= 0 && n > kShortRowMax) continue;
      V sum[kAcc];
#pragma unroll
      for (int j = 0; j < kAcc; ++j) sum[j] = (r == 0) ? s_carry[kpar * kAcc + j] : V(0);
      const V* q = sprod + lo;
      // rows of up to kUnroll edges (the common case) without a loop: every load is issued before the first add,
      // and threads whose rows differ in length do not diverge
      constexpr int kUnroll = (kAcc * sizeof(V) <= 8) ? 8 : ((kAcc * sizeof(V) <= 16) ? 4 : 2);
      if (n <= kUnroll) {
        V v[kUnroll][kAcc];
#pragma unroll
        for (int u = 0; u < kUnroll; ++u) {
#pragma unroll
          for (int j = 0; j < kAcc; ++j) v[u][j] = (u < n) ? q[j * Cfg::kTile + u] : V(0);
        }
#pragma unroll
        for (int u = 0; u < kUnroll; ++u) {
          if (u < n) {
#pragma unroll
            for (int j = 0; j < kAcc; ++j) sum[j] += v[u][j];
          }
        }
        n = 0;
      }
      for (; n >= 4; n -= 4, q += 4) {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
#pragma unroll
          for (int j = 0; j < kAcc; ++j) sum[j] += q[j * Cfg::kTile + u];
        }
      }
      for (; n > 0; --n, ++q) {
#pragma unroll
        for (int j = 0; j < kAcc; ++j) sum[j] += q[j * Cfg::kTile];
      }
      if (r < t.nrows) {
        store_row(t.row0 + r, sum);
      } else {
#pragma unroll
        for (int j = 0; j < kAcc; ++j) s_carry[(kpar ^ 1) * kAcc + j] = sum[j];
      }
    }
  };

  // ---- phase 2, long rows: every thread reduces its merge-path span: exactly n_items steps, each
  //      consuming one edge (accumulate) or one row end (store the row, reset); the carries are combined
  //      by a warp-shuffle segmented scan and a cross-warp fold (one barrier inside) -------------------
  auto reduce_long = [&](const TileRef& t, int kpar, const V* sprod, const int* srel, int xs, int ys, int n_items) {
    V acc[kAcc], first_val[kAcc];
#pragma unroll
    for (int j = 0; j < kAcc; ++j) { acc[j] = V(0); first_val[j] = V(0); }
    int row = xs;
    {
      int nz = ys, re = srel[xs];
#pragma unroll
      for (int i = 0; i < IPT; ++i) {
        if (i < n_items) {
          if (nz < re) {
#pragma unroll
            for (int j = 0; j < kAcc; ++j) acc[j] += sprod[j * Cfg::kTile + nz];
            ++nz;
          } else {
            // the first row a thread closes may have begun in earlier threads: keep it for after the scan
            if (row == xs) {
#pragma unroll
              for (int j = 0; j < kAcc; ++j) first_val[j] = acc[j];
            } else {
              store_row(t.row0 + row, acc);
            }
#pragma unroll
            for (int j = 0; j < kAcc; ++j) acc[j] = V(0);
            ++row;
            re = srel[row];
          }
        }
      }
    }
    // segmented inclusive scan of the carries (key = row the carry belongs to)
    const int key = row;
    V val[kAcc];
#pragma unroll
    for (int i = 0; i < kAcc; ++i) val[i] = acc[i];
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int k2 = __shfl_up_sync(0xffffffffu, key, off);
#pragma unroll
      for (int i = 0; i < kAcc; ++i) {
        const V v2 = shfl_up_any(val[i], off);
        if (lane >= off && k2 == key) val[i] += v2;
      }
    }
    if (lane == 31) {
      s_wkey[warp] = key;
#pragma unroll
      for (int i = 0; i < kAcc; ++i) s_wval[warp * kAcc + i] = val[i];
    }
    const int pk = __shfl_up_sync(0xffffffffu, key, 1);
    V pv[kAcc];
#pragma unroll
    for (int i = 0; i < kAcc; ++i) pv[i] = shfl_up_any(val[i], 1);
    named_bar_sync(1, BLOCK);   // [B] warp aggregates visible
    // fold: CTA carry (belongs to local row 0) then the aggregates of the warps before this one
    int fk = 0;
    V fv[kAcc];
#pragma unroll
    for (int i = 0; i < kAcc; ++i) fv[i] = s_carry[kpar * kAcc + i];
    for (int w = 0; w < warp; ++w) {
      const int wk = s_wkey[w];
      if (wk == fk) {
#pragma unroll
        for (int i = 0; i < kAcc; ++i) fv[i] += s_wval[w * kAcc + i];
      } else {
        fk = wk;
#pragma unroll
        for (int i = 0; i < kAcc; ++i) fv[i] = s_wval[w * kAcc + i];
      }
    }
    if (tid == BLOCK - 1) {   // carry into the next tile = inclusive value of the last thread
#pragma unroll
      for (int i = 0; i < kAcc; ++i) s_carry[(kpar ^ 1) * kAcc + i] = (fk == key) ? fv[i] + val[i] : val[i];
    }
    if (lane > 0) {
      if (pk == fk) {
#pragma unroll
        for (int i = 0; i < kAcc; ++i) fv[i] += pv[i];
      } else {
#pragma unroll
        for (int i = 0; i < kAcc; ++i) fv[i] = pv[i];
      }
    }
    if (row > xs) {   // first closed row = what earlier threads / tiles carried + this thread's part
#pragma unroll
      for (int i = 0; i < kAcc; ++i) first_val[i] = fv[i] + first_val[i];
      store_row(t.row0 + xs, first_val);
    }
  };
  auto thread_span = [&](const TileRef& t, const int* srel, int& xs, int& ys, int& n_items) {
    const int total_items = t.nrows + t.nnz;
    const int d0 = min(tid * IPT, total_items);
    n_items = min(d0 + IPT, total_items) - d0;
    merge_path_search<int, int>(d0, srel, 0, t.nrows, t.nnz, xs, ys);
  };

  if constexpr (!G::kGatherNeedsRow && !Cfg::kPipeline) {
    // ---- plain loop: stage -> registers -> gathers -> products -> classify -> reduce --------------------
    for (int k = 0; k < count; ++k) {
      TileRef t{0, 0, 0, 0, 0};
      TileT tile;
      const OffsetT* rend = nullptr;
      if (!acquire(k, t, tile, rend)) { failed = true; break; }
      last_row1 = t.row0 + t.nrows;
#ifdef FLEX_STREAM_ONLY
      release(k);
      continue;
#endif
      if (tid == 0) s_nlong[(k + 1) & 1] = 0;   // the previous tile's list has been consumed (barrier in acquire)
      const bool my_long = convert(t, rend, s_rel, k & 1);
      {
        typename G::EReg er[IPT];
        typename G::GEdge ge[IPT];
        typename G::GRow gr[1];
        if (WIN && t.win) {
          map_load_gather_win(t, tile, er, ge);
          release(k);
        } else {
          map_load(t, tile, er);
          release(k);     // as early as possible: the refill latency of this stage is what bounds the kernel
          map_gather(t, er, ge, gr);
        }
        map_products(t, er, ge, gr, s_prod);
      }
      const bool long_tile = named_bar_or(1, BLOCK, my_long);   // [P] products, s_rel and the long-row list complete
#ifdef FLEX_MERGE_WALK_REDUCE
      if (long_tile) {
        int xs, ys, n_items;
        thread_span(t, s_rel, xs, ys, n_items);
        reduce_long(t, k & 1, s_prod, s_rel, xs, ys, n_items);
        continue;
      }
#endif
      reduce_short(t, k & 1, s_prod, s_rel, long_tile ? (k & 1) : -1);   // the next tile's first barrier orders these reads
    }
  } else if constexpr (!G::kGatherNeedsRow) {
    // ---- software-pipelined loop: the gathers of tile k are in flight while tile k-1 is reduced.
    //      s_rel and s_prod are double-buffered by tile parity; one classifying barrier per tile. -------
    TileRef prev{0, 0, 0, 0, 0};
    bool prev_long = false;
    for (int k = 0; k <= count; ++k) {
      const bool have = k < count;
      TileRef cur{0, 0, 0, 0, 0};
      bool my_long = false;
      typename G::EReg er[IPT];
      typename G::GEdge ge[IPT];
      typename G::GRow gr[1];
      int* srel_k = s_rel + (k & 1) * (Cfg::kTile + 1);
      V* sprod_k = s_prod + (size_t)(k & 1) * kAcc * Cfg::kTile;
      if (have) {
        TileT tile;
        const OffsetT* rend = nullptr;
        if (!acquire(k, cur, tile, rend)) { failed = true; break; }
        last_row1 = cur.row0 + cur.nrows;
#ifdef FLEX_STREAM_ONLY
        release(k);
        continue;
#endif
        // long-row counters rotate over three slots: k % 3 is filled now, (k - 1) % 3 is read by the reduction
        // below, (k + 1) % 3 was last read before the barrier in acquire and is cleared for the next tile
        if (tid == 0) s_nlong[(k + 1) % 3] = 0;
        my_long = convert(cur, rend, srel_k, k % 3, k & 1);
        map_load(cur, tile, er);
        release(k);
        map_gather(cur, er, ge, gr);
      }
      if (k > 0) {
        const int* srel_p = s_rel + ((k - 1) & 1) * (Cfg::kTile + 1);
        const V* sprod_p = s_prod + (size_t)((k - 1) & 1) * kAcc * Cfg::kTile;
        reduce_short(prev, (k - 1) & 1, sprod_p, srel_p, prev_long ? (k - 1) % 3 : -1, (k - 1) & 1);
      }
      if (have) map_products(cur, er, ge, gr, sprod_k);
      prev_long = named_bar_or(1, BLOCK, my_long);   // [P] products, s_rel and long-row list of tile k complete
      prev = cur;
    }
  } else {
    // ---- the map needs per-row data (row-identity selectors) ---------------------------------------------
    for (int k = 0; k < count; ++k) {
      TileRef t{0, 0, 0, 0, 0};
      TileT tile;
      const OffsetT* rend = nullptr;
      if (!acquire(k, t, tile, rend)) { failed = true; break; }
      last_row1 = t.row0 + t.nrows;
      const bool my_long = convert(t, rend, s_rel, -1);
#ifdef FLEX_FORCE_EDGE_PARALLEL
      const bool long_tile = named_bar_or(1, BLOCK, true);      // experiment: every tile takes the edge-parallel path
#else
      const bool long_tile = named_bar_or(1, BLOCK, my_long);   // [R] s_rel complete, tile classified
#endif
      if (!long_tile) {
        // short rows: one thread per row does gather + map + sum in registers (the row's own vertex data is
        // loaded once) and stores the row; local row 0 continues the CTA's carry, local row `nrows`
        // (partial) becomes the next carry
        for (int r = tid; r <= t.nrows; r += BLOCK) {
          const int lo = r ? s_rel[r - 1] : 0;
          const int hi = r < t.nrows ? s_rel[r] : t.nnz;
          V sum[kAcc];
#pragma unroll
          for (int j = 0; j < kAcc; ++j) sum[j] = (r == 0) ? s_carry[(k & 1) * kAcc + j] : V(0);
          typename G::GRow grow;
          if (lo < hi) G::gather_row(p, t.row0 + r, grow);
          for (int e0 = lo; e0 < hi; e0 += Cfg::kBatch) {
            typename G::EReg er[Cfg::kBatch];
            typename G::GEdge ge[Cfg::kBatch];
#pragma unroll
            for (int b = 0; b < Cfg::kBatch; ++b)
              if (e0 + b < hi) { G::load_edge(p, tile, e0 + b, t.nz0 + e0 + b, er[b]); G::gather_edge(p, er[b], ge[b]); }
#pragma unroll
            for (int b = 0; b < Cfg::kBatch; ++b)
              if (e0 + b < hi) G::map(p, er[b], t.nz0 + e0 + b, grow, ge[b], sum);
          }
          if (r < t.nrows) {
            store_row(t.row0 + r, sum);
          } else {
#pragma unroll
            for (int j = 0; j < kAcc; ++j) s_carry[((k + 1) & 1) * kAcc + j] = sum[j];
          }
        }
        release(k);
        continue;
      }
      // a tile with a long row: whole warps take the rows one at a time -- every lane holds the row's own record,
      // lanes map edges 32 apart, a shuffle tree folds the lanes' partial sums (no shared-memory buffers)
      for (int r = warp; r <= t.nrows; r += Cfg::kWarps) {
        const int lo = r ? s_rel[r - 1] : 0;
        const int hi = r < t.nrows ? s_rel[r] : t.nnz;
        V sum[kAcc];
#pragma unroll
        for (int j = 0; j < kAcc; ++j) sum[j] = V(0);
        if (lo < hi) {
          typename G::GRow grow;
          G::gather_row(p, t.row0 + r, grow);
          for (int e = lo + lane; e < hi; e += 32) {
            typename G::EReg er;
            typename G::GEdge ge;
            G::load_edge(p, tile, e, t.nz0 + e, er);
            G::gather_edge(p, er, ge);
            G::map(p, er, t.nz0 + e, grow, ge, sum);
          }
#pragma unroll
          for (int off = 16; off > 0; off >>= 1) {
#pragma unroll
            for (int j = 0; j < kAcc; ++j) sum[j] += shfl_down_any(sum[j], off);
          }
        }
        if (lane == 0) {
          if (r == 0) {
#pragma unroll
            for (int j = 0; j < kAcc; ++j) sum[j] = s_carry[(k & 1) * kAcc + j] + sum[j];
          }
          if (r < t.nrows) {
            store_row(t.row0 + r, sum);
          } else {
#pragma unroll
            for (int j = 0; j < kAcc; ++j) s_carry[((k + 1) & 1) * kAcc + j] = sum[j];
          }
        }
      }
      release(k);
    }
  }

  // ---- hand the CTA's carry to the last CTA ---------------------------------------------------------
  // (nothing to hand over when the plan put the boundaries between this launch's CTAs on row ends)
  if (s_flag[1]) return;
  named_bar_sync(1, BLOCK);
  if (tid < kAcc) {
    V* cv = static_cast<V*>(a.carry_val) + (size_t)blockIdx.x * kAcc;
    cv[tid] = failed ? V(0) : s_carry[(count & 1) * kAcc + tid];
  }
  if (tid == 0) a.carry_row[blockIdx.x] = (failed || count == 0) ? a.num_rows : last_row1;
  named_bar_sync(1, BLOCK);
  if (tid == 0) {
    // one fence after the barrier orders every consumer thread's stores (rows, carries) before the ticket
    __threadfence();
    const unsigned t = atomicAdd(&a.header->ticket, 1u);
    s_flag[0] = (t == gridDim.x - 1) ? 1 : 0;
  }
  named_bar_sync(1, BLOCK);
  if (s_flag[0]) {
    __threadfence();
    const int n_cta = gridDim.x;
    const V* cvals = static_cast<const V*>(a.carry_val);
    for (int c = tid; c < n_cta; c += BLOCK) {
      // the CTA's row, its neighbours' rows and its value are requested together: one memory round trip
      const long long row = __ldcg(a.carry_row + c);
      const long long row_before = c > 0 ? __ldcg(a.carry_row + c - 1) : -1;
      long long row_after = c + 1 < n_cta ? __ldcg(a.carry_row + c + 1) : -1;
      V sum[kAcc];
#pragma unroll
      for (int i = 0; i < kAcc; ++i) sum[i] = __ldcg(cvals + (size_t)c * kAcc + i);
      if (row >= a.num_rows) continue;
      if (row_before == row) continue;   // not the head of its run
      for (int c2 = c + 1; c2 < n_cta && row_after == row; ++c2, row_after = c2 < n_cta ? __ldcg(a.carry_row + c2) : -1) {
#pragma unroll
        for (int i = 0; i < kAcc; ++i) sum[i] += __ldcg(cvals + (size_t)c2 * kAcc + i);
      }
      static_for<G::kNumReducers>([&](auto R) {
        constexpr int d = G::template red_dim<R.value>();
        constexpr int o = G::template red_off<R.value>();
        V* dst = G::template red_out<R.value>(p) + (size_t)row * d;
#pragma unroll
        for (int i = 0; i < d; ++i) dst[i] = __ldcg(dst + i) + sum[o + i];
      });
    }
    if (tid == 0) a.header->ticket = 0;
  }
}

}  // namespace flex
