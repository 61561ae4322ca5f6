// Host side of one generated graph: workspace sizing, planning (merge-path partition into the
// workspace), launch.  FLEXSPMV_DEFINE_GRAPH(symbol_suffix, GraphStruct, Cfg...) emits the five
// extern "C" entry points declared by FLEXSPMV_DECLARE_GRAPH in include/flexspmv.h.
//
// Replaces the reference's host dispatch (merged_spmv_dispatch / merged_spmv_launch,
// include/merged_spmv.cuh:22-182): no per-call device-attribute queries, no per-call temp-storage
// allocation, one kernel launch per operator call, partition cached in the caller's workspace.
#pragma once
#include <atomic>
#include <cstdlib>
#include <mutex>

#include "flex_common.cuh"
#include "flex_edge_kernel.cuh"
#include "flex_tile_kernel.cuh"
#include "flex_warp_ahead.cuh"
#include "flex_warp_kernel.cuh"

namespace flex {

// implemented in flex_core.cu
int partition_launch(const void* d_row_offsets, int offset_bits, long long num_rows, long long num_edges,
                     int tile_items, void* d_coords, cudaStream_t stream, void* ws, const WorkspaceHeader* h);
int device_sm_count();
void note_kernel(int which, int row_batch = 0);      // for flexspmv_debug_last_kernel, flexspmv_debug_last_row_batch
int header_init_launch(void* ws, const WorkspaceHeader& h, cudaStream_t stream);
int snap_cta_boundaries_launch(const void* d_row_offsets, int offset_bits, long long num_rows, long long num_tiles, int grid,
                               const TileRoom& room, void* d_coords, void* ws, cudaStream_t stream);
int whole_rows_launch(const void* d_row_offsets, int offset_bits, long long num_rows, long long num_edges, long long num_tiles,
                      const TileRoom& room, const RowLoopRule& rule, int grid, void* d_coords, void* ws, cudaStream_t stream);
int window_plan_launch(const void* d_coords, int offset_bits, long long num_tiles, const int* d_idx, int rec_bytes,
                       int win_bytes, void* d_table, void* d_local_idx, cudaStream_t st);
int window_ready_launch(void* ws, cudaStream_t st);

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

struct NoWindows {   // in place of CfgWin: the gather-window variant of the kernel is not built and the flag is ignored
  static constexpr int kTile = 0;
};

struct NoLean {      // in place of CfgLean: the warp kernel for matrices with random columns is not built
  static constexpr int kChunk = 0;
};

struct NoBig {       // in place of CfgBig: one configuration of the tile kernel for launches of every size
  static constexpr int kTile = 0, kIpt = 0, kMinCtas = 1, kWarps = 1;
};

template <class G, class Cfg, class CfgWin = Cfg, class CfgLean = NoLean, class CfgBig = NoBig>
struct GraphApi {
  static constexpr bool kBigBuilt = !std::is_same_v<CfgBig, NoBig>;
  static constexpr bool kWindowsBuilt = !std::is_same_v<CfgWin, NoWindows>;
  static constexpr bool kLeanBuilt = !std::is_same_v<CfgLean, NoLean>;
  using V = typename G::V;
  // edge kernel: 256 threads x 4 edges per thread (measured on B200, 2^27 edges: 2 / 4 / 8 edges per thread give
  // 91.5 / 90.8 / 62.9 % of the HBM peak for a product + global sum and 76.4 / 94.2 / 77.9 % for a gather written in place)
  static constexpr int kEdgeBlock = 256, kEdgeIpt = 4;
  // Row-mode graphs run one thread per row, the trailing partial row of the tile included: on a mesh with
  // exactly kIpt merge items per row (3 edges + the row end at kIpt = 4) a full tile holds kBlock rows plus
  // that partial row, which would cost a second pass over the rows for one thread's worth of work (measured
  // on the shallow-water model graph: 40.7 % -> 48.7 % of the HBM peak).  One row less per tile avoids it.
  static constexpr int kDefaultTile = Cfg::kTile - (G::kHasReducer && G::kGatherNeedsRow ? Cfg::kIpt : 0);

  // Gather windows are used when the graph supports them and the caller asked for them in the descriptor.
  static bool use_win(const flexspmv_desc* d) {
    if constexpr (G::kHasReducer && kWindowsBuilt) return G::kWindowGather && (d->reserved & FLEXSPMV_FLAG_GATHER_WINDOWS) != 0;
    return false;
  }
  // The warp kernel (flex_warp_kernel.cuh) is used when it was built for the graph and the caller says that the
  // gathers have no locality; it wins over the gather windows when both flags are set.
  static bool use_lean(const flexspmv_desc* d) {
    if constexpr (G::kHasReducer && kLeanBuilt) return (d->reserved & FLEXSPMV_FLAG_RANDOM_GATHER) != 0;
    return false;
  }
  // Launches of more than a tile for each SM, of rows about as short as the configuration was made for, run one large CTA an SM
  // (CfgBig), unless the launch is a small one.  The row-mode loop is bound by what an SM has in flight: its 24 warps in
  // one CTA of 768 threads have 80 registers each (three CTAs of 288: 72; bytes spilled there and here, the stage of the shallow-water step 48 and 0,
  // swe_delta 60 and 16, Rusanov fp64 68 and 28 - 32, spring-mass fp64 in 56 and 72 registers 88 and 0), share one stage of a group
  // of 32 rows for every warp, and the one producer's book-keeping is per 735 rows instead of 191 or 255.  us, CfgBig / Cfg (steps: one model
  // replayed):
  //   shallow-water step fp64  260^2 45.0 / 49.4, 310^2 52.8 / 66.7, 400^2 78.0 / 88.3, 520^2 102.9 / 121.4, 800^2 221 / 248, 1024^2 332 / 368, 1200^2
  //                            455 / 503; 200^2, a small launch there: 32.8 / 28.4
  //   Rusanov fp64             400^2 15.3 / 15.6, 450^2 18.7 / 19.8, 520^2 23.4 / 24.6, 800^2 48.0 / 50.0, 1024^2 74.0 / 76.3, 1200^2 100 / 106
  //   spring-mass fp64         600^2 26.1 / 32.2, 1024^2 62.0 / 70.2, 1500^2 123 / 135; fp32 (with words of four edges) 600^2 14.8 / 16.2, 1024^2 35.9 / 38.3,
  //                            1500^2 65.9 / 72.7
  //   Rusanov fp32             450^2 11.4 / 12.3, 520^2 14.1 / 15.8, 800^2 29.4 / 32.9, 1024^2 45.8 / 48.9, 1200^2 59.3 / 64.0
  // A tile has to hold about a row a thread (7 to 11 for ten), or warps wait for a stage, or go round it twice.  8 M items: rows of 8 Rusanov fp64
  // 116 / 103, fp32 59.4 / 56.8, swe_delta fp64 102 / 98; of 6 81.8 / 85.0, 47.7 / 46.4, 68.9 / 76.9; of 4 76.7 / 83.6, 45.4 / 46.4, 64.9 / 71.8; of 1 - 7
  // 103.8 / 114.4, 59.4 / 67.3, 77.6 / 89.8; of 2 76.6 / 81.8, 47.7 / 49.2, 70.6 / 65.4 (3 M items: 32.9 / 36.7, 20.7 / 20.1, 30.4 / 28.4).
  // Spring-mass fp32, 9 M items: rows of 8 31.3 / 42.3, of 4 - 12 46.7 / 52.4, of 9 38.6 / 36.5 (three words for a row, which single indices read
  // without conflicts): 8.5 rows for ten threads at least.
  // So a row of more than kWholeRowMax edges costs a launch far more there (the loop with carries, one barrier for 24 warps), and nothing in the
  // description tells: a caller who has seen the plan names the longest row (FLEXSPMV_LONGEST_ROW), and others get the usual configuration.  Units
  // with an epilogue take plans of whole rows only.  us, CfgBig / Cfg, without whole rows, columns within 300 rows: one row in 1000 of 40 edges among rows of 3, 8 M
  // items Rusanov fp64 270 / 227, fp32 170 / 131, swe_delta 215 / 172; one in 5000 of 1000 531 / 276, 271 / 172, 338 / 194 (one in 100 of 40 384 / 397, 216 / 212, 284 /
  // 338; one in ten of 14 among rows of 2 238 / 250, 130 / 158, 173 / 187); one row of 40 among rows of 8, spring-mass fp32 9 M 51.9 / 46.9, fp64 4 M 51.2 / 48.8; SpMV, one
  // of 40 among rows of 27 fp64 4.5 M 16.0 / 15.3, fp32 2.2 M 9.6 / 8.4, 3 M 9.8 / 10.1, of 900 among rows of 31 2.2 M 12.2 / 8.8, 6 M 18.0 / 21.2.
  // Of whole rows the plan says that there is no longest one where it has more than four times the mean's edges, behind which lanes idle (RowLoopRule::most_row):
  // one row of 12, 24 among rows of 3 Rusanov fp64 3 M items 30.0 / 30.8, 34.0 / 33.3; of 32 among rows of 8 spring-mass 9 M fp32 33.2 / 42.2, fp64 69.3 / 79.9 -- and for
  // 8-byte values of graphs that read edge tensors in place where rows are uneven (most_slots: more than 1.005 lane-steps an edge): lattices with one edge in 20
  // left out, spring-mass fp64 500^2 20.8 / 19.1, 600^2 27.4 / 30.2, 1024^2 65.4 / 63.3, 1300^2 101.6 / 92.8, one in ten 64.5 / 61.8 and 103 / 90; one in 100 1300^2 103 / 99.
  // (fp32 one in 20 600^2 16.0 / 18.3, 1024^2 39.9 / 43.8, one in five 38.3 / 39.8, though rows of 6 - 10 with columns side by side 4 M items 32.1 / 25.9.  Graphs that stage
  // their edge tensors: rows of 0 - 6 fp64 Rusanov 3 M items 53.5 / 57.6, 8 M 131 / 133, swe_delta 41.3 / 42.1, 98.6 / 98.7, fp32 Rusanov 28.5 / 33.3.)
  // Callers that name a tile or a number of CTAs get the configuration that they know.
  static constexpr int kBigTile = CfgBig::kTile - (G::kGatherNeedsRow ? CfgBig::kIpt : 0), kLeastRows = G::kGroup > 1 ? 17 : 14;      // rows a tile, for 20 threads
  // Two-phase graphs (SpMV): rows of 21 to 32 edges on average.  A tile of 1280 items holds 45 rows of 27, so that a warp has 32 of them or 13, and
  // a row takes seven rounds of four gathers; two CTAs of 12 warps leave registers for nine at a time and hold 100 or 125 rows.  us, CfgBig / Cfg,
  // 27 columns a row: fp32 300 007 rows 15.3 / 18.4, 1 M 39.8 / 49.9, 3 M 116 / 149; fp64 21.8 / 23.6, 60.3 / 65.4, 175 / 189.  12 M items, columns side by side, fp32
  // and fp64: rows of 24 29.2 / 30.6, 42.4 / 43.9; of 31 20.6 / 25.4, 28.8 / 31.8; of 32 61.7 / 67.3, 64.7 / 65.3; of 20 - 32 22.8 / 25.8, 33.5 / 33.8.  Shorter ones gain where
  // they begin in many banks, and lose where they do not: of 18 18.4 / 24.1, 26.3 / 29.0, of 20 21.7 / 22.4, 31.4 / 30.1 (3 M items fp32 9.4 / 8.8), of 16 42.4 / 40.7, 64.5 / 63.8.
  static constexpr int kBigRowEdges = 21;
  static int longest_row(const flexspmv_desc* d) {
    const unsigned n = (unsigned)d->reserved >> 8;
    return n <= (unsigned)kWholeRowMax ? (int)n : 0;
  }
  static int uses_longest_row(const flexspmv_desc* d) {
    if constexpr (G::kHasReducer) {
      if (check_desc(d) != 0) return 0;
      flexspmv_desc known = *d;
      known.reserved = (d->reserved & 255) | FLEXSPMV_LONGEST_ROW(kWholeRowMax);
      if (use_big(&known)) return G::kEpilogue ? 0 : 1;
      if (kOneRoundBuilt<Cfg> && !use_lean(d) && !use_win(d)) return row_edges_within(d, 4, sizeof(V) == 4 ? 7 : 5) ? 2 : 0;
    }
    return 0;
  }
  static bool use_big(const flexspmv_desc* d) {
    if constexpr (kBigBuilt) {
      if (!G::kEpilogue && !longest_row(d)) return false;
      // (a launch asks several times: what needs no look at the device first)
      const long long items = d->num_rows + d->num_edges;
      if (items <= kBigTile || d->tile_items > 0 || d->max_ctas > 0 || use_lean(d) || use_win(d)) return false;
      if constexpr (G::kGatherNeedsRow) {
        const long long ten_rows = 10 * d->num_rows * kBigTile, each_a_row = items * CfgBig::kBlock;
        if (2 * ten_rows < kLeastRows * each_a_row || ten_rows > 11 * each_a_row) return false;
      } else if (d->num_edges < (long long)kBigRowEdges * d->num_rows || d->num_edges > (long long)kWholeRowMax * d->num_rows) {
        return false;
      }
      const long long sms = device_sm_count();
      if (items <= sms * CfgBig::kMinCtas * kBigTile) return false;
      if constexpr (G::kGatherNeedsRow) {
        // No more rows a tile than threads, or a warp goes round it for one group of 32.  us, triangles of 1024^2 squares, one edge in 100 left out: Rusanov fp64 (741
        // rows for 736) 82.4 / 79.0, swe_delta 72.9 / 69.0, in 20 (764) 72.6 / 68.0; Rusanov fp32 45.7 / 50.2 (998 for 992), 54.1 / 50.2 (1030).
        const long long ctas = sms * CfgBig::kMinCtas, tile = big_tile(d);
        if (100 * d->num_rows * tile > (sizeof(V) == 4 ? 101ll : 100ll) * CfgBig::kBlock * items) return false;
        // A CTA's warps take its tiles' groups of 32 rows in turns; a last turn that leaves 215 of 1000 of all their lanes without a row costs 8-byte values of
        // graphs that stage their edge tensors what the large tiles gain, up to four turns: by the share with a row, Rusanov fp64 0.75 16.4 / 15.9, 0.76 15.6 / 14.9, 0.78 16.7 /
        // 16.2, 0.79 17.1 / 17.3, 0.80 12.9 / 13.6; swe_delta 0.74 10.8 / 10.5, 0.775 13.4 / 13.0, 0.79 13.5 / 14.1.  (Spring-mass lattices fp64 0.67 19.1 / 19.8, 0.73 20.6 / 20.3,
        // 0.75 25.1 / 27.0; a stage of the shallow-water step, 406^2 squares, 0.76 17.9 / 21.2.)
        if constexpr (G::kValuesStaged && sizeof(V) == 8 && !G::kEpilogue) {
          const long long each = (items + ctas * kBigTile - 1) / (ctas * kBigTile), tile_rows = (d->num_rows * tile + items - 1) / items;
          const long long turns = (each * ((tile_rows + 31) / 32) + CfgBig::kWarps - 1) / CfgBig::kWarps;
          if (1000 * d->num_rows < 785 * 32 * ctas * turns * CfgBig::kWarps) return false;
        }
      }
      const long long tiles = (items + kDefaultTile - 1) / kDefaultTile, slots = sms * Cfg::kMinCtas;
      return !small_launch(d, tiles, tiles < slots ? tiles : slots, Cfg::kBlock + 32);
    }
    return false;
  }
  struct LargeTileRows { long long most_row = 0; int most_slots = 0; };
  static LargeTileRows large_tile_rows(const flexspmv_desc* d) {
    LargeTileRows r;
    if constexpr (kBigBuilt && G::kGatherNeedsRow && !G::kEpilogue) {
      if (use_big(d)) {
        r.most_row = 4 * d->num_edges / d->num_rows;
        r.most_slots = G::kValuesStaged || sizeof(V) == 4 ? 0 : 1005;
      }
    }
    return r;
  }
  // Up to 16 tiles a CTA are made equal in number: with tiles of one size 7.07 a CTA are as long as 8.
  static int big_tile(const flexspmv_desc* d) {
    const long long ctas = (long long)device_sm_count() * CfgBig::kMinCtas, items = d->num_rows + d->num_edges;
    const long long each = (items + ctas * kBigTile - 1) / (ctas * kBigTile);
    return (int)(each <= 16 ? (items + ctas * each - 1) / (ctas * each) : kBigTile);
  }
  static int compiled_tile(const flexspmv_desc* d) {
    if (use_lean(d)) return CfgLean::kChunk;
    return use_win(d) ? CfgWin::kTile : Cfg::kTile;
  }
  // The tile kernel's shared-memory carve-up is compiled for Cfg::kTile items; a smaller tile is allowed
  // (tests exercise odd sizes), a larger one is not.  (Shrinking the default tile on small problems until every
  // CTA gets the same number of tiles was measured on B200 and changed nothing: 13.1 us against 13.0 us per
  // launch on the 2-D Poisson 512^2 matrix.)
  static int tile_items(const flexspmv_desc* d) {
    if (d->tile_items > 0) return d->tile_items;
    if (use_lean(d)) return CfgLean::kChunk;
    if (use_big(d)) return big_tile(d);
    return use_win(d) ? CfgWin::kTile : kDefaultTile;
  }
  static int max_ctas(const flexspmv_desc* d, int resident) {
    int m = d->max_ctas > 0 ? d->max_ctas : device_sm_count() * resident;
    return m > kMaxCtas ? kMaxCtas : (m < 1 ? 1 : m);
  }
  static int check_desc(const flexspmv_desc* d) {
    if (!d) return FLEXSPMV_ERR_BAD_ARG;
    if (d->num_rows < 0 || d->num_edges < 0) return FLEXSPMV_ERR_BAD_ARG;
    if (G::kHasReducer && d->offset_bits != 32 && d->offset_bits != 64) return FLEXSPMV_ERR_BAD_ARG;
    if (G::kHasReducer && d->tile_items > compiled_tile(d)) return FLEXSPMV_ERR_TOO_LARGE;
    if (G::kHasReducer && d->offset_bits == 32 && d->num_rows + d->num_edges >= (1ll << 31)) return FLEXSPMV_ERR_TOO_LARGE;
    return 0;
  }
  static long long num_tiles(const flexspmv_desc* d) {
    if (!G::kHasReducer) return 0;
    const long long t = tile_items(d);
    return (d->num_rows + d->num_edges + t - 1) / t;
  }
  static void layout(const flexspmv_desc* d, WorkspaceHeader& h) {
    const long long tiles = num_tiles(d);
    const uint64_t pair = (d->offset_bits == 64 ? 16u : 8u);
    h.coords_offset = sizeof(WorkspaceHeader);
    h.carry_row_offset = align_up(h.coords_offset + (uint64_t)(tiles + 1) * pair, 256);
    const uint64_t carries = use_lean(d) ? kMaxWarpCarries : kMaxCtas;      // one carry per CTA, or per warp
    h.carry_val_offset = align_up(h.carry_row_offset + carries * 8u, 256);
    const int width = G::kHasReducer ? G::kAccDim : (G::kAggDim > 0 ? G::kAggDim : 1);
    h.total_bytes = align_up(h.carry_val_offset + carries * width * sizeof(V), 256);
    h.win_table_offset = h.win_index_offset = 0;
    if (use_win(d) && !use_lean(d)) {
      h.win_table_offset = h.total_bytes;
      h.win_index_offset = align_up(h.win_table_offset + (uint64_t)tiles * kWinEntryInts * 4u, 256);
      h.total_bytes = align_up(h.win_index_offset + (uint64_t)d->num_edges * 2u, 256);
    }
  }

  static int info(flexspmv_graph_info* o) {
    if (!o) return FLEXSPMV_ERR_BAD_ARG;
    o->num_values = G::kNumValues; o->num_indices = G::kNumIndices; o->num_outputs = G::kNumOutputs;
    o->has_reducer = G::kHasReducer ? 1 : 0; o->value_bytes = (int)sizeof(V);
    o->default_tile_items = kDefaultTile; o->block_threads = Cfg::kBlock; o->items_per_thread = Cfg::kIpt;
    o->stages = Cfg::kStages;
    o->smem_bytes = 0;
    if constexpr (G::kHasReducer) o->smem_bytes = TileSmemLayout<G, long long, Cfg>::kTotal;
    o->acc_dim = G::kHasReducer ? G::kAccDim : G::kAggDim;
    o->reserved = 0;
    // bit 0: the graph can use gather windows, bit 1: the warp kernel for random columns is built
    if constexpr (G::kHasReducer) o->reserved = ((G::kWindowGather && kWindowsBuilt) ? 1 : 0) | (kLeanBuilt ? 2 : 0);
    return 0;
  }

  static int workspace_bytes(const flexspmv_desc* d, size_t* bytes) {
    if (int e = check_desc(d)) return e;
    if (!bytes) return FLEXSPMV_ERR_BAD_ARG;
    WorkspaceHeader h{};
    layout(d, h);
    *bytes = (size_t)h.total_bytes;
    return 0;
  }

  // What a tile of the kernel compiled with configuration C can take (the layout of its stage).
  template <class C>
  static TileRoom tile_room(const flexspmv_desc* d) {
    TileRoom room;
    room.max_edges = C::kTile;
    room.edge_bytes = G::kStreamBytesPerEdge;
    room.offset_bytes = d->offset_bits / 8;
    room.stage_bytes = d->offset_bits == 64 ? TileSmemLayout<G, long long, C>::kRecordBytes : TileSmemLayout<G, int, C>::kRecordBytes;
    if (G::kDirectLoads) room.stage_bytes = 0x7fffffff;
    return room;
  }

  static TileRoom room_of(const flexspmv_desc* d) {
    if constexpr (kBigBuilt) if (use_big(d)) return tile_room<CfgBig>(d);
    return tile_room<Cfg>(d);
  }

  // `whole_rows`: also look for a matrix of short rows whose tiles can all hold whole rows.
  // `indices` (may be null): the launch's index arrays, which the choice of the loop on such tiles looks at.
  static int plan(const flexspmv_desc* d, const void* const* indices, const void* row_offsets, void* ws, size_t ws_bytes, cudaStream_t st,
                  bool whole_rows = true) {
    if (int e = check_desc(d)) return e;
    if (!ws) return FLEXSPMV_ERR_WORKSPACE;
    WorkspaceHeader h{};
    layout(d, h);
    if (ws_bytes < h.total_bytes) return FLEXSPMV_ERR_WORKSPACE;
    if (!aligned16(ws)) return FLEXSPMV_ERR_ALIGN;
    h.magic = kMagic; h.ticket = 0; h.status = 0; h.offset_bits = d->offset_bits;
    h.num_rows = d->num_rows; h.num_edges = d->num_edges; h.num_tiles = num_tiles(d);
    h.tile_items = tile_items(d); h.max_ctas = d->max_ctas;
    if constexpr (G::kHasReducer) {
      if (!row_offsets) return FLEXSPMV_ERR_BAD_ARG;
      if (!aligned16(row_offsets)) return FLEXSPMV_ERR_ALIGN;
      char* const coords = static_cast<char*>(ws) + h.coords_offset;
      if (int e = partition_launch(row_offsets, d->offset_bits, d->num_rows, d->num_edges, tile_items(d), coords, st, ws, &h)) return e;
      if (use_lean(d)) return 0;
      // the tile kernel: the grid it will have
      int grid = 0;
      bool win = false;
      if constexpr (G::kWindowGather && kWindowsBuilt) win = use_win(d);
      if (h.num_tiles > 1) {
        int resident = 0, e = 0;
        if constexpr (G::kWindowGather && kWindowsBuilt) {
          if (win) e = d->offset_bits == 64 ? resident_ctas<long long, CfgWin, true>(&resident) : resident_ctas<int, CfgWin, true>(&resident);
        }
        bool big = false;
        if constexpr (kBigBuilt) {
          big = use_big(d);
          if (big) e = d->offset_bits == 64 ? resident_ctas<long long, CfgBig>(&resident) : resident_ctas<int, CfgBig>(&resident);
        }
        if (!win && !big) e = d->offset_bits == 64 ? resident_ctas<long long>(&resident) : resident_ctas<int>(&resident);
        if (e) return e;
        const long long most = max_ctas(d, resident);
        grid = (int)(most < h.num_tiles ? most : h.num_tiles);
      }
      if constexpr (WholeRows<G, Cfg, false>::value) {
        RowLoopRule rule{};
        rule.edge_lanes = !G::kGatherNeedsRow;
        rule.heavy = !G::kLightMap;
        rule.accumulators = G::kAccDim;
        if (rule.edge_lanes && indices && d->num_edges > 0)
          rule.gathers = G::gathers(indices, rule.index, rule.record_bytes, RowLoopRule::kMaxGathers);
        for (int i = 0; i < rule.gathers; ++i) if (!rule.index[i]) return FLEXSPMV_ERR_BAD_ARG;
        if (const LargeTileRows suits = large_tile_rows(d); suits.most_row) { rule.most_row = suits.most_row; rule.most_slots = suits.most_slots; }
        if (grid > 0 && !use_big(d) && small_launch(d, h.num_tiles, grid, Cfg::kBlock + 32)) {
          rule.share_items = 3 * ((h.num_tiles + grid - 1) / grid) * tile_items(d) / 2;
          rule.share_row_edges = kSmallRowEdges;
        }
        // rows longer than kWholeRowMax on average: no need to look
        if (whole_rows && !use_win(d) && d->num_rows > 0 && d->num_edges <= (long long)kWholeRowMax * d->num_rows)
          return whole_rows_launch(row_offsets, d->offset_bits, d->num_rows, d->num_edges, h.num_tiles, room_of(d), rule, grid, coords, ws, st);
      }
      // boundaries between the CTAs of that grid moved onto row ends where the tiles have room
      TileRoom room = room_of(d);
      if constexpr (G::kWindowGather && kWindowsBuilt) { if (win) room = tile_room<CfgWin>(d); }
      return snap_cta_boundaries_launch(row_offsets, d->offset_bits, d->num_rows, h.num_tiles, grid, room, coords, ws, st);
    } else {
      (void)indices; (void)row_offsets; (void)whole_rows;
      return header_init_launch(ws, h, st);   // a one-thread kernel: stream-ordered, no host sync
    }
  }

  // Whether a launch takes the kernel without stages (kSmall): it is a few round trips long -- a row's ends, then its records and its
  // gathers for every kRowBatch edges -- where stages take a tile's in one copy each, behind coordinates, copies and barriers.  That
  // pays while the rows are short and the tiles few; and lanes that read rows a row length apart touch more lines an edge the longer
  // the rows are.  us, with stages / without, where lines below are drawn:
  //   tiles a CTA   5-point fp64 1.1 5.74 / 4.2, 2.1 7.13 / 5.63, 2.9 8.84 / 8.08, 3.9 10.14 / 10.46; 7-point 2.3 7.49 / 6.10, 5.4 11.98 / 14.2.
  //                 Row-mode graphs: spring-mass fp32 0.7 7.40 / 6.82, 1.9 11.4 / 11.4; Rusanov fp64 0.7 6.84 / 5.8, 1.6 11.2 / 9.9, 2.8 15.7 / 16.7
  //   edges a row   SpMV, 1 tile a CTA: fp32 12 4.2 / 3.8, 15 4.2 / 3.9, 16 5.3 / 5.6 (such rows begin in two banks: the plan takes the other
  //                 loop), 27 4.8 / 5.1; fp64 10 4.5 / 4.0, 12 4.8 / 4.7, 13 4.6 / 4.4, 15 4.7 / 4.8, 18 4.9 / 5.7, 27 5.3 / 6.3.  At 2.9: fp64 12 9.6 / 7.9,
  //                 13 9.0 / 9.2, 27 9.2 / 13.9.  Row-mode, 0.6 M items: spring-mass fp32 10 6.2 / 5.8, 14 7.4 / 7.2, 16 9.9 / 10.3; fp64 8 8.7 / 8.2,
  //                 12 10.8 / 11.0, 16 12.8 / 14.8; Rusanov fp32 6 6.7 / 6.7, 8 7.3 / 8.8, 16 9.8 / 15.8; fp64 4 11.3 / 7.4, 6 (0.15 M) 5.8 / 6.3;
  //                 swe_delta fp32 6 6.4 / 6.4, 8 7.1 / 8.2
  //   rows a CTA    (several a thread, one after the other) SpMV fp64 800 7.8 / 6.6, 896 7.8 / 8.4, 1408 of one edge 8.1 / 8.9; fp32 1600 8.2 / 7.3,
  //                 1792 8.2 / 8.2, 1914 8.3 / 10.8
  //   epilogues     (as long as a row: in 8-byte values a thread's second row is as dear as a CTA's second tile) a shallow-water step, rows a
  //                 thread and tiles a CTA fp64 1 and 1.4 49.4 / 36.8, 2 and 1.7 51.2 / 53.2, 2 and 2.0 53.4 / 55.8, 2 and 2.1 68.4 / 55.9; fp32 2 and
  //                 0.3 37.6 / 34.8, 2 and 1 45.7 / 42.2, 2 and 1.4 57.0 / 45.8
  static constexpr long long kSmallQuarters = G::kGatherNeedsRow ? 9 : 4 * kSmallTiles;
  static constexpr int least(int a, int b) { return a < b ? a : b; }
  static constexpr int within(int bytes_a_row) { return G::kStreamBytesPerEdge > 0 ? bytes_a_row / G::kStreamBytesPerEdge : bytes_a_row; }
  static constexpr int kSmallRowEdges = G::kGatherNeedsRow ? least(G::kValuesStaged ? 6 : 10, within(112))
                                                           : least(G::kLightMap ? 15 : 7, within(144));
  static bool small_launch(const flexspmv_desc* d, long long tiles, long long grid, int threads) {
    if (4 * tiles > kSmallQuarters * grid || d->num_edges > kSmallRowEdges * d->num_rows) return false;
    const long long rows_a_thread = (rows_a_cta(d->num_rows, grid) + threads - 1) / threads;
    if (!G::kGatherNeedsRow) return rows_a_thread * (long long)sizeof(V) <= 24;
    return !(G::kEpilogue && sizeof(V) == 8 && rows_a_thread > 1 && rows_a_thread * grid >= tiles);
  }
  // A small launch splits the rows evenly, not the tiles.  Where a CTA's share then holds half as much again as the tiles that a CTA has at
  // most, or longer rows than above, the plan says so (share_items and share_row_edges below, WorkspaceHeader::uneven_shares) and the loop
  // with stages runs, 0.2 - 0.5 us behind the plain kernel, which a launch cannot choose without waiting for the plan.  us, plain / without
  // stages / as it is now:  SpMV, 1 and 30 edges a row in the matrix's halves, fp32 6.1 / 8.4 / 6.2, 7.9 / 15.5 / 7.9 (long on average: plain), fp64 7.5 / 10.7 /
  // 7.5; 3 and in a tenth of the rows 20 fp64 5.7 / 16.7 / 6.1; 2 and 14 fp32 5.3 / 4.3 / 4.4, 7.3 / 7.6 / 7.7, fp64 4.7 / 5.6 / 4.9, 9.0 / 13.5 / 9.1; 2 and 6 fp32 7.4 / 5.3 /
  // 5.4, fp64 5.8 / 4.8 / 4.8.  1 and 5 edges: spring-mass fp64 7.2 / 9.7 / 7.7, Rusanov fp32 6.6 / 8.6 / 7.1, swe_delta fp64 7.7 / 8.9 / 8.2.

  // Where the gathered vectors are larger than this, tiles of whole rows go round the CTAs (round_tile in flex_tile_kernel.cuh).
  // Smaller ones stay in L2 (126 MB, shared with the streams) whatever the order, and a CTA's own run keeps more of its neighbours in L1.
  // us in runs of its own / in rounds, by the size of the vectors:
  //   two-phase graphs  7-point fp32 12 MB 42.6 / 45.0, 32 112.3 / 110.6, 37 129.0 / 126.6, 43 146.9 / 146.3, 49 165.7 / 166.7, 70 247.6 / 241.4; fp64 24 MB
  //                     55.9 / 55.7, 30 69.8 / 67.9, 36 81.4 / 80.9, 41 92.2 / 89.9, 47 105.8 / 102.6; 27 columns a row fp64 24 MB 188 / 194; 5-point
  //                     fp64 23 MB 43.8 / 43.1, 27 51.8 / 51.2, 37 68.1 / 67.1, 42 78.5 / 76.1, 72 128 / 118: level up to 50 MB, with the losses below 25
  //   row-mode graphs   a shallow-water step fp64 7.7 MB 92.7 / 92.7, 12 123.5 / 114.8, 17 170.4 /
  //                     162.1, 25 247 / 227, 35 340 / 314, 50 450 / 398; spring-mass fp32 6.5 MB 32.1 / 31.4, 16 66.3 / 64.8, 20 85.0 / 81.0, 32 130.8 / 123.0,
  //                     fp64 11.6 MB 51.0 / 50.6, 25 103.2 / 99.0, 41 164.8 / 158.0; Rusanov fp64 7.7 MB 15.7 / 15.7, 12 23.9 / 23.6, 25 42.7 / 42.1, 50 84.3 / 81.3, fp32
  //                     13.5 MB 28.5 / 28.6, 26 51.6 / 52.2, 35 64.6 / 64.1, 54 100.4 / 97.8
  static constexpr long long kKeepBytes = (G::kGatherNeedsRow ? 10ll : 40ll) << 20;

  // SpMV on rows of more than four edges on average and five at most (five-point grids), and in 4-byte values seven at most (seven-point ones):
  // batches of as many, so that a row is one round of gathers instead of two, in launches without stages and in tiles a CTA's own run.  us, batches of
  // four / five: 512^2 fp64 4.9 / 4.6, 600^2 7.9 / 7.5, fp32 5.7 / 4.8; 700^2 fp64 10.1 / 9.3, 1500^2 34.5 / 33.4, fp32 26.1 / 24.0; four / seven, fp32: 60^3 4.46 / 4.18, 80^3 10.2 /
  // 9.9, 145^3 42.1 / 40.9, 200^3 110.5 / 107.5, rows of 6, 8 M items 16.6 / 16.1.  Not in rounds, where more gathers at a time leave L2 earlier: 2500^2 fp64
  // 83.0 / 86.1, 240^3 fp32 182 / 192.  Other lengths gain less than they lose: five at a time fp64, 1.2 M items without stages, rows of 4 5.25 / 5.40, of 6
  // 6.0 / 6.4, 145^3 55.2 / 58.0; seven at a time fp32, 8 M items, rows of 3 16.3 / 18.2, of 8 23.4 / 24.9, 0 - 30 22.0 / 22.8, fp64 145^3 55.2 / 68.7.  A longer row takes
  // two rounds either way, the first of which then waits for more: five at a time, fp64 rows of 4 - 6 3 M items 10.1 / 10.9, 8 M 21.1 / 23.3, 3 - 7 10.2 / 10.9, 21.8 /
  // 22.7; seven, fp32 6 - 8 8 M 16.0 / 18.2, 4 - 9 18.4 / 19.5.  So the caller has to name the longest row, which the plan knows (FLEXSPMV_LONGEST_ROW).  int64 as fp64: rows
  // of 5 3 M 10.4 / 9.3, 8 M 21.2 / 19.9, of 4 - 5 23.3 / 21.2; fp32 rows of 2 - 7 seven at a time 8 M 17.8 / 16.9 (five 19.0), one in ten of 7 among rows of 4 17.7 / 16.9.
  template <class C>
  static constexpr bool kOneRoundBuilt = !G::kGatherNeedsRow && G::kLightMap && G::kAccDim == 1 && C::kRowBatch == 4 && !C::kPipeline && !C::kLarge;
  static bool row_edges_within(const flexspmv_desc* d, int above, int most) {
    return d->num_edges > above * d->num_rows && d->num_edges <= most * d->num_rows;
  }

  // CTAs of the tile kernel that one SM holds.  The shared-memory opt-in and the occupancy are per device: looked up
  // once for each device of the process, then one word is read (a launch asks twice, for the plan's grid and for the form that it takes).
  template <typename OffsetT, class C = Cfg, bool WIN = false, int MODE = kPlain>
  static int resident_ctas(int* out) {
    using L = TileSmemLayout<G, OffsetT, C, WIN>;
    static_assert(L::kTotal <= 227 * 1024, "tile kernel needs more shared memory than one sm_100a CTA can have");
    constexpr int kMaxDevices = 64;
    static std::atomic<int> resident_of[kMaxDevices];      // 0: not looked up yet
    int dev = 0;
    if (cudaError_t e = cudaGetDevice(&dev); e != cudaSuccess) return (int)e;
    if (dev < 0 || dev >= kMaxDevices) return FLEXSPMV_ERR_BAD_ARG;
    int resident = resident_of[dev].load(std::memory_order_acquire);
    if (resident == 0) {
      static std::mutex mu;
      std::lock_guard<std::mutex> lock(mu);
      auto kernel = flex_tile_kernel<G, OffsetT, C, WIN, MODE>;
      constexpr int kThreads = C::kBlock + (G::kDirectLoads ? 0 : 32);
      cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kTotal);
      int r = 0;
      if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&r, kernel, kThreads, L::kTotal);
      if (e != cudaSuccess) { (void)cudaGetLastError(); return (int)e; }
      resident = r < 1 ? -1 : r;
      resident_of[dev].store(resident, std::memory_order_release);
    }
    if (resident < 1) return FLEXSPMV_ERR_TOO_LARGE;
    *out = resident;
    return 0;
  }

  template <typename OffsetT, class C = Cfg, bool WIN = false>
  static int launch_tiles(const flexspmv_desc* d, const typename G::Params& p, const void* row_offsets, void* ws,
                          const WorkspaceHeader& h, cudaStream_t st, bool whole_rows) {
    using L = TileSmemLayout<G, OffsetT, C, WIN>;
    auto kernel = flex_tile_kernel<G, OffsetT, C, WIN>;
    constexpr int kThreads = C::kBlock + (G::kDirectLoads ? 0 : 32);   // staged mode adds the producer warp
    int resident = 0;
    if (int e = resident_ctas<OffsetT, C, WIN>(&resident)) return e;
    const long long tiles = h.num_tiles;
    note_kernel(FLEXSPMV_KERNEL_NONE);
    if (tiles == 0) return 0;
    long long grid = max_ctas(d, resident);
    if (grid > tiles) grid = tiles;
    TileKernelArgs a;
    a.row_offsets = row_offsets;
    a.coords = static_cast<char*>(ws) + h.coords_offset;
    a.header = static_cast<WorkspaceHeader*>(ws);
    a.carry_row = reinterpret_cast<long long*>(static_cast<char*>(ws) + h.carry_row_offset);
    a.carry_val = static_cast<char*>(ws) + h.carry_val_offset;
    a.num_rows = d->num_rows; a.num_edges = d->num_edges; a.num_tiles = tiles;
    a.rounds = 0;
    a.win_table = nullptr; a.win_index = nullptr; a.num_vertices = d->num_vertices;
    if constexpr (WIN) {
      if (d->num_vertices <= 0) return FLEXSPMV_ERR_BAD_ARG;
      if (!aligned16(G::gather_base(p))) return FLEXSPMV_ERR_ALIGN;   // window sources are 16-byte aligned only then
      a.win_table = reinterpret_cast<const int*>(static_cast<char*>(ws) + h.win_table_offset);
      a.win_index = reinterpret_cast<const unsigned short*>(static_cast<char*>(ws) + h.win_index_offset);
    }
    int form = FLEXSPMV_KERNEL_TILE, row_batch = C::kRowBatch;
    if constexpr (L::kWhole) if (whole_rows) {
      const long long vertices = d->num_vertices > d->num_rows ? d->num_vertices : d->num_rows;
      bool small = false;
      if constexpr (!std::is_same_v<C, CfgBig>) {
        small = small_launch(d, tiles, grid, kThreads);
        if (small) {
          form = FLEXSPMV_KERNEL_TILE_SMALL;
          kernel = flex_tile_kernel<G, OffsetT, C, WIN, kSmall>;
          if (int e = resident_ctas<OffsetT, C, WIN, kSmall>(&resident)) return e;      // the grid stays the plan's
        }
      }
      if (!small && vertices * G::kGatherRecordBytes > kKeepBytes && tiles >= grid * C::kTileRun) {
        a.rounds = (int)(tiles / (grid * C::kTileRun));
        form = FLEXSPMV_KERNEL_TILE_ROUNDS;
        kernel = flex_tile_kernel<G, OffsetT, C, WIN, kRounds>;
        if (int e = resident_ctas<OffsetT, C, WIN, kRounds>(&resident)) return e;
      }
    }
    if constexpr (L::kWhole && !WIN && kOneRoundBuilt<C>) {
      auto batch_of = [&](auto edges) -> int {
        using One = TileCfg<C::kBlock, C::kIpt, C::kStages, C::kMinCtas, C::kBatch, false, edges.value>;      // (the same stages and tiles)
        static_assert(TileSmemLayout<G, OffsetT, One>::kTotal == L::kTotal);
        const bool small = form == FLEXSPMV_KERNEL_TILE_SMALL;
        kernel = small ? flex_tile_kernel<G, OffsetT, One, false, kSmall> : flex_tile_kernel<G, OffsetT, One, false, kPlain>;
        return small ? resident_ctas<OffsetT, One, false, kSmall>(&resident) : resident_ctas<OffsetT, One, false, kPlain>(&resident);
      };
      const int longest = longest_row(d);
      if (whole_rows && form != FLEXSPMV_KERNEL_TILE_ROUNDS && longest && row_edges_within(d, 4, longest)) {
        int e = 0;
        if (longest <= 5) { e = batch_of(IntC<5>{}); row_batch = 5; }
        else if constexpr (sizeof(V) == 4) { if (longest <= 7) { e = batch_of(IntC<7>{}); row_batch = 7; } }
        if (e) return e;
      }
    }
    note_kernel(form, row_batch);
    return launch_pdl(kernel, (unsigned)grid, kThreads, L::kTotal, st, p, a);
  }

  static constexpr int whole_warps(int threads) { return threads < 32 ? 32 : threads / 32 * 32; }
  template <typename OffsetT, class C = CfgLean, bool SMALL = false>
  static int launch_lean(const flexspmv_desc* d, const typename G::Params& p, const void* row_offsets, void* ws,
                         const WorkspaceHeader& h, cudaStream_t st) {
    if constexpr (G::kHasReducer && kLeanBuilt) {
      // Few chunks a warp: the other form, on fewer warps.  Chunks a warp, us in this form / in that: power-law rows fp32 17.4 51.0 / 45.8,
      // 20.3 60.8 / 55.7, 24.7 64.5 / 65.6, 29 73.6 / 75.2; fp64 17.4 51.8 / 48.3, 19.2 53.5 / 52.6, 20.9 56.9 / 56.6, 24.4 63.9 / 63.7, 29.6 75.1 / 74.2.
      // Of the grid that the launch will have: a few CTAs have many chunks each on a small matrix too.
      constexpr int kFewChunks = 22;
      using Small = WarpCfg<whole_warps(C::kBlock * (sizeof(V) == 4 ? 9 : 10) / 12), C::kIpt, C::kMinCtas>;
      if constexpr (!SMALL) {
        const long long ctas = d->max_ctas > 0 ? d->max_ctas : (long long)device_sm_count() * C::kMinCtas;
        if (h.num_tiles < kFewChunks * ctas * Small::kWarps) return launch_lean<OffsetT, Small, true>(d, p, row_offsets, ws, h, st);
      }
      const auto kernel = [] {          // (the other one is not compiled for this configuration)
        if constexpr (SMALL) return &flex_warp_ahead_kernel<G, OffsetT, C>;
        else return &flex_warp_kernel<G, OffsetT, C>;
      }();
      // per warp: the product slots and marker words of one chunk (WarpSmem, the layout of flex_warp_kernel)
      constexpr int kSmem = WarpSmem<G, C>::template cta_bytes<OffsetT>();
      constexpr int kMaxDevices = 64;
      static std::mutex mu;
      static int resident_of[kMaxDevices] = {};      // 0: not initialised yet
      int dev = 0;
      if (cudaError_t e = cudaGetDevice(&dev); e != cudaSuccess) return (int)e;
      if (dev < 0 || dev >= kMaxDevices) return FLEXSPMV_ERR_BAD_ARG;
      int resident = 0;
      {
        std::lock_guard<std::mutex> lock(mu);
        if (resident_of[dev] == 0) {
          cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
          int r = 0;
          if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&r, kernel, C::kBlock, kSmem);
          if (e != cudaSuccess) { (void)cudaGetLastError(); return (int)e; }
          resident_of[dev] = r < 1 ? -1 : r;
        }
        resident = resident_of[dev];
      }
      if (resident < 1) return FLEXSPMV_ERR_TOO_LARGE;
      const long long chunks = h.num_tiles;
      note_kernel(FLEXSPMV_KERNEL_NONE);
      if (chunks == 0) return 0;
      long long grid = d->max_ctas > 0 ? d->max_ctas : (long long)device_sm_count() * resident;
      const long long need = (chunks + C::kWarps - 1) / C::kWarps;
      if (grid > need) grid = need;
      if (grid > kMaxWarpCarries / C::kWarps) grid = kMaxWarpCarries / C::kWarps;
      if (SMALL && grid > WarpSmem<G, C>::template carries<OffsetT>()) grid = WarpSmem<G, C>::template carries<OffsetT>();
      if (grid < 1) grid = 1;
      WarpKernelArgs a;
      a.row_offsets = row_offsets;
      a.coords = static_cast<char*>(ws) + h.coords_offset;
      a.header = static_cast<WorkspaceHeader*>(ws);
      a.carry_row = reinterpret_cast<long long*>(static_cast<char*>(ws) + h.carry_row_offset);
      a.carry_val = static_cast<char*>(ws) + h.carry_val_offset;
      a.num_rows = d->num_rows; a.num_edges = d->num_edges; a.num_chunks = chunks;
      note_kernel(SMALL ? FLEXSPMV_KERNEL_WARP_AHEAD : FLEXSPMV_KERNEL_WARP);
      return launch_pdl(kernel, (unsigned)grid, C::kBlock, kSmem, st, p, a);
    } else {
      (void)d; (void)p; (void)row_offsets; (void)ws; (void)h; (void)st;
      return FLEXSPMV_ERR_BAD_ARG;
    }
  }

  // Second planning step for descriptors with FLEXSPMV_FLAG_GATHER_WINDOWS (after plan, same workspace): reads the
  // index array of the graph's one gather and fills the per-tile segment table and the per-edge positions.
  // Until it has run, a launch treats every tile as having no windows.
  static int plan_windows(const flexspmv_desc* d, const void* const* indices, void* ws, size_t ws_bytes, cudaStream_t st) {
    if (int e = check_desc(d)) return e;
    if (!use_win(d) || use_lean(d)) return 0;          // nothing to do for graphs / descriptors without windows
    if constexpr (G::kHasReducer && G::kWindowGather && kWindowsBuilt) {
      if (!ws) return FLEXSPMV_ERR_WORKSPACE;
      if (!indices || !indices[0]) return FLEXSPMV_ERR_BAD_ARG;
      WorkspaceHeader h{};
      layout(d, h);
      if (ws_bytes < h.total_bytes) return FLEXSPMV_ERR_WORKSPACE;
      char* base = static_cast<char*>(ws);
      if (int e = window_plan_launch(base + h.coords_offset, d->offset_bits, num_tiles(d), static_cast<const int*>(indices[0]),
                                     G::kGatherRecBytes, G::kWinBytes, base + h.win_table_offset, base + h.win_index_offset, st))
        return e;
      return window_ready_launch(ws, st);
    }
    return 0;
  }

  // `whole_rows`: false where the plan did not look for whole rows (the forms that are for them only cost such a launch).
  static int launch(const flexspmv_desc* d, const void* const* values, const void* const* indices,
                    const void* row_offsets, void* const* outputs, void* ws, size_t ws_bytes, cudaStream_t st, bool whole_rows = true) {
    if (int e = check_desc(d)) return e;
    if (!ws) return FLEXSPMV_ERR_WORKSPACE;
    if ((G::kNumValues && !values) || (G::kNumIndices && !indices) || (G::kNumOutputs && !outputs)) return FLEXSPMV_ERR_BAD_ARG;
    WorkspaceHeader h{};
    layout(d, h);
    if (ws_bytes < h.total_bytes) return FLEXSPMV_ERR_WORKSPACE;
    h.num_tiles = num_tiles(d);
    for (int i = 0; i < G::kNumValues; ++i) if (!values[i]) return FLEXSPMV_ERR_BAD_ARG;
    for (int i = 0; i < G::kNumIndices; ++i) if (!indices[i]) return FLEXSPMV_ERR_BAD_ARG;
    for (int i = 0; i < G::kNumOutputs; ++i) if (!outputs[i]) return FLEXSPMV_ERR_BAD_ARG;
    typename G::Params p = G::make_params(values, indices, outputs);
    if (!G::pointers_aligned(p)) return FLEXSPMV_ERR_ALIGN;
    if constexpr (G::kHasReducer) {
      if (!row_offsets) return FLEXSPMV_ERR_BAD_ARG;
      if (!aligned16(row_offsets)) return FLEXSPMV_ERR_ALIGN;
      if (use_lean(d)) {
        if (d->offset_bits == 64) return launch_lean<long long>(d, p, row_offsets, ws, h, st);
        return launch_lean<int>(d, p, row_offsets, ws, h, st);
      }
      if constexpr (G::kWindowGather && kWindowsBuilt) {
        if (use_win(d)) {
          if (d->offset_bits == 64) return launch_tiles<long long, CfgWin, true>(d, p, row_offsets, ws, h, st, whole_rows);
          return launch_tiles<int, CfgWin, true>(d, p, row_offsets, ws, h, st, whole_rows);
        }
      }
      if constexpr (kBigBuilt) {
        if (use_big(d)) {
          if (d->offset_bits == 64) return launch_tiles<long long, CfgBig>(d, p, row_offsets, ws, h, st, whole_rows);
          return launch_tiles<int, CfgBig>(d, p, row_offsets, ws, h, st, whole_rows);
        }
      }
      if (d->offset_bits == 64) return launch_tiles<long long>(d, p, row_offsets, ws, h, st, whole_rows);
      return launch_tiles<int>(d, p, row_offsets, ws, h, st, whole_rows);
    } else {
    note_kernel(FLEXSPMV_KERNEL_NONE);
    if (d->num_edges == 0 && G::kAggDim == 0) return 0;
    note_kernel(FLEXSPMV_KERNEL_EDGE);
    const long long tile_edges = (long long)kEdgeBlock * kEdgeIpt;
    long long grid = (d->num_edges + tile_edges - 1) / tile_edges;
    const long long cap = max_ctas(d, 2048 / kEdgeBlock);
    if (grid > cap) grid = cap;
    if (grid < 1) grid = 1;
    EdgeKernelArgs a;
    a.header = static_cast<WorkspaceHeader*>(ws);
    a.partials = static_cast<char*>(ws) + h.carry_val_offset;
    a.num_edges = d->num_edges;
    return launch_pdl(flex_edge_kernel<G, kEdgeBlock, kEdgeIpt>, (unsigned)grid, kEdgeBlock, 0, st, p, a);
    }
  }

  static int device_status(const void* ws, int32_t* d_out, cudaStream_t st) {
    if (!ws || !d_out) return FLEXSPMV_ERR_BAD_ARG;
    const char* src = static_cast<const char*>(ws) + offsetof(WorkspaceHeader, status);
    return (int)cudaMemcpyAsync(d_out, src, sizeof(int32_t), cudaMemcpyDefault, st);
  }
};

}  // namespace flex

// (behind CFGWIN: the configuration of the warp kernel, and where there is one that of large launches)
#define FLEXSPMV_DEFINE_GRAPH(SYM, GRAPH, CFG, CFGWIN, ...)                                                          \
  extern "C" {                                                                                                  \
  int flexspmv_##SYM##_info(flexspmv_graph_info* info) { return flex::GraphApi<GRAPH, CFG, CFGWIN, __VA_ARGS__>::info(info); } \
  int flexspmv_##SYM##_workspace_bytes(const flexspmv_desc* d, size_t* b) {                                     \
    return flex::GraphApi<GRAPH, CFG, CFGWIN, __VA_ARGS__>::workspace_bytes(d, b);                                           \
  }                                                                                                             \
  int flexspmv_##SYM##_plan(const flexspmv_desc* d, const void* ro, void* ws, size_t wb, void* st) {            \
    return flex::GraphApi<GRAPH, CFG, CFGWIN, __VA_ARGS__>::plan(d, nullptr, ro, ws, wb, static_cast<cudaStream_t>(st));     \
  }                                                                                                             \
  int flexspmv_##SYM##_plan_indexed(const flexspmv_desc* d, const void* const* ix, const void* ro, void* ws, size_t wb, void* st) { \
    if (!ix) return FLEXSPMV_ERR_BAD_ARG;                                                                       \
    return flex::GraphApi<GRAPH, CFG, CFGWIN, __VA_ARGS__>::plan(d, ix, ro, ws, wb, static_cast<cudaStream_t>(st));          \
  }                                                                                                             \
  int flexspmv_##SYM##_plan_windows(const flexspmv_desc* d, const void* const* ix, void* ws, size_t wb, void* st) { \
    return flex::GraphApi<GRAPH, CFG, CFGWIN, __VA_ARGS__>::plan_windows(d, ix, ws, wb, static_cast<cudaStream_t>(st));      \
  }                                                                                                             \
  int flexspmv_##SYM##_launch(const flexspmv_desc* d, const void* const* v, const void* const* ix,              \
                              const void* ro, void* const* o, void* ws, size_t wb, void* st) {                  \
    return flex::GraphApi<GRAPH, CFG, CFGWIN, __VA_ARGS__>::launch(d, v, ix, ro, o, ws, wb, static_cast<cudaStream_t>(st));  \
  }                                                                                                             \
  int flexspmv_##SYM##_uses_longest_row(const flexspmv_desc* d) {                                               \
    return flex::GraphApi<GRAPH, CFG, CFGWIN, __VA_ARGS__>::uses_longest_row(d);                                \
  }                                                                                                             \
  int flexspmv_##SYM##_device_status(const void* ws, int32_t* out, void* st) {                                  \
    return flex::GraphApi<GRAPH, CFG, CFGWIN, __VA_ARGS__>::device_status(ws, out, static_cast<cudaStream_t>(st));           \
  }                                                                                                             \
  }


// ---- an entry point for callers that cannot allocate device memory -----------------------------------
// FLEXSPMV_DEFINE_STATIC_SCRATCH_LAUNCH(symbol_suffix, GraphStruct, Cfg, BYTES) expands, inside the
// translation unit of one graph, to a file-scope device array of BYTES bytes and to
//   int flexspmv_<suffix>_launch_static(desc, values, indices, row_offsets, outputs, stream)
// which plans the problem into that array and launches the fused pass, calling no allocator of any kind.
// The array's name is only a host-side handle for the symbol; its device address is looked up once per
// device with cudaGetSymbolAddress (with that device current) and cached.
#define FLEXSPMV_DEFINE_STATIC_SCRATCH_LAUNCH(SYM, GRAPH, CFG, BYTES)                                           \
  static __device__ __align__(256) unsigned char flexspmv_static_scratch_##SYM[BYTES];                          \
  namespace {                                                                                                   \
  struct StaticScratch_##SYM {                                                                                  \
    std::mutex mu;                                                                                              \
    void* ptr[64] = {};                                                                                         \
    int lookup(void** out) {                                                                                    \
      int dev = -1;                                                                                             \
      cudaError_t e = cudaGetDevice(&dev);                                                                      \
      if (e != cudaSuccess) return (int)e;                                                                      \
      if (dev < 0 || dev >= 64) return FLEXSPMV_ERR_BAD_ARG;                                                    \
      std::lock_guard<std::mutex> lock(mu);                                                                     \
      if (!ptr[dev]) {                                                                                          \
        void* p = nullptr;                                                                                      \
        e = cudaGetSymbolAddress(&p, flexspmv_static_scratch_##SYM);                                            \
        if (e != cudaSuccess) return (int)e;                                                                    \
        ptr[dev] = p;                                                                                           \
      }                                                                                                         \
      *out = ptr[dev];                                                                                          \
      return 0;                                                                                                 \
    }                                                                                                           \
  } static_scratch_##SYM;                                                                                       \
  }                                                                                                             \
  extern "C" int flexspmv_##SYM##_launch_static(const flexspmv_desc* d_in, const void* const* v,                \
                                                const void* const* ix, const void* ro, void* const* o,          \
                                                void* st) {                                                     \
    using Api = flex::GraphApi<GRAPH, CFG, flex::NoWindows>;                                                    \
    if (!d_in) return FLEXSPMV_ERR_BAD_ARG;                                                                     \
    flexspmv_desc desc = *d_in;                                                                                 \
    desc.reserved = 0; /* gather windows need a second planning step and 2 bytes of scratch per edge: not here */ \
    const flexspmv_desc* d = &desc;                                                                             \
    size_t need = 0;                                                                                            \
    if (int e = Api::workspace_bytes(d, &need)) return e;                                                       \
    if (need > (size_t)(BYTES)) return FLEXSPMV_ERR_STATIC_SCRATCH;                                             \
    void* ws = nullptr;                                                                                         \
    if (int e = static_scratch_##SYM.lookup(&ws)) return e;                                                     \
    cudaStream_t stream = static_cast<cudaStream_t>(st);                                                        \
    /* the array keeps the previous call's contents: planning rewrites the header (ticket, status) and */      \
    /* every tile coordinate this problem reads; the carry slots are written before they are read      */      \
    if (int e = Api::plan(d, nullptr, ro, ws, (size_t)(BYTES), stream, false)) return e;                             \
    return Api::launch(d, v, ix, ro, o, ws, (size_t)(BYTES), stream, false);                                    \
  }                                                                                                             \
  extern "C" int flexspmv_##SYM##_static_device_status(int32_t* d_out, void* st) {                              \
    void* ws = nullptr;                                                                                         \
    if (int e = static_scratch_##SYM.lookup(&ws)) return e;                                                     \
    return flex::GraphApi<GRAPH, CFG, flex::NoWindows>::device_status(ws, d_out, static_cast<cudaStream_t>(st)); \
  }
