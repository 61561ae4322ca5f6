// A whole Runge-Kutta step of the shallow-water model in one cooperative launch, for meshes that fit the chip: the four flux
// evaluations of flex_swe_rk.cuh one after the other, with a barrier of the grid in front of each but the first.  No
// reference counterpart.
//
// As four launches (flex_tile_kernel.cuh) a stage of a small mesh is a chain of a launch and five to nine round trips, and the mesh comes
// from L2 again every time.  Here a CTA keeps what does not change -- its cells' row ends, its edges' indices, alpha, sx and sy -- in
// shared memory from the beginning, and the running sums with them, so that a stage is a barrier, the gathers and the cell's own
// records, and its arithmetic; the wall terms, which need the CTA's own cells only, are made while the other CTAs arrive.  us a step,
// replayed, fp64, squares a side, four launches (before their large CTAs) / one: 50 22.5 / 20.5, 101 24.6 / 20.6, 150 28.7 / 21.0, 200 30.5 / 22.5, 260
// 51.4 (44.5 with them) / 28.7, 320 72 (54) / 38.4, 370 85 (68) / 49.2; fp32 101 29.1 / 20.5, 300 42.5 / 28.7, 400 49.5 / 43.7, 480 87 / 62.7.
// Bound, on 101^2, by latencies: of 35 000 cycles 5500 up to the edges, 2000 for the first wall terms (a pow), four times 3500 for three
// gathers and their arithmetic, three times 4300 for a barrier (1400 to write out and arrive, 700 a poll, the wall terms beside it).
// Replays of a captured step begin 2.05 us apart or a multiple of it.  Measured and left out: an edge a lane, the cells' lanes adding up
// (101^2 22.5, 260^2 40.9); the next edge's gather ahead (23.7 -> 24.6); 2 - 4 gathers of a cell together (260^2 34.9); a warp for the
// wall terms beside the fluxes (320^2 44.5).
// The operations and their order are those of the launches of a stage each: the same bits.
#pragma once
#include "flex_graph_api.cuh"
#include "flex_swe_rk.cuh"

namespace flex {

constexpr int kStepSmem = 227 * 1024 - 1024;
// Threads of a CTA at most: 80 registers a thread, and 64 (a few bytes spilled) where that takes a round of cells less (260^2 34.7 /
// 28.7 us, 370^2 55.4 / 49.2; 150^2, one round either way, 21.3 / 23.9).  At least 384, so that the edges are fetched in a round or two
// (up to 125^2 22.5 -> 20.5 us).
constexpr int kStepThreads = 768, kStepMoreThreads = 1024, kStepLeastThreads = 384;

// Shared memory of a CTA: per edge its record; per cell its row's end, its first wall record and three sums.
template <class G>
struct StepShape {
  using V = typename G::V;
  static constexpr int kEdgeBytes = 3 * int(sizeof(V)) + 4, kCellBytes = 3 * int(sizeof(V)) + 4 + 4;
  long long grid, share, edges;       // CTAs, cells of each, edges of each that are kept
  int threads;                        // a cell each, a round
  bool more;
  size_t bytes;
  // False where a CTA's cells and about as many edges do not fit.  A CTA an SM, or as many as the descriptor caps them at.
  // (Goes by the mesh's mean; what heavy cells cost: ShallowWaterStep._shares_are_even.)
  bool fit(const flexspmv_desc* d, long long sms) {
    if (d->num_rows < 1) return false;
    const long long most = d->max_ctas > 0 && d->max_ctas < sms ? d->max_ctas : sms;
    grid = (d->num_rows + 31) / 32;
    if (grid > most) grid = most;
    share = rows_a_cta(d->num_rows, grid);
    const long long mean = share * d->num_edges / d->num_rows + 1, left = kStepSmem - share * kCellBytes;
    if (mean * kEdgeBytes > left) return false;
    edges = mean + mean / 4 + 32;                      // some CTAs have more than others
    if (edges > left / kEdgeBytes) edges = left / kEdgeBytes;
    edges &= ~1ll;
    bytes = (size_t)(share * kCellBytes + edges * kEdgeBytes);
    const long long rounds = (share + kStepThreads - 1) / kStepThreads, fewer = (share + kStepMoreThreads - 1) / kStepMoreThreads;
    threads = (int)(((share + fewer - 1) / fewer + 31) / 32 * 32);
    more = fewer < rounds;
    if (!more) threads = (int)(((share + rounds - 1) / rounds + 31) / 32 * 32);
    if (threads < kStepLeastThreads) threads = kStepLeastThreads;
    return true;
  }
};

struct StepArgs {
  const void* row_offsets;
  WorkspaceHeader* header;
  long long num_rows, num_edges, num_tiles;
  long long share;
  int edges;                          // kept in shared memory; those behind them are read where they lie
};

// What changes from stage to stage.
template <typename V>
struct StepStages {
  V* state[2][3];                     // where the first and the third stage, and the second one, leave the next state
  SweRkCoef<V> coef[4];
};

// Per-edge arrays in shared memory.
template <class G>
struct KeptTile {
  using V = typename G::V;
  const V* v[3];
  const int* idx;
  template <int I, class T>
  __device__ __forceinline__ const T* stream(int e) const {
    if constexpr (I < 3) return v[I] + e;
    else return idx + e;
  }
};

// The wall terms of `cell`, whose first record is j (swe_wall_terms, without the search).
template <typename V>
__device__ __noinline__ WallTerms<V> swe_step_wall(const V* h, const int* wall_cell, const V* bsx, const V* bsy, int j, int end, int cell) {
  WallTerms<V> t{V(0), V(0)};
  const V half_sq = fx::vmul(V(0.5), fx::vpow(h[cell], V(2)));
  do {
    t.uh = fx::vadd(t.uh, fx::vmul(half_sq, __ldg(bsx + j)));
    t.vh = fx::vadd(t.vh, fx::vmul(half_sq, __ldg(bsy + j)));
  } while (++j < end && __ldg(wall_cell + j) == cell);
  return t;
}

// A barrier of the grid in two halves: what the CTA's threads wrote before step_arrive is seen by every CTA behind its step_wait.  One
// counter in the header that only grows, by kStepBarrier a barrier whatever the launch's grid (the first CTA counts for those that it
// does not have), so that launches of different grids may follow one another on a workspace; the barrier is open at `all`.  The wait
// is bounded (a second) and ends in FLEXSPMV_ERR_TIMEOUT.
constexpr uint64_t kStepBarrier = 1u << 20;
__device__ __forceinline__ void step_arrive(WorkspaceHeader* h, bool withhold) {
  __syncthreads();
  const uint64_t n = blockIdx.x == 0 ? kStepBarrier - (gridDim.x - 1) : 1;
  if (threadIdx.x == 0 && !withhold) asm volatile("fence.acq_rel.gpu;\n\tred.release.gpu.global.add.u64 [%0], %1;" ::"l"(&h->step_barrier), "l"(n) : "memory");
}
__device__ __forceinline__ bool step_wait(WorkspaceHeader* h, uint64_t all, int* s_ok) {
  if (threadIdx.x == 0) {
    int ok = 1;
    uint64_t t0 = 0;
    for (uint32_t i = 1;; ++i) {
      uint64_t seen;
      asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(seen) : "l"(&h->step_barrier) : "memory");
      if (seen >= all) break;
      if ((i & 63u) == 0) {
        const uint64_t t = global_timer_ns();
        if (t0 == 0) t0 = t;
        if (t - t0 > kWaitPolls) { ok = 0; raise_status(h, FLEXSPMV_ERR_TIMEOUT); break; }
      }
    }
    *s_ok = ok;
  }
  __syncthreads();
  return *s_ok != 0;
}

template <class G, typename OffsetT, int MAX_THREADS>
__global__ void __launch_bounds__(MAX_THREADS, 1) flex_swe_step_kernel(const typename G::Params params, const StepStages<typename G::V> st, const StepArgs a) {
  using V = typename G::V;
  extern __shared__ __align__(16) unsigned char s_step[];
  __shared__ int s_ok;
  const int tid = threadIdx.x, threads = blockDim.x;
  const long long first = blockIdx.x * a.share;
  const int cells = (int)(first >= a.num_rows ? 0 : (a.num_rows - first < a.share ? a.num_rows - first : a.share));
  V* const s_sum = reinterpret_cast<V*>(s_step);                      // [3][share]
  V* const s_val = s_sum + 3 * a.share;                               // alpha, sx, sy: [3][edges]
  int* const s_idx = reinterpret_cast<int*>(s_val + 3 * a.edges);     // [edges]
  int* const s_end = s_idx + a.edges;                                 // [share]: row ends, counted from the CTA's first edge
  int* const s_wall = s_end + a.share;                                // [share]: first wall record, -1: none
  const OffsetT* const ro = static_cast<const OffsetT*>(a.row_offsets);

  // the CTA's edges and wall records, the thread's first row and the header in one round trip (the first row begins at edge 0 whatever
  // row_offsets[0] says)
  const long long e_first = cells && first ? (long long)ro[first] : 0, e_last = cells ? (long long)ro[first + cells] : 0;
  const int j_first = cells ? __ldg(params.wall_start + (first >> 5)) : 0, j_last = cells ? __ldg(params.wall_start + ((first + cells + 31) >> 5)) : 0;
  OffsetT end = 0;
  if (tid < cells) end = ro[first + tid + 1];
  const WorkspaceHeader* const h = a.header;
  const uint64_t count = *reinterpret_cast<const volatile uint64_t*>(&h->step_barrier);
  if (h->magic != kMagic || h->num_tiles != a.num_tiles || h->num_rows != a.num_rows || h->num_edges != a.num_edges ||
      h->offset_bits != (int)(8 * sizeof(OffsetT)) || h->whole_rows != 1) {
    if (tid == 0 && blockIdx.x == 0) raise_not_planned(a.header);
    return;
  }
  const bool withhold = h->debug[7] != 0 && blockIdx.x == 0;      // testing aid (flexspmv_debug_withhold_stage): a CTA that never arrives
  for (int i = tid; i < cells; i += threads) s_wall[i] = -1;
  if (__syncthreads_or(h->status != 0)) return;    // an earlier launch gave up: its counter says nothing
  // as this CTA has not come to a barrier yet, fewer than all have come to the first one
  uint64_t all = count / kStepBarrier * kStepBarrier;
  const int kept = (int)(e_last - e_first < a.edges ? e_last - e_first : a.edges);
  for (int j = j_first + tid; j < j_last; j += threads) {
    const int cell = __ldg(params.wall_cell + j), before = j > j_first ? __ldg(params.wall_cell + j - 1) : -1;
    if (cell != before && cell >= first && cell < first + cells) s_wall[cell - first] = j;
  }
#pragma unroll 4
  for (int i = tid; i < kept; i += threads) {
    const V alpha = __ldg(params.alpha + e_first + i), sx = __ldg(params.sx + e_first + i), sy = __ldg(params.sy + e_first + i);
    const int idx = __ldg(params.gather_src_idx + e_first + i);
    s_val[i] = alpha; s_val[a.edges + i] = sx; s_val[2 * a.edges + i] = sy;
    s_idx[i] = idx;
  }
  for (int i = tid; i < cells; i += threads) s_end[i] = (int)((long long)(i == tid ? end : ro[first + i + 1]) - e_first);
  __syncthreads();
  // The wall terms of the thread's cells in the state h: into the arrays that the launches of a stage each keep their sums in.
  auto walls = [&](const V* h_now) {
    for (int i = tid; i < cells; i += threads)
      if (s_wall[i] >= 0) {
        const int cell = (int)(first + i);
        const WallTerms<V> t = swe_step_wall<V>(h_now, params.wall_cell, params.bsx, params.bsy, s_wall[i], j_last, cell);
        params.acc_uh[cell] = t.uh; params.acc_vh[cell] = t.vh;
      }
  };
  walls(params.h);
  const KeptTile<G> tile{{s_val, s_val + a.edges, s_val + 2 * a.edges}, s_idx};
  const LdgTile<G> rest{&params};

#pragma unroll 1
  for (int k = 0; k < 4; ++k) {
    typename G::Params p = params;    // with the stage's states
    const bool even = (k & 1) == 0;
    if (k > 0) {
      p.h = even ? st.state[1][0] : st.state[0][0];
      p.uh = even ? st.state[1][1] : st.state[0][1];
      p.vh = even ? st.state[1][2] : st.state[0][2];
      all += kStepBarrier;
      step_arrive(a.header, withhold);
      walls(p.h);                     // of the thread's own cells, while the other CTAs arrive
      if (!step_wait(a.header, all, &s_ok)) return;
    }
    const SweRkCoef<V> coef = st.coef[k];
    V* const next[3] = {even ? st.state[0][0] : st.state[1][0], even ? st.state[0][1] : st.state[1][1], even ? st.state[0][2] : st.state[1][2]};
#pragma unroll 1
    for (int i = tid; i < cells; i += threads) {
      const long long row = first + i;
      const int lo = i ? s_end[i - 1] : 0, hi = s_end[i];
      // what the update reads of the cell itself travels with the gathers
      const V area = __ldg(p.area + row);
      const V at[3] = {p.x_h[row], p.x_uh[row], p.x_vh[row]};
      V wall[3] = {V(0), V(0), V(0)};
      if (s_wall[i] >= 0) { wall[1] = p.acc_uh[row]; wall[2] = p.acc_vh[row]; }
      typename G::GRow grow;
      G::template gather_row<false>(p, row, grow);
      V sum[3] = {V(0), V(0), V(0)};
#pragma unroll 1
      for (int e = lo; e < hi; ++e) {
        typename G::EReg er;
        typename G::GEdge ge;
        if (e < kept) G::load_edge(p, tile, e, e_first + e, er);
        else G::load_edge(p, rest, e_first + e, e_first + e, er);
        G::template gather_edge<false>(p, er, ge);
        G::map(p, er, e_first + e, grow, ge, sum);
      }
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        if (j > 0) sum[j] = fx::vadd(sum[j], wall[j]);
        const V d = fx::vdiv(-sum[j], area);
        V* const acc = s_sum + j * a.share + i;
        const V s = coef.first ? d : fx::vadd(*acc, d);
        if (coef.last) {
          (j == 0 ? p.x_h : (j == 1 ? p.x_uh : p.x_vh))[row] = fx::vadd(at[j], fx::vmul(coef.w, s));
        } else {
          *acc = s;
          next[j][row] = fx::vadd(at[j], fx::vmul(coef.c, d));
        }
      }
    }
  }
}

// Host side: what flexspmv_swe_delta_rk_T_step and _step_fits do (include/flexspmv.h).
template <class G, class Api>
struct StepApi {
  using V = typename G::V;
  static int fits(const flexspmv_desc* d) {
    StepShape<G> s;
    if (Api::check_desc(d) != 0 || !s.fit(d, device_sm_count())) return 0;
    return (d->offset_bits == 64 ? resident<long long>(s.more) : resident<int>(s.more)) ? (int)s.share : 0;
  }
  template <typename OffsetT>
  static auto kernel_of(bool more) {
    return more ? flex_swe_step_kernel<G, OffsetT, kStepMoreThreads> : flex_swe_step_kernel<G, OffsetT, kStepThreads>;
  }
  // Whether the device launches cooperatively and an SM holds the largest CTA (looked up once for each device of the process; 1 where
  // there is none to ask).
  template <typename OffsetT>
  static int resident(bool more) {
    constexpr int kMaxDevices = 64;
    static std::atomic<int> known[2][kMaxDevices];       // 0: not looked up yet, 1: yes, -1: no
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) { (void)cudaGetLastError(); return 1; }
    if (dev < 0 || dev >= kMaxDevices) return 0;
    int answer = known[more][dev].load(std::memory_order_acquire);
    if (answer == 0) {
      int cooperative = 0, ctas = 0;
      const auto kernel = kernel_of<OffsetT>(more);
      const bool held = cudaDeviceGetAttribute(&cooperative, cudaDevAttrCooperativeLaunch, dev) == cudaSuccess && cooperative &&
          cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kStepSmem) == cudaSuccess &&
          cudaOccupancyMaxActiveBlocksPerMultiprocessor(&ctas, kernel, more ? kStepMoreThreads : kStepThreads, kStepSmem) == cudaSuccess && ctas > 0;
      if (!held) (void)cudaGetLastError();
      answer = held ? 1 : -1;
      known[more][dev].store(answer, std::memory_order_release);
    }
    return answer > 0;
  }
  template <typename OffsetT>
  static int launch_as(const flexspmv_desc* d, const typename G::Params& p, const StepStages<V>& st, const void* row_offsets, void* ws, cudaStream_t stream) {
    StepShape<G> s;
    if (!s.fit(d, device_sm_count())) return FLEXSPMV_ERR_TOO_LARGE;
    const auto kernel = kernel_of<OffsetT>(s.more);
    if (cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kStepSmem); e != cudaSuccess) return (int)e;
    StepArgs a;
    a.row_offsets = row_offsets; a.header = static_cast<WorkspaceHeader*>(ws);
    a.num_rows = d->num_rows; a.num_edges = d->num_edges; a.num_tiles = Api::num_tiles(d);
    a.share = s.share; a.edges = (int)s.edges;
    note_kernel(FLEXSPMV_KERNEL_STEP);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)s.grid); cfg.blockDim = dim3((unsigned)s.threads); cfg.dynamicSmemBytes = s.bytes; cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;        // all CTAs at once: they wait for one another
    attr[0].val.cooperative = 1;
    cfg.attrs = attr; cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, p, st, a);
    if (e != cudaErrorCooperativeLaunchTooLarge) return (int)e;
    (void)cudaGetLastError();                 // the context has fewer SMs than the device: nothing was enqueued
    return FLEXSPMV_ERR_TOO_LARGE;
  }
  // What the launch writes lies apart from what other cells read meanwhile: the state that it advances, the two states in between and
  // the wall terms from one another, and from the state that the first stage gathers what that stage writes.
  static bool apart(long long cells, const void* const* values, void* const* outputs) {
    uintptr_t at[3 + 6 + 2];
    for (int i = 0; i < 6; ++i) at[i] = reinterpret_cast<uintptr_t>(outputs[i]);
    for (int i = 0; i < 2; ++i) at[6 + i] = reinterpret_cast<uintptr_t>(values[15 + i]);
    for (int i = 0; i < 3; ++i) at[8 + i] = reinterpret_cast<uintptr_t>(values[11 + i]);
    const uintptr_t bytes = (uintptr_t)cells * sizeof(V);
    auto meet = [&](uintptr_t a, uintptr_t b) { return (a > b ? a - b : b - a) < bytes; };
    for (int i = 0; i < 11; ++i)
      for (int j = 0; j < i; ++j)
        if (meet(at[i], at[j])) return false;
    for (int i = 0; i < 3; ++i)
      for (int j = 0; j < 8; ++j)
        if ((j < 3 || j >= 6) && meet(reinterpret_cast<uintptr_t>(values[3 + i]), at[j])) return false;
    return true;
  }
  static int launch(const flexspmv_desc* d, const void* const* values, const void* const* indices, const void* row_offsets, void* const* outputs,
                    void* ws, size_t ws_bytes, cudaStream_t stream) {
    if (int e = Api::check_desc(d)) return e;
    size_t need = 0;
    if (int e = Api::workspace_bytes(d, &need)) return e;
    if (!ws || ws_bytes < need) return FLEXSPMV_ERR_WORKSPACE;
    if (!values || !indices || !outputs || !row_offsets) return FLEXSPMV_ERR_BAD_ARG;
    for (int i = 0; i < G::kNumValues; ++i) if (!values[i]) return FLEXSPMV_ERR_BAD_ARG;
    for (int i = 0; i < G::kNumIndices; ++i) if (!indices[i]) return FLEXSPMV_ERR_BAD_ARG;
    for (int i = 0; i < 6; ++i) if (!outputs[i]) return FLEXSPMV_ERR_BAD_ARG;
    if (!apart(d->num_rows, values, outputs)) return FLEXSPMV_ERR_BAD_ARG;
    const typename G::Params p = G::make_params(values, indices, outputs);
    if (!G::pointers_aligned(p) || !aligned16(row_offsets)) return FLEXSPMV_ERR_ALIGN;
    StepStages<V> st;
    for (int i = 0; i < 6; ++i) st.state[i / 3][i % 3] = static_cast<V*>(outputs[i]);
    for (int k = 0; k < 4; ++k) st.coef[k] = SweRkCoef<V>::read(static_cast<const V*>(values[G::kNumValues - 1]) + 4 * k);
    if (d->offset_bits == 64) return launch_as<long long>(d, p, st, row_offsets, ws, stream);
    return launch_as<int>(d, p, st, row_offsets, ws, stream);
  }
};

}  // namespace flex

#define FLEXSPMV_DEFINE_STEP(SYM, GRAPH, CFG, CFGWIN, ...)                                                                 \
  extern "C" int flexspmv_##SYM##_step_fits(const flexspmv_desc* d) {                                                                  \
    return flex::StepApi<GRAPH, flex::GraphApi<GRAPH, CFG, CFGWIN, __VA_ARGS__>>::fits(d);                                          \
  }                                                                                                                                    \
  extern "C" int flexspmv_##SYM##_step(const flexspmv_desc* d, const void* const* v, const void* const* ix, const void* ro, void* const* o, \
                                       void* ws, size_t wb, void* st) {                                                                \
    return flex::StepApi<GRAPH, flex::GraphApi<GRAPH, CFG, CFGWIN, __VA_ARGS__>>::launch(d, v, ix, ro, o, ws, wb, static_cast<cudaStream_t>(st)); \
  }
