// The warp kernel (flex_warp_kernel.cuh: chunks, runs, marker bytes, carries) for launches of few chunks a warp.
//
// The warps of such a launch all start at once, and with the gathers at the head of their own chunk they wait and compute in
// step: on 200 003 power-law rows in fp64 the gathers alone take 11 us and the instructions 11 us, and the launch took the sum.
// Here a warp asks for the next chunk's gathers before it sums the present one, also from one run to the next, and fewer
// warps do the work (us, 4-byte values 1024 / 768 threads, 8-byte ones 768 / 640; power-law rows): fp64 200 003 30.8 / 27.4,
// 70 000 20.6 / 18.4, 500 000 51.8 / 48.3; fp32 100 000 24.9 / 20.7, 300 000 36.5 / 32.1, 500 000 48.0 / 45.4, 700 000 60.8 / 55.7.  Launches
// of many chunks a warp drift apart by themselves and are bound by the gathers: 2^24 rows fp32 1227 / 1252, 4 M rows fp64 307 / 309.
// They keep the other form (the line: GraphApi::launch_lean).  What is done with a chunk and with the carries is the same (WarpParts).
#pragma once
#include <type_traits>

#include "flex_warp_kernel.cuh"

namespace flex {

template <class G, typename OffsetT, class Cfg>
__global__ void __launch_bounds__(Cfg::kBlock, Cfg::kMinCtas)
flex_warp_ahead_kernel(const typename G::Params p, const WarpKernelArgs a) {
  using V = typename G::V;
  using W = WarpParts<G, OffsetT, Cfg>;
  constexpr int kAcc = G::kAccDim;
  constexpr int IPT = Cfg::kIpt, CH = Cfg::kChunk;
  static_assert(!G::kGatherNeedsRow, "the warp kernel takes graphs whose gathers all depend on the edge");

  extern __shared__ __align__(16) unsigned char smem_w[];
  __shared__ unsigned long long s_next;
  constexpr int kMaxRuns = WarpSmem<G, Cfg>::kMaxRuns;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int kWarpBytes = WarpSmem<G, Cfg>::kBytes;
  unsigned char* wbase = smem_w + (size_t)warp * kWarpBytes;
  V* sp = reinterpret_cast<V*>(wbase);                                   // this warp's product slots, [kAcc][CH]
  // per item: the row (inside the chunk) whose last edge it is, or 0xff; the IPT items of a lane sit in one 8-byte word
  unsigned char* mk = wbase + (size_t)kAcc * CH * sizeof(V);
  const OffsetT* ro = static_cast<const OffsetT*>(a.row_offsets);
  const OffsetT* coords = static_cast<const OffsetT*>(a.coords);

  // launched while the kernel before it on the stream drains, as the other form is
  pdl_wait();
  pdl_launch_dependents();
  if (a.header->magic != kMagic || a.header->num_tiles != a.num_chunks || a.header->num_rows != a.num_rows ||
      a.header->num_edges != a.num_edges || a.header->offset_bits != (int)(8 * sizeof(OffsetT))) {
    if (tid == 0 && blockIdx.x == 0) raise_not_planned(a.header);
    return;
  }

  // The CTA owns a contiguous range of chunks.  Its warps take runs of consecutive chunks from it one after the other
  // (s_next: next free chunk of the range in the low half, runs handed out so far in the high half).  A run is
  // 1/kWarps of what is left, at least min_run chunks: long runs first, short ones at the end, so that the warps of
  // the CTA finish together whatever their speeds were.  The sequence of runs depends only on the range, not on
  // which warp takes which, so results stay the same from launch to launch.
  const long long q = a.num_chunks / gridDim.x, rem = a.num_chunks % gridDim.x;
  const long long cta_begin = (long long)blockIdx.x * q + (blockIdx.x < rem ? blockIdx.x : rem);
  const unsigned cta_chunks = (unsigned)(q + (blockIdx.x < rem ? 1 : 0));
  OffsetT* s_run_row = reinterpret_cast<OffsetT*>(smem_w + (size_t)Cfg::kWarps * kWarpBytes);   // [kMaxRuns] row a run left open
  V* s_run_val = reinterpret_cast<V*>(s_run_row + kMaxRuns);                                     // [kMaxRuns][kAcc] its partial sums
  const unsigned min_run = cta_chunks >= 16u * Cfg::kWarps ? 4u : 1u;     // a run pays for one pipeline start
  if (tid == 0) s_next = 0ull;
  __syncthreads();

  StreamTile<G> tile{&p};
  // The warp's chunks in the order it takes them, across its runs; requests go out ahead of the work: a chunk's boundaries
  // two chunks ahead, its indices and row ends one chunk ahead, and its gathers and values before the chunk in front of it
  // is summed.
  struct Ahead { OffsetT x0, y0, x1, y1; int run; };        // boundaries of a chunk and its run (-1: no more chunks)
  unsigned run_at = 0, run_left = 0;                        // what is left of the run taken last
  int run_id = -1;
  auto next_chunk = [&](const Ahead& last) -> Ahead {       // `last`: the chunk taken before
    const bool goes_on = run_left != 0;
    if (!goes_on) {
      unsigned pos = 0, len = 0, id = 0;
      if (lane == 0) {
        unsigned long long seen = *reinterpret_cast<volatile unsigned long long*>(&s_next);
        for (;;) {
          pos = (unsigned)seen; id = (unsigned)(seen >> 32);
          if (pos >= cta_chunks) { len = 0; break; }
          const unsigned left = cta_chunks - pos;
          len = left / Cfg::kWarps;
          if (len < min_run) len = min_run;
          if (len > left || id == (unsigned)kMaxRuns - 1) len = left;
          const unsigned long long want = ((unsigned long long)(id + 1) << 32) | (pos + len);
          const unsigned long long got = atomicCAS(&s_next, seen, want);
          if (got == seen) break;
          seen = got;
        }
      }
      run_at = __shfl_sync(0xffffffffu, pos, 0);
      run_left = __shfl_sync(0xffffffffu, len, 0);
      run_id = (int)__shfl_sync(0xffffffffu, id, 0);
      if (run_left == 0) run_id = -1;
    }
    Ahead c{0, 0, 0, 0, run_id};
    if (run_id >= 0) {
      // every lane reads the same pair (one broadcast transaction, no shuffles); inside a run a chunk begins where the one
      // before it ends
      using Pair = std::conditional_t<sizeof(OffsetT) == 4, int2, longlong2>;
      const Pair* at = reinterpret_cast<const Pair*>(coords) + (cta_begin + run_at);
      if (goes_on) {
        c.x0 = last.x1; c.y0 = last.y1;
      } else {
        const Pair u = __ldg(at);
        c.x0 = u.x; c.y0 = u.y;
      }
      const Pair w = __ldg(at + 1);
      c.x1 = w.x; c.y1 = w.y;
      ++run_at;
      --run_left;
    }
    return c;
  };
  // indices of one chunk into registers (lanes on consecutive edges), and the end of row x0 + lane (the first 32 rows that
  // end inside the chunk)
  auto load_indices = [&](const Ahead& c, typename G::EReg (&er)[IPT], OffsetT& row_end) {
    const int ne = (int)(c.y1 - c.y0);
    const long long e0 = (long long)c.y0 + lane;
#pragma unroll
    for (int i = 0; i < IPT; ++i)
      if (i * 32 + lane < ne) {
        G::load_edge_idx(tile, e0 + i * 32, er[i]);
      }
    row_end = 0;
    if (lane < (int)(c.x1 - c.x0)) row_end = ro[(long long)c.x0 + 1 + lane];
  };
  auto start = [&](const Ahead& c, typename G::EReg (&er)[IPT], typename G::GEdge (&ge)[IPT]) {
    const int ne = (int)(c.y1 - c.y0);
    const long long e0 = (long long)c.y0 + lane;
#pragma unroll
    for (int i = 0; i < IPT; ++i)
      if (i * 32 + lane < ne) {
        G::gather_edge(p, er[i], ge[i]);
        G::load_edge_vals(p, tile, e0 + i * 32, e0 + i * 32, er[i]);
      }
  };

  Ahead cur = next_chunk(Ahead{0, 0, 0, 0, -1});
  if (cur.run >= 0) {
    Ahead nxt = next_chunk(cur);
    typename G::EReg er[IPT], er_next[IPT];
    typename G::GEdge ge[IPT];
    OffsetT row_end = 0, row_end_next = 0;
    load_indices(cur, er, row_end);
    if (nxt.run >= 0) load_indices(nxt, er_next, row_end_next);
    start(cur, er, ge);
    V carry[kAcc];
#pragma unroll
    for (int j = 0; j < kAcc; ++j) carry[j] = V(0);

    for (;;) {
      const Ahead then = nxt.run >= 0 ? next_chunk(nxt) : Ahead{0, 0, 0, 0, -1};
      const OffsetT x0 = cur.x0, y0 = cur.y0;
      const int ne = (int)(cur.y1 - y0), nr = (int)(cur.x1 - x0);

      W::mark_rows(p, ro, x0, y0, nr, row_end, mk, lane, carry);
      W::products(p, y0, ne, er, ge, sp, lane);

      // the next chunk's gathers, and the indices of the one after it
      if (nxt.run >= 0) {
#pragma unroll
        for (int i = 0; i < IPT; ++i) er[i] = er_next[i];
        start(nxt, er, ge);
        row_end = row_end_next;
        if (then.run >= 0) load_indices(then, er_next, row_end_next);
      }

      W::close_rows(p, x0, sp, mk, lane, carry);
      __syncwarp();                                      // the slots are rewritten by the next chunk
      if (nxt.run != cur.run) {
        // the run's carry: the row it left open and the partial sums of that row
        if (lane == 0) {
          s_run_row[cur.run] = cur.x1;
#pragma unroll
          for (int j = 0; j < kAcc; ++j) s_run_val[cur.run * kAcc + j] = carry[j];
        }
        if (nxt.run < 0) break;
#pragma unroll
        for (int j = 0; j < kAcc; ++j) carry[j] = V(0);
      }
      cur = nxt;
      nxt = then;
    }
  }

  __syncthreads();
  W::template fold_carries<true>(p, a, smem_w, (int)(s_next >> 32), s_run_row, s_run_val);
}

}  // namespace flex
