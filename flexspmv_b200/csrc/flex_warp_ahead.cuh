// The warp kernel (flex_warp_kernel.cuh: chunks, runs, marker bytes, carries) for launches of few chunks a warp.
//
// The warps of such a launch all start at once, and with the gathers at the head of their own chunk they wait and compute in
// step: on 200 003 power-law rows in fp64 the gathers alone take 11 us and the instructions 11 us, and the launch took the sum.
// Here a warp asks for the next chunk's gathers before it sums the present one, also from one run to the next, and fewer
// warps do the work (us, 4-byte values 1024 / 768 threads, 8-byte ones 768 / 640; power-law rows): fp64 200 003 30.8 / 27.5,
// 70 000 20.6 / 18.4, 500 000 51.8 / 50.1; fp32 100 000 24.7 / 20.7, 300 000 36.9 / 32.4, 500 000 48.3 / 45.5.  Launches of many
// chunks a warp drift apart by themselves and are bound by the gathers: 2^24 rows fp32 1227 / 1252, 4 M rows fp64 307 / 309.  They
// keep the other kernel.  The last CTA reads all CTAs' carries at once instead of one after the other.
#pragma once
#include <type_traits>

#include "flex_warp_kernel.cuh"

namespace flex {

template <class G, typename OffsetT, class Cfg>
__global__ void __launch_bounds__(Cfg::kBlock, Cfg::kMinCtas)
flex_warp_ahead_kernel(const typename G::Params p, const WarpKernelArgs a) {
  using V = typename G::V;
  constexpr int kAcc = G::kAccDim;
  constexpr int IPT = Cfg::kIpt, CH = Cfg::kChunk;
  static_assert(!G::kGatherNeedsRow, "the warp kernel takes graphs whose gathers all depend on the edge");

  extern __shared__ __align__(16) unsigned char smem_w[];
  __shared__ int s_last;
  __shared__ unsigned long long s_next;
  constexpr int kMaxRuns = WarpSmem<G, Cfg>::kMaxRuns;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  static_assert(CH <= 255, "row numbers inside a chunk are kept in marker bytes");
  static_assert(IPT <= 8, "a lane's markers are read as one 8-byte word");
  constexpr int kWarpBytes = WarpSmem<G, Cfg>::kBytes;
  unsigned char* wbase = smem_w + (size_t)warp * kWarpBytes;
  V* sp = reinterpret_cast<V*>(wbase);                                   // this warp's product slots, [kAcc][CH]
  // per item: the row (inside the chunk) whose last edge it is, or 0xff; the IPT items of a lane sit in one 8-byte word
  unsigned char* mk = wbase + (size_t)kAcc * CH * sizeof(V);
  const OffsetT* ro = static_cast<const OffsetT*>(a.row_offsets);
  const OffsetT* coords = static_cast<const OffsetT*>(a.coords);

  // launched while the kernel before it on the stream drains (see flex_tile_kernel.cuh): 200 003 power-law rows fp64,
  // back to back, 31.8 -> 30.2 us (medians of 25 runs in turn, quartiles 0.2 apart)
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

      // end of row x0 + lane relative to the chunk's first edge (rows past the chunk: unused)
      const OffsetT* ro0 = ro + x0 + 1;
      int rel_end = 0;
      if (lane < nr) rel_end = (int)(row_end - y0);
      reinterpret_cast<uint2*>(mk)[lane] = make_uint2(0xffffffffu, 0xffffffffu);
      __syncwarp();

      // rows that end inside the chunk, one lane per row: the last edge of a row is marked with the row's number;
      // a row without edges in this chunk is finished here (row x0 then takes the whole carry)
      const bool seed_used = __any_sync(0xffffffffu, lane == 0 && nr > 0 && rel_end == 0);
      int before = 0;                                      // where the row before this batch's first row ended
      for (int r0 = 0; r0 < nr; r0 += 32) {
        const int r = r0 + lane;
        if (r0) {
          before = __shfl_sync(0xffffffffu, rel_end, 31);
          rel_end = 0;
          if (r < nr) rel_end = (int)(ro0[r] - y0);
        }
        int prev = __shfl_up_sync(0xffffffffu, rel_end, 1);
        if (lane == 0) prev = before;
        if (r < nr) {
          if (rel_end > prev) {
            const int q = rel_end - 1, owner = q / IPT;
            mk[owner * 8 + (q - owner * IPT)] = (unsigned char)r;
          } else {
            static_for<G::kNumReducers>([&](auto R) {
              constexpr int d = G::template red_dim<R.value>();
              constexpr int o = G::template red_off<R.value>();
              V* dst = G::template red_out<R.value>(p) + (size_t)((long long)x0 + r) * d;
#pragma unroll
              for (int j = 0; j < d; ++j) dst[j] = (r == 0) ? carry[o + j] : V(0);
            });
          }
        }
      }
      if (seed_used) {
#pragma unroll
        for (int j = 0; j < kAcc; ++j) carry[j] = V(0);
      }

      // products into this warp's slots (lanes on consecutive edges; slots past the chunk's edges hold zero)
      typename G::GRow gr;
#pragma unroll
      for (int i = 0; i < IPT; ++i) {
        V prod[kAcc];
#pragma unroll
        for (int j = 0; j < kAcc; ++j) prod[j] = V(0);
        if (i * 32 + lane < ne) G::map(p, er[i], (long long)y0 + (i * 32 + lane), gr, ge[i], prod);
#pragma unroll
        for (int j = 0; j < kAcc; ++j) sp[j * CH + i * 32 + lane] = prod[j];
      }
      __syncwarp();

      // the next chunk's gathers, and the indices of the one after it
      if (nxt.run >= 0) {
#pragma unroll
        for (int i = 0; i < IPT; ++i) er[i] = er_next[i];
        start(nxt, er, ge);
        row_end = row_end_next;
        if (then.run >= 0) load_indices(then, er_next, row_end_next);
      }

      // blocked pass: every lane sums IPT consecutive items and closes the rows that end inside its span
      V run[kAcc], first[kAcc];
#pragma unroll
      for (int j = 0; j < kAcc; ++j) { run[j] = V(0); first[j] = V(0); }
      int first_row = -1;
      {
        V pv[IPT][kAcc];
        int pm[IPT];
        const uint2 mw = reinterpret_cast<const uint2*>(mk)[lane];
#pragma unroll
        for (int i = 0; i < IPT; ++i) {
          pm[i] = (int)(((i < 4 ? mw.x : mw.y) >> (8 * (i & 3))) & 0xffu);
#pragma unroll
          for (int j = 0; j < kAcc; ++j) pv[i][j] = sp[j * CH + lane * IPT + i];
        }
#pragma unroll
        for (int i = 0; i < IPT; ++i) {
#pragma unroll
          for (int j = 0; j < kAcc; ++j) run[j] += pv[i][j];
          if (pm[i] != 0xff) {
            if (first_row < 0) {                         // may have begun in earlier lanes: finished after the scan
              first_row = pm[i];
#pragma unroll
              for (int j = 0; j < kAcc; ++j) first[j] = run[j];
            } else {
              static_for<G::kNumReducers>([&](auto R) {
                constexpr int d = G::template red_dim<R.value>();
                constexpr int o = G::template red_off<R.value>();
                V* dst = G::template red_out<R.value>(p) + (size_t)((long long)x0 + pm[i]) * d;
#pragma unroll
                for (int j = 0; j < d; ++j) dst[j] = run[o + j];
              });
            }
#pragma unroll
            for (int j = 0; j < kAcc; ++j) run[j] = V(0);
          }
        }
      }
      // segmented inclusive scan of the open partial sums: a lane that closed a row passes on only what follows it.
      // Which lanes closed a row is one ballot; a lane takes a value from `d` lanes down only while that lane is not
      // before the nearest closing lane at or below it (lane 0 when there is none).
      const unsigned closed = __ballot_sync(0xffffffffu, first_row >= 0);
      const unsigned closed_le = closed & (0xffffffffu >> (31 - lane));
      const int reach = lane - (closed_le ? 31 - __clz(closed_le) : 0);      // lanes below this one in its segment
      V scan[kAcc];
#pragma unroll
      for (int j = 0; j < kAcc; ++j) scan[j] = run[j];
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
#pragma unroll
        for (int j = 0; j < kAcc; ++j) {
          const V v_up = shfl_up_any(scan[j], d);
          if (reach >= d) scan[j] = v_up + scan[j];
        }
      }
      // what the lanes before this one left open (plus the warp's carry when none of them closed a row)
      const bool f_ex = (closed_le & ~(1u << lane)) != 0;
      V in[kAcc];
#pragma unroll
      for (int j = 0; j < kAcc; ++j) {
        V v_ex = shfl_up_any(scan[j], 1);
        if (lane == 0) v_ex = V(0);
        in[j] = f_ex ? v_ex : carry[j] + v_ex;
      }
      if (first_row >= 0) {
        static_for<G::kNumReducers>([&](auto R) {
          constexpr int d = G::template red_dim<R.value>();
          constexpr int o = G::template red_off<R.value>();
          V* dst = G::template red_out<R.value>(p) + (size_t)((long long)x0 + first_row) * d;
#pragma unroll
          for (int j = 0; j < d; ++j) dst[j] = in[o + j] + first[o + j];
        });
      }
      // the warp's new carry: what is still open behind the last lane
      {
        const bool f31 = closed != 0;
#pragma unroll
        for (int j = 0; j < kAcc; ++j) {
          const V v31 = __shfl_sync(0xffffffffu, scan[j], 31);
          carry[j] = f31 ? v31 : carry[j] + v31;
        }
      }
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

  // ---- the CTA folds the carries of its runs; what its last run left open goes to the last CTA -------------------
  __syncthreads();
  {
    const int n_runs = (int)(s_next >> 32);
    const long long tail_row = n_runs ? (long long)s_run_row[n_runs - 1] : a.num_rows;
    for (int c = tid; c < n_runs; c += Cfg::kBlock) {
      const long long row = (long long)s_run_row[c];
      if (c > 0 && (long long)s_run_row[c - 1] == row) continue;     // not the first carry of its row
      V sum[kAcc];
#pragma unroll
      for (int i = 0; i < kAcc; ++i) sum[i] = s_run_val[c * kAcc + i];
      for (int c2 = c + 1; c2 < n_runs && (long long)s_run_row[c2] == row; ++c2) {
#pragma unroll
        for (int i = 0; i < kAcc; ++i) sum[i] += s_run_val[c2 * kAcc + i];
      }
      if (row == tail_row) {
        // still open at the end of the range (or no row at all): another CTA may finish it, so it waits for all of them
        V* cv = static_cast<V*>(a.carry_val) + (size_t)blockIdx.x * kAcc;
#pragma unroll
        for (int i = 0; i < kAcc; ++i) cv[i] = sum[i];
      } else {
        // finished by a later run of this CTA: every store to it is behind the barrier above
        static_for<G::kNumReducers>([&](auto R) {
          constexpr int d = G::template red_dim<R.value>();
          constexpr int o = G::template red_off<R.value>();
          V* dst = G::template red_out<R.value>(p) + (size_t)row * d;
#pragma unroll
          for (int i = 0; i < d; ++i) dst[i] = dst[i] + sum[o + i];
        });
      }
    }
    if (tid == 0) a.carry_row[blockIdx.x] = tail_row;
  }
  __threadfence();
  __syncthreads();
  if (tid == 0) {
    const unsigned t = atomicAdd(&a.header->ticket, 1u);
    s_last = (t == gridDim.x - 1) ? 1 : 0;
  }
  __syncthreads();
  if (s_last) {
    __threadfence();
    // all carries into shared memory first (nothing else is in use any more; the launch has no more CTAs than fit): a row that
    // spans many CTAs is added up there, not one round trip through L2 after the other
    const int n_carry = (int)gridDim.x;
    const V* cvals = static_cast<const V*>(a.carry_val);
    long long* s_row = reinterpret_cast<long long*>(smem_w);
    V* s_val = reinterpret_cast<V*>(s_row + n_carry);
    for (int c = tid; c < n_carry; c += Cfg::kBlock) {
      s_row[c] = __ldcg(a.carry_row + c);
#pragma unroll
      for (int i = 0; i < kAcc; ++i) s_val[(size_t)c * kAcc + i] = __ldcg(cvals + (size_t)c * kAcc + i);
    }
    __syncthreads();
    for (int c = tid; c < n_carry; c += Cfg::kBlock) {
      const long long row = s_row[c];
      if (row >= a.num_rows) continue;
      if (c > 0 && s_row[c - 1] == row) continue;   // not the head of its run
      V sum[kAcc];
#pragma unroll
      for (int i = 0; i < kAcc; ++i) sum[i] = s_val[(size_t)c * kAcc + i];
      for (int c2 = c + 1; c2 < n_carry && s_row[c2] == row; ++c2) {
#pragma unroll
        for (int i = 0; i < kAcc; ++i) sum[i] += s_val[(size_t)c2 * kAcc + i];
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
