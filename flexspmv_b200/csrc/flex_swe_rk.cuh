// What the shallow-water model does with a cell's three flux sums, as the epilogue of the kernel that forms them: the
// wall terms of boundary cells, d = -(r [+ wall]) / area and the Runge-Kutta update of the stage
// (shallow_water_equation/swe_main.py:86-146).  Every operation is the one, in the order, of the separate launches it
// stands for (the swe_boundary graph's pow / mul / sum and flexspmv_swe_rk_stage), so the states are bit-identical to
// theirs.  In the flux kernel the sums never leave their registers and the wall terms cost nothing on cells without a
// wall: per cell 16 bytes of memory traffic a sum, 32 a wall sum and two launches a stage less.
// Bound by the latency of the gathers and of the cell's own records (23 warps per SM at 80 registers, 57 % of DRAM); the
// producer warp therefore asks for those records in L2 when it stages a tile (prefetch_rows: 510 -> 454 us a step).  A step of
// the model on 2 097 152 cells, fp64: 606 us as 12 launches, 329 - 333 us as 4 (1024 x 1024 squares, one model replayed, three in turn 348; 369 in three CTAs of 9
// warps, GraphApi::use_big);
// on 20 402 cells 57.4 -> 23.8 us (30.8 with stages), as one launch (flex_swe_step.cuh) 20.5.
// fp64 batches of 1 / 2 edges per thread at 3 CTAs per SM, 3 at 2, 1 at 4 (before the prefetch): 510 / 546 / 625 / 555 us;
// fp32, 4 CTAs per SM, batches of 4 / 1: 327 / 286 us.
#pragma once
#include "flex_tensor.cuh"

namespace flex {

// The records of `cell` among j0 .. j1-1, added in order.  Out of line: few cells have a wall.  The first one is bisected: a
// group of 32 cells may hold many records (a thin mesh, several walls a cell), and one lane after the other would walk them
// all (2 097 152 cells, a step: one record on every cell 704 -> 556 us, three on every cell 1300 -> 652; three launches a
// stage 594 and 624.  Cells beside the rim no longer pay for pow: 20 402 cells 32.9 -> 30.8 us).
template <typename V>
struct WallTerms { V uh, vh; };
template <typename V>
__device__ __noinline__ WallTerms<V> swe_wall_terms(const V* h, const int* wall_cell, const V* bsx, const V* bsy, int j0, int j1, int cell) {
  WallTerms<V> t{V(0), V(0)};
  const int end = j1;
  while (j0 < j1) {
    const int mid = (j0 + j1) >> 1;
    if (__ldg(wall_cell + mid) < cell) j0 = mid + 1; else j1 = mid;
  }
  if (j0 >= end || __ldg(wall_cell + j0) != cell) return t;
  const V half_sq = fx::vmul(V(0.5), fx::vpow(__ldg(h + cell), V(2)));
  do {
    t.uh = fx::vadd(t.uh, fx::vmul(half_sq, __ldg(bsx + j0)));
    t.vh = fx::vadd(t.vh, fx::vmul(half_sq, __ldg(bsy + j0)));
  } while (++j0 < end && __ldg(wall_cell + j0) == cell);
  return t;
}

// P: Params of a generated graph with the fields named below.  `coef` points to host memory that is read when the
// launch is made: c, w, first, last.  Records of the walls: wall_cell ascending, wall_start[i] = first record of a cell
// >= 32 i (cells / 32 rounded up, plus one, entries).
// What the update reads of the cell itself is asked for in one go, in front of its first store: a load behind a store to another
// array waits for it, and the three sums took a round trip each (2 097 152 cells, fp64: 383 -> 368 us a step, 540 800 131 -> 121,
// 20 402 24.9 -> 23.8; asked for before the edges instead, 7 doubles more in registers meanwhile: 405, 135 and 24.6).
template <typename V>
struct SweRkOwn { V area, at[3], a[3]; int j0, j1; };      // at: the state, a: the running sums; j0, j1: the records of the cell's group of 32
template <typename V, class P>
__device__ __forceinline__ void swe_rk_load(const P& p, long long row, SweRkOwn<V>& o) {
  o.area = __ldg(p.area + row);
  o.j0 = __ldg(p.wall_start + (row >> 5)); o.j1 = __ldg(p.wall_start + (row >> 5) + 1);
  V* const x[3] = {p.x_h, p.x_uh, p.x_vh};
  V* const acc[3] = {p.acc_h, p.acc_uh, p.acc_vh};
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    o.at[k] = x[k][row];
    o.a[k] = p.coef.first ? V(0) : acc[k][row];
  }
}
template <typename V, class P>
__device__ __forceinline__ void swe_rk_row(const P& p, long long row, const V* r, const SweRkOwn<V>& o) {
  V* const x[3] = {p.x_h, p.x_uh, p.x_vh};
  V* const acc[3] = {p.acc_h, p.acc_uh, p.acc_vh};
  V* const next[3] = {p.out_r_h, p.out_r_uh, p.out_r_vh};
  // (copies, not the members: 80 bytes spilled in the kernel without stages, 116 with them)
  const V area = o.area;
  const int j0 = o.j0, j1 = o.j1;
  V at[3] = {o.at[0], o.at[1], o.at[2]}, a[3] = {o.a[0], o.a[1], o.a[2]};
  WallTerms<V> wall{V(0), V(0)};
  if (j0 < j1) wall = swe_wall_terms<V>(p.h, p.wall_cell, p.bsx, p.bsy, j0, j1, (int)row);
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    V sum = r[k];
    if (k > 0) sum = fx::vadd(sum, k == 1 ? wall.uh : wall.vh);
    const V d = fx::vdiv(-sum, area);
    a[k] = p.coef.first ? d : fx::vadd(a[k], d);
    if (p.coef.last) {
      x[k][row] = fx::vadd(at[k], fx::vmul(p.coef.w, a[k]));
    } else {
      acc[k][row] = a[k];
      next[k][row] = fx::vadd(at[k], fx::vmul(p.coef.c, d));
    }
  }
}

template <typename V>
struct SweRkCoef {
  V c, w;
  bool first, last;
  static SweRkCoef read(const void* host) {
    const V* v = static_cast<const V*>(host);
    return SweRkCoef{v[0], v[1], v[2] != V(0), v[3] != V(0)};
  }
};

}  // namespace flex
