"""The tile kernel's loop over whole rows: which matrices the plan sends there (short rows that every tile can hold
whole), and its results against the CPU oracle at the edges -- rows of 0, 1, a batch, a batch more, 32 and 33 edges,
tiles smaller than a row, one row, both offset widths -- and against the loop with carries."""
import ctypes

import numpy as np
import pytest
import torch

from flexspmv_b200 import graphs, problems
from flexspmv_b200.codegen import emit_cuda
from flexspmv_b200.binding import Desc, FlexSpmvError, GraphExtension, load_library
from oracle import ir_eval
from parity import assert_outputs_match
from test_gpu_parity import run_gpu

pytestmark = pytest.mark.gpu


def with_lengths(ir, lengths, seed, dtype):
    """A random problem of the given row lengths."""
    lengths = np.asarray(lengths)
    rows, nnz = lengths.size, int(lengths.sum())
    prob = problems.random_problem(ir, rows, rows, nnz, seed=seed, dtype=dtype)
    prob.row_offsets = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)
    for s in ir.selector_register:
        if s.get("row_identity"):
            prob.indices[s["selector_name"]] = np.repeat(np.arange(rows, dtype=np.int32), lengths)
    return prob


LENGTHS = {
    "empty_and_full": ([0, 32, 0, 31, 1, 32, 32] * 300 + [0] * 5, None),   # at the limit: depends on the rows a tile holds
    "all_5": ([5] * 4001, 1),
    "all_8": ([8] * 3000, 1),
    "batch_and_one_more": ([4, 5] * 1500 + [9] * 7, 1),
    "all_32": ([32] * 777, 1),
    "a_row_of_33": ([8] * 1000 + [33] + [8] * 1000, -1),
    "one_row": ([7], 0),                                                  # one lane of a warp
    "uneven": ([1] * 310 + [32] * 10 + [1] * 3000, 1),
    "mostly_empty": (([0] * 31 + [32]) * 100, 0),                         # one lane in 32 would work
    "leading_and_trailing_empty": ([0] * 100 + [6] * 500 + [0] * 100, 1),
}


@pytest.mark.parametrize("gname,dt", [("spmv", "float64"), ("spmv", "float32"), ("spmv", "int64"), ("spring_mass", "float32"),
                                      ("rusanov", "float64"), ("swe_delta", "float32"), ("ops_zoo", "float64")])
@pytest.mark.parametrize("case", sorted(LENGTHS))
def test_whole_rows_match_the_oracle(gname, dt, case):
    ir, dtype = graphs.ALL_GRAPHS[gname](), np.dtype(dt)
    lengths, planned = LENGTHS[case]
    prob = with_lengths(ir, lengths, 7, dtype)
    ref, _, sums = ir_eval.run_graph(ir, prob, dtype, num_threads=4, want_abs_sums=True)
    for kw, offsets in (({}, np.int32), ({}, np.int64), ({"tile_items": 5, "max_ctas": 3}, np.int32),
                        ({"tile_items": 40, "max_ctas": 7}, np.int64), ({"max_ctas": 1}, np.int32)):
        ext = GraphExtension(ir, random_gather=False, **kw)
        got, _ = run_gpu(ext, ir, prob, dtype, offsets_dtype=offsets)
        assert_outputs_match(ir, got, ref, sums, dtype, what=f"{gname}/{dt}/{case}/{kw}")
        ext.check()
        # tiles of a few rows leave most lanes of a warp idle: refused; the small tiles of other graphs have no room for
        # the front of a 32-edge row
        if planned is not None and "tile_items" not in kw and (case != "all_32" or gname == "spmv"):
            assert ext.planned_whole_rows() == (planned == 1), (case, kw)


def row_loop_planned(ext):
    """Whether the last plan chose the loop over whole rows (workspace header, int32 at byte 156)."""
    return int(next(reversed(ext._plans.values())).ws[:256].cpu().numpy().view(np.int32)[39])


@pytest.mark.parametrize("gname,dt,lengths,expected", [
    ("spmv", "float64", [3, 8, 5] * 2000 + [32] * 50, 1), ("rusanov", "float64", [3, 8, 5] * 2000 + [32] * 50, 1),
    ("swe_boundary", "float32", [3, 8, 5] * 2000 + [32] * 50, 1), ("ops_zoo", "float64", [3, 8, 5] * 2000 + [32] * 50, 0),
    ("ops_zoo", "float32", [3, 8, 5] * 2000 + [32] * 50, 0), ("ops_zoo", "float64", [4, 6] * 4000, 0), ("ops_zoo", "float32", [0, 8] * 4000, 0),
    ("ops_zoo", "float64", [7] * 9000, 1), ("ops_zoo", "float32", [3] * 9000, 1)])
def test_maps_that_divide_keep_the_two_phase_loop(gname, dt, lengths, expected):
    """A two-phase graph whose map takes tens of instructions an edge: its tiles hold whole rows, so no grid hands carries
    over, but lanes stay on consecutive edges unless every lane has a row of about the same few edges."""
    ir, dtype = graphs.ALL_GRAPHS[gname](), np.dtype(dt)
    prob = with_lengths(ir, lengths, 29, dtype)
    ref, _, sums = ir_eval.run_graph(ir, prob, dtype, num_threads=4, want_abs_sums=True)
    results = []
    for max_ctas in (0, 1, 7, 50):
        ext = GraphExtension(ir, random_gather=False, max_ctas=max_ctas)
        got, _ = run_gpu(ext, ir, prob, dtype)
        ext.check()
        assert_outputs_match(ir, got, ref, sums, dtype, what=f"{gname} {max_ctas}")
        assert ext.planned_whole_rows() and row_loop_planned(ext) == expected
        results.append(got)
    for got in results[1:]:                    # no carries: the grid changes no bit
        assert all(np.array_equal(a, b, equal_nan=True) for a, b in zip(got, results[0]))


@pytest.mark.parametrize("gname,dt", [("spmv", "float64"), ("spmv", "float32"), ("spmv", "int64"), ("spring_mass", "float32")])
@pytest.mark.parametrize("lengths,same_bank", [([8] * 3000, 0), ([16] * 3000, 1), ([24] * 2000, 0), ([32] * 1500, 1), ([31] * 1500, 0),
                                               ([16, 0] * 2500, 0), ([0] * 31 + [32] * 997 + [0] * 400, 1), ([7, 9] * 2000, 0), ([15, 16] * 1000, 0)])
def test_rows_that_begin_in_one_bank_keep_lanes_on_consecutive_edges(gname, dt, lengths, same_bank):
    """Rows of 16 or 32 edges all begin in two shared-memory banks or in one: graphs whose other loop walks consecutive edges
    take that one on the tiles of whole rows; graphs with per-row data have a thread per row in both."""
    ir, dtype = graphs.ALL_GRAPHS[gname](), np.dtype(dt)
    prob = with_lengths(ir, lengths, 31, dtype)
    ref, _, sums = ir_eval.run_graph(ir, prob, dtype, num_threads=4, want_abs_sums=True)
    for kw, offsets in (({}, np.int32), ({"max_ctas": 2}, np.int64)):
        ext = GraphExtension(ir, random_gather=False, **kw)
        got, _ = run_gpu(ext, ir, prob, dtype, offsets_dtype=offsets)
        ext.check()
        assert_outputs_match(ir, got, ref, sums, dtype, what=f"{gname} {dt} {lengths[:3]} {kw}")
        assert ext.planned_whole_rows()
        assert row_loop_planned(ext) == (1 if gname == "spring_mass" else 1 - same_bank)


def with_columns(ir, prob, kind, seed):
    """Columns of a matrix: consecutive ones from an arbitrary start per row ("runs"), consecutive rows side by side
    ("stencil"), the first half of the rows one way and the second half the other ("both"), anywhere ("random")."""
    rng = np.random.default_rng(seed)
    lengths = np.diff(prob.row_offsets)
    n, own = lengths.size, np.repeat(np.arange(lengths.size), lengths)
    place = np.arange(own.size) - prob.row_offsets[own]
    runs = rng.integers(0, n, n)[own] + place
    stencil = own + 50 * place
    cols = {"runs": runs, "stencil": stencil, "both": np.where(own < n // 2, stencil, runs), "random": rng.integers(0, n, own.size)}[kind]
    for k in prob.indices:
        prob.indices[k] = (cols % n).astype(np.int32)
    return prob


@pytest.mark.parametrize("dt", ["float64", "float32", "int64"])
@pytest.mark.parametrize("kind,row_loop", [("runs", 0), ("stencil", 1), ("both", None), ("random", 1)])
@pytest.mark.parametrize("lengths", [[20] * 2500, [9] * 9000, [0, 9, 3, 12] * 1500, [3] * 40, [7] * 9])
def test_either_loop_on_whole_rows_gives_the_same_bits(dt, kind, row_loop, lengths):
    """The plan looks at a sample of the columns and leaves rows that are runs of columns on the two-phase loop, whose lanes
    walk consecutive edges.  Whichever loop runs, on whatever grid, a row is its products from left to right: the bits of the
    loop with carries on one CTA (the same matrix with a row of 33 edges behind it)."""
    ir, dtype = graphs.spmv_graph(), np.dtype(dt)
    n = len(lengths)
    prob = with_columns(ir, with_lengths(ir, lengths, 37, dtype), kind, 41)
    carry = with_lengths(ir, lengths + [33], 37, dtype)
    carry.values["vals"][:prob.nnz], carry.values["x"][:n] = prob.values["vals"], prob.values["x"]
    carry.indices["selector"][:prob.nnz] = prob.indices["selector"]
    ext = GraphExtension(ir, random_gather=False, max_ctas=1)
    want, _ = run_gpu(ext, ir, carry, dtype)
    assert not ext.planned_whole_rows()
    for kw, offsets in (({}, np.int32), ({}, np.int64), ({"max_ctas": 1}, np.int32), ({"max_ctas": 2}, np.int64), ({"max_ctas": 7}, np.int32),
                        ({"tile_items": 200, "max_ctas": 3}, np.int32)):
        ext = GraphExtension(ir, random_gather=False, **kw)
        got, _ = run_gpu(ext, ir, prob, dtype, offsets_dtype=offsets)
        ext.check()
        assert ext.planned_whole_rows() or "tile_items" in kw or n < 32
        if not kw and n > 1000 and row_loop is not None:
            assert row_loop_planned(ext) == row_loop
        assert np.array_equal(got[0], want[0][:n]), (kw, offsets)


def test_a_plan_that_has_not_seen_the_columns_goes_by_the_rows():
    """flexspmv_G_plan and flexspmv_G_plan_indexed differ in the loop they choose for runs of columns and in nothing else; the
    sample reads no column of matrices whose offsets lead outside of the arrays."""
    lib = load_library()
    ir, dtype = graphs.spmv_graph(), np.float64
    prob = with_columns(ir, with_lengths(ir, [12] * 4000, 53, dtype), "runs", 59)
    cols, ro = (torch.from_numpy(a).cuda() for a in (prob.indices["selector"], prob.row_offsets.astype(np.int64)))
    for name in ("workspace_bytes", "plan", "plan_indexed"):
        getattr(lib, f"flexspmv_spmv_f64_{name}").restype = ctypes.c_int
    desc = Desc(prob.num_rows, prob.nnz, prob.num_cols, 64, 0, 0, 0)
    nbytes = ctypes.c_size_t()
    assert lib.flexspmv_spmv_f64_workspace_bytes(ctypes.byref(desc), ctypes.byref(nbytes)) == 0
    ix = (ctypes.c_void_p * 1)(cols.data_ptr())
    none = (ctypes.c_void_p * 1)(None)

    def planned(indexed, offsets):
        ws = torch.zeros(nbytes.value, dtype=torch.uint8, device="cuda")
        args = [ctypes.c_void_p(offsets.data_ptr()), ctypes.c_void_p(ws.data_ptr()), nbytes, None]
        if indexed:
            assert lib.flexspmv_spmv_f64_plan_indexed(ctypes.byref(desc), ix, *args) == 0
        else:
            assert lib.flexspmv_spmv_f64_plan(ctypes.byref(desc), *args) == 0
        torch.cuda.synchronize()
        header = ws[:256].cpu().numpy().view(np.int32)
        tiles = -(-(prob.num_rows + prob.nnz) // 1280)
        return header[38:40].tolist(), ws[256:256 + 16 * (tiles + 1)].cpu()

    (by_rows, coords), (by_columns, same) = planned(False, ro), planned(True, ro)
    assert by_rows == [1, 1] and by_columns == [1, 0] and torch.equal(coords, same)
    for wrong in (ro - 40, ro + 10 ** 9, ro.flip(0).contiguous(), ro * 1000):
        assert planned(True, wrong)[0] == [-1, 0]
    # no index arrays
    ws = torch.zeros(nbytes.value, dtype=torch.uint8, device="cuda")
    args = [ctypes.c_void_p(ro.data_ptr()), ctypes.c_void_p(ws.data_ptr()), nbytes, None]
    assert lib.flexspmv_spmv_f64_plan_indexed(ctypes.byref(desc), None, *args) == -1
    assert lib.flexspmv_spmv_f64_plan_indexed(ctypes.byref(desc), none, *args) == -1


@pytest.mark.parametrize("gname,dt,kind", [("spmv", "float64", "runs"), ("spmv", "float64", "stencil"), ("spring_mass", "float32", None),
                                           ("ops_zoo", "float64", None)])
def test_bounded_wait_runs_out_on_tiles_of_whole_rows(gname, dt, kind):
    """A stage that is never filled, on matrices of short rows: the consumers of either loop give up after their bounded wait,
    the status says so, and a fresh plan gives the full result."""
    lib = load_library()
    lib.flexspmv_debug_withhold_stage.restype = ctypes.c_int
    ir, dtype = graphs.ALL_GRAPHS[gname](), np.dtype(dt)
    prob = with_lengths(ir, [9] * 3000, 43, dtype)
    if kind:
        prob = with_columns(ir, prob, kind, 47)
    ref, _, sums = ir_eval.run_graph(ir, prob, dtype, num_threads=4, want_abs_sums=True)
    for withhold in (1, 2, 6):
        ext = GraphExtension(ir, random_gather=False, max_ctas=2)
        non_gather, gathers, index_names = graphs.operator_signature(ir)
        v = [torch.from_numpy(np.ascontiguousarray(prob.values[n])).cuda() for n in non_gather + gathers]
        ix = [torch.from_numpy(prob.indices[n]).cuda() for n in index_names]
        ro = torch.from_numpy(prob.row_offsets).cuda()
        outs = [torch.full(o.shape, float("nan"), dtype=v[0].dtype, device="cuda") for o in map(torch.from_numpy, ref)]
        ext.prepare(v, ix, ro, outs, prob.num_rows, prob.nnz, prob.num_cols)
        assert ext.planned_whole_rows()
        ws = next(reversed(ext._plans.values())).ws
        assert lib.flexspmv_debug_withhold_stage(ctypes.c_void_p(ws.data_ptr()), ctypes.c_uint32(withhold), None) == 0
        ext.launch_into(v, ix, ro, outs, prob.num_rows, prob.nnz, prob.num_cols)
        with pytest.raises(FlexSpmvError, match="bounded device-side wait"):
            ext.check()
        again = GraphExtension(ir, random_gather=False, max_ctas=2)
        got, _ = run_gpu(again, ir, prob, dtype)
        again.check()
        assert_outputs_match(ir, got, ref, sums, dtype, what=f"{gname} after a wait ran out")


def test_whole_rows_equal_the_two_phase_loop_bit_for_bit():
    """The same matrix with one row of 33 edges behind it goes through the loop with carries; all other rows are the
    same sums, left to right."""
    ir = graphs.spmv_graph()
    rng = np.random.default_rng(3)
    lengths = rng.integers(0, 17, 5000)
    a = with_lengths(ir, lengths, 11, np.float64)
    b = with_lengths(ir, np.concatenate([lengths, [33]]), 11, np.float64)
    n, nnz = a.num_rows, a.nnz
    b.values["vals"][:nnz] = a.values["vals"]
    b.values["x"][:n] = a.values["x"]
    b.indices["selector"][:nnz] = a.indices["selector"]
    whole, carry = GraphExtension(ir, max_ctas=1), GraphExtension(ir, max_ctas=1)
    got_a, _ = run_gpu(whole, ir, a, np.float64)
    got_b, _ = run_gpu(carry, ir, b, np.float64)
    assert whole.planned_whole_rows() and not carry.planned_whole_rows()
    assert np.array_equal(got_a[0], got_b[0][:n])


@pytest.mark.parametrize("bits", [32, 64])
def test_a_moved_boundary_never_overfills_a_stage(bits):
    """Many rows of one edge behind a long row that a boundary between two CTAs cuts: with the cut part moved behind
    the boundary the tile's records and row ends would take more bytes than its stage holds, so the plan must leave
    the boundaries alone (header, int32 at byte 132)."""
    ir, dtype = graphs.spmv_graph(), np.float64
    tile = 1280
    lengths = np.ones(40 * tile, dtype=np.int64)
    # rows in front of the second tile's boundary: the cut row has 600 edges in front of it and ends in the second tile
    lengths[(tile - 600) // 2] = 601
    prob = with_lengths(ir, lengths, 13, dtype)
    ref, _, sums = ir_eval.run_graph(ir, prob, dtype, num_threads=4, want_abs_sums=True)
    lib = load_library()
    desc = Desc(prob.num_rows, prob.nnz, prob.num_cols, bits, 0, 0, 0)
    nbytes = ctypes.c_size_t()
    for name in ("workspace_bytes", "plan", "launch"):
        getattr(lib, f"flexspmv_spmv_f64_{name}").restype = ctypes.c_int
    assert lib.flexspmv_spmv_f64_workspace_bytes(ctypes.byref(desc), ctypes.byref(nbytes)) == 0
    ws = torch.zeros(nbytes.value, dtype=torch.uint8, device="cuda")
    ro = torch.from_numpy(prob.row_offsets.astype(np.int32 if bits == 32 else np.int64)).cuda()
    assert lib.flexspmv_spmv_f64_plan(ctypes.byref(desc), ctypes.c_void_p(ro.data_ptr()), ctypes.c_void_p(ws.data_ptr()),
                                      ctypes.c_size_t(nbytes.value), None) == 0
    torch.cuda.synchronize()
    raw = ws[:256].cpu().numpy().view(np.int32)
    coords = ws[256:256 + 48].cpu().numpy().view(np.int32 if bits == 32 else np.int64)
    rows_behind, begin = int(coords[4] - coords[2]), int(prob.row_offsets[coords[2]])
    extra = int(coords[3]) - begin
    assert 0 < extra <= rows_behind                                  # the row count alone would have allowed it ...
    assert (int(coords[5]) - begin) * 12 + rows_behind * bits // 8 > tile * 12 + 32 * 12     # ... the bytes do not
    assert raw[33] == 0
    got, _ = run_gpu(GraphExtension(ir), ir, prob, dtype, offsets_dtype=np.int32 if bits == 32 else np.int64)
    assert_outputs_match(ir, got, ref, sums, np.dtype(dtype), what="cut row in front of short ones")


@pytest.mark.parametrize("gname,dt", [("spmv", "float64"), ("rusanov", "float32")])
@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("first_len,first_offset,unused,whole", [(5, 3, 0, True),      # the first row is [0, ends[0]) whatever
                                                                 (5000, 5000, 0, False), (5000, 4999, 0, False),
                                                                 (7, 0, 9, True), (7, 0, 9000, True)])    # edges of no row
def test_offsets_that_do_not_span_the_edges_keep_every_tile_in_bounds(gname, dt, bits, first_len, first_offset, unused, whole):
    """Offsets are taken as row ends: the leading one counts as 0 and edges behind the last row belong to none.  A boundary
    moved to such a row start must not leave a tile with more edges than its stage holds (coordinates in the workspace),
    and the rows are those of the same matrix with a leading 0 and without the unused edges."""
    ir, dtype = graphs.ALL_GRAPHS[gname](), np.dtype(dt)
    prob = with_lengths(ir, [first_len] + [4, 6] * 1500, 17, dtype)
    ref, _, sums = ir_eval.run_graph(ir, prob, dtype, num_threads=4, want_abs_sums=True)
    prob.row_offsets[0] = first_offset
    edge_arrays = {s["target"] for s in ir.selector_register if s.get("selector") != 1}
    for name in edge_arrays:
        v = prob.values[name]
        prob.values[name] = np.concatenate([v, v[:1].repeat(unused, axis=0)])
    for k, v in prob.indices.items():
        prob.indices[k] = np.concatenate([v, np.zeros(unused, v.dtype)])
    for kw in ({}, {"max_ctas": 3}):
        ext = GraphExtension(ir, random_gather=False, **kw)
        got, _ = run_gpu(ext, ir, prob, dtype, offsets_dtype=np.int32 if bits == 32 else np.int64)
        ext.check()
        assert_outputs_match(ir, got, ref, sums, dtype, what=f"{gname} {first_len} {first_offset} {unused} {kw}")
        assert ext.planned_whole_rows() == whole
        info = ext.symbols(torch.float64 if dt == "float64" else torch.float32).graph_info
        tiles = -(-(prob.num_rows + prob.indices[ext.index_names[0]].size) // info.default_tile_items)
        raw = next(reversed(ext._plans.values())).ws[256:256 + (tiles + 1) * bits // 4].cpu().numpy()
        coords = raw.view(np.int32 if bits == 32 else np.int64).reshape(-1, 2)
        steps = np.diff(coords[:, 1])
        assert steps.min() >= 0 and steps.max() <= info.block_threads * info.items_per_thread


def test_row_mode_rows_on_both_sides_of_edge_two_to_the_31():
    """Rows of 16 edges with 64-bit offsets up to 2^31 + 160 000: in the tile around edge 2^31 the positions of a row's ends
    differ in sign as 32-bit numbers.  The rows there, the first and the last ones against the map in torch."""
    if torch.cuda.get_device_properties(0).total_memory < 120 * 2 ** 30:
        pytest.skip("needs a 180 GB device")
    rows = 2 ** 27 + 10_000
    ne = 16 * rows
    assert ne > 2 ** 31
    rng = torch.Generator(device="cuda")
    rng.manual_seed(23)
    rest, stiff = (torch.rand(ne, generator=rng, device="cuda", dtype=torch.float32) for _ in range(2))
    pos = torch.rand(rows, 2, generator=rng, device="cuda", dtype=torch.float32)
    src = torch.arange(rows, device="cuda", dtype=torch.int32).repeat_interleave(16)
    dst = src + torch.randint(1, 1000, (ne,), generator=rng, device="cuda", dtype=torch.int32)
    dst[dst >= rows] -= rows
    ro = torch.arange(rows + 1, device="cuda", dtype=torch.int64) * 16
    ext = GraphExtension(graphs.spring_mass_graph())
    (got,) = ext.merged_spmv_launch(rest, stiff, pos, src, dst, ro, rows, rows)
    ext.check()
    assert ext.planned_whole_rows()
    for first in (0, 2 ** 27 - 5000, rows - 5000):
        e = slice(16 * first, 16 * (first + 5000))
        k, rest_len = stiff[e, None].double(), rest[e, None].double()
        d = (pos[dst[e].long()] - pos[src[e].long()]).double()       # one rounding, the same as the map's
        n = d.norm(dim=1, keepdim=True)
        f = (k * (n - rest_len) * d / n).view(5000, 16, 2)
        # in units of 2^-24: the norm is off by 3 n, which k d / n turns into 3 k |d|; five more roundings of the term and
        # fifteen additions of at most the sum of the magnitudes
        bound = (3 * (k * d.abs()).view(5000, 16, 2) + 20 * f.abs()).sum(dim=1) * 2.0 ** -24
        assert ((got[first:first + 5000].double() - f.sum(dim=1)).abs() <= bound).all()
    del rest, stiff, pos, src, dst, ro, got
    torch.cuda.empty_cache()


@pytest.mark.parametrize("gname,dt,lengths,kw,planned", [
    ("spmv", "float64", [5] * 3000, {}, 4),                                 # partition, look, move; status mirror
    ("spmv", "float64", [40] * 3000, {}, 3),                                # partition, boundaries between CTAs; mirror
    ("spmv", "float64", [40] * 20, {}, 2),                                  # one tile: partition; mirror
    ("spmv", "float64", [40] * 3000, {"random_gather": True}, 2),           # partition into chunks; mirror
    ("spmv", "float64", [5] * 3000, {"gather_windows": True}, 5),           # partition, boundaries, windows, their flag; mirror
    ("mixed_dims", "float32", [5] * 3000, {}, 3),
    ("edge_sum", "float32", [5] * 3000, {}, 2)])                            # header; mirror
def test_the_launch_count_holds_the_plans_kernels(gname, dt, lengths, kw, planned):
    ir, dtype = graphs.ALL_GRAPHS[gname](), np.dtype(dt)
    ext = GraphExtension(ir, **{"random_gather": False, "gather_windows": False, **kw})
    prob = with_lengths(ir, lengths, 61, dtype)
    run_gpu(ext, ir, prob, dtype)
    assert ext.launches == planned + 1


def planned_state(ext, ir, dt, bits, num_rows, num_edges):
    """(coordinates, whole_rows, row_loop, snapped grid) of the last plan's workspace, and the room of its tiles."""
    ws = next(reversed(ext._plans.values())).ws
    header = ws[:256].cpu().numpy().view(np.int32)
    tile_items = int(header[10])
    tiles = -(-(num_rows + num_edges) // tile_items)
    coords = ws[256:256 + (tiles + 1) * bits // 4].cpu().numpy().view(np.int32 if bits == 32 else np.int64).reshape(-1, 2)
    info = ext.symbols(torch.from_numpy(np.zeros(1, dt)).dtype).graph_info
    per_edge, _ = emit_cuda._stream_bytes_per_edge(ir, np.dtype(dt).itemsize)
    tile = info.block_threads * info.items_per_thread
    moves = not emit_cuda.stores_per_edge(ir)
    room = ir_eval.TileRoom(tile, tile * max(bits // 8, per_edge) + (32 * per_edge if moves else 0), per_edge, bits // 8)
    return coords, int(header[38]), int(header[39]), int(header[33]), tile_items, room


PLANS = {
    "all_5": [5] * 6001, "all_16": [16] * 2000, "all_32": [32] * 700, "long_row_late": [8] * 4000 + [33] + [8] * 10,
    "uneven": [1] * 310 + [32] * 10 + [1] * 3000, "mostly_empty": ([0] * 31 + [32]) * 100, "empty_ends": [0] * 700 + [6] * 900 + [0] * 700,
    "cut_long_rows": [300, 1, 1, 1] * 60, "many_short_behind_a_long": [1] * 340 + [601] + [1] * 9000, "one_row": [7],
    "any": np.random.default_rng(67).integers(0, 33, 5000).tolist(), "any_short": np.random.default_rng(71).integers(0, 4, 60000).tolist(),
}


@pytest.mark.parametrize("gname,dt", [("spmv", "float64"), ("spmv", "float32"), ("spring_mass", "float32"), ("swe_delta", "float64"),
                                      ("ops_zoo", "float64"), ("mixed_dims", "float32")])
@pytest.mark.parametrize("case", sorted(PLANS))
def test_plan_coordinates_equal_their_restatement(gname, dt, case):
    """Every coordinate, and what the header says about them, against the steps restated with numpy: partition, boundaries
    of whole rows, or boundaries between the CTAs of the plan's grid."""
    ir, dtype = graphs.ALL_GRAPHS[gname](), np.dtype(dt)
    prob = with_lengths(ir, PLANS[case], 73, dtype)
    needs_row = any(s.get("row_identity") for s in ir.selector_register)
    light = emit_cuda.light_map(ir)
    gathers = [(prob.indices[s["selector_name"]], dtype.itemsize * graphs.dim_of(s["shape"])) for s in ir.selector_register
               if s.get("selector") == 1 and not s.get("row_identity")] if not needs_row else []
    acc = sum(graphs.dim_of(o["shape"]) for o in ir.outputs if str(o["target"]) == "reducer")
    for bits, kw in ((32, {"max_ctas": 5}), (64, {"max_ctas": 40}), (32, {"max_ctas": 3, "tile_items": 100}), (64, {"max_ctas": 1})):
        ext = GraphExtension(ir, random_gather=False, gather_windows=False, **kw)
        run_gpu(ext, ir, prob, dtype, offsets_dtype=np.int32 if bits == 32 else np.int64)
        got, whole, loop, snapped, tile_items, room = planned_state(ext, ir, dt, bits, prob.num_rows, prob.nnz)
        ro = prob.row_offsets.astype(np.int32 if bits == 32 else np.int64)
        want = ir_eval.tile_coordinates(ro, tile_items)
        want_whole = want_loop = 0
        if not emit_cuda.stores_per_edge(ir) and prob.nnz <= 32 * prob.num_rows:
            want, want_whole, want_loop = ir_eval.whole_rows_plan(want, ro, prob.nnz, room, edge_lanes=not needs_row, heavy=not light,
                                                                  accumulators=acc, gathers=gathers)
        tiles = want.shape[0] - 1
        grid = min(kw["max_ctas"], tiles)
        ok = want_whole == 1 and grid >= 2
        if want_whole != 1:
            want, ok = ir_eval.snap_cta_boundaries(want, ro, grid, room)
        assert (whole, loop, snapped) == (want_whole, want_loop, grid if ok else 0), (bits, kw)
        assert np.array_equal(got, want), (bits, kw)


def test_boundaries_aligned_for_one_grid_and_cut_for_another_hand_carries_over():
    """Rows of few edges that stay on the loop with carries (one lane in ten would have an edge to work on): the plan puts the
    boundaries between the CTAs of its grid on row ends; other grids find boundaries that cut rows and hand carries over."""
    lib = load_library()
    ir = graphs.spmv_graph()
    lengths = ([32] + [1] * 40) * 400
    prob = with_lengths(ir, lengths, 79, np.float64)
    ref, _, sums = ir_eval.run_graph(ir, prob, np.float64, num_threads=4, want_abs_sums=True)
    ext = GraphExtension(ir, random_gather=False, max_ctas=7)
    run_gpu(ext, ir, prob, np.float64)
    coords, whole, _, snapped, tile_items, room = planned_state(ext, ir, "float64", 32, prob.num_rows, prob.nnz)
    assert not ext.planned_whole_rows() and whole == 0 and snapped == 7
    tiles, ro = coords.shape[0] - 1, prob.row_offsets
    cut = {t for t in range(1, tiles) if coords[t, 0] < prob.num_rows and coords[t, 1] != ro[coords[t, 0]]}
    plan = next(reversed(ext._plans.values()))
    v, x = (torch.from_numpy(prob.values[k]).cuda() for k in ("vals", "x"))
    cols, ro_t = torch.from_numpy(prob.indices["selector"]).cuda(), plan.keep[0]
    y = torch.empty(prob.num_rows, dtype=torch.float64, device="cuda")
    vp, ip, op = (ctypes.c_void_p * 2)(v.data_ptr(), x.data_ptr()), (ctypes.c_void_p * 1)(cols.data_ptr()), (ctypes.c_void_p * 1)(y.data_ptr())
    lib.flexspmv_spmv_f64_launch.restype = ctypes.c_int
    for grid in (7, 1, 5, 11, 29, tiles):
        starts = {c * (tiles // grid) + min(c, tiles % grid) for c in range(1, grid)}
        assert bool(starts & cut) == (grid not in (1, 7))               # carries between the CTAs of the other grids
        desc = Desc(prob.num_rows, prob.nnz, prob.num_cols, 32, 0, grid, 0)
        y.fill_(float("nan"))
        assert lib.flexspmv_spmv_f64_launch(ctypes.byref(desc), vp, ip, ctypes.c_void_p(ro_t.data_ptr()), op, ctypes.c_void_p(plan.ws.data_ptr()),
                                            ctypes.c_size_t(plan.nbytes), None) == 0
        torch.cuda.synchronize()
        assert_outputs_match(ir, [y.cpu().numpy()], ref, sums, np.dtype(np.float64), what=f"grid {grid}")
    ext.check()


@pytest.mark.parametrize("offset_dtype", [torch.int32, torch.int64])
def test_a_matrix_without_edges_can_be_planned(offset_dtype):
    """Empty index tensors have no address: binding and planning such a block (a rank's empty share) is no error."""
    ext = GraphExtension(graphs.spmv_graph(), random_gather=False)
    vals, x = torch.empty(0, dtype=torch.float64, device="cuda"), torch.ones(50, dtype=torch.float64, device="cuda")
    cols, ro = torch.empty(0, dtype=torch.int32, device="cuda"), torch.zeros(51, dtype=offset_dtype, device="cuda")
    ext.prepare([vals, x], [cols], ro, [torch.empty(50, dtype=torch.float64, device="cuda")], 50, 0, 50)
    ext.check()
