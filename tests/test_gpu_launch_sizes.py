"""Kernels picked by the size of a launch, each test saying which one it means: the tile kernel without stages (few tiles a CTA, short
rows, even shares) and with tiles going round the CTAs (large gathered vectors) against its plain form, bit for bit; the warp kernel's
two forms; the sort's 10-bit digits and its two ways to the offsets; small CTAs for wide records."""
import ctypes

import numpy as np
import pytest
import torch

from flexspmv_b200 import graphs, problems
from flexspmv_b200.binding import GraphExtension, load_library
from flexspmv_b200.python_wrapper.dynamic_replace_submodule import sort_edges_by_row
from oracle import ir_eval
from parity import assert_outputs_match
from test_gpu_parity import NP2T, run_gpu
from test_gpu_whole_rows import with_lengths

pytestmark = pytest.mark.gpu

GRAPHS = [("spmv", "float64"), ("spmv", "float32"), ("spmv", "int64"), ("spring_mass", "float32"), ("rusanov", "float64"),
          ("swe_delta", "float32"), ("swe_boundary", "float64"), ("ops_zoo", "float64")]
TILE, SMALL, ROUNDS, WARP, AHEAD = 1, 2, 3, 4, 5      # FLEXSPMV_KERNEL_* of include/flexspmv.h


def last_kernel():
    return load_library().flexspmv_debug_last_kernel()


def header_word(ext, i):
    """An int32 of the header of the workspace that was planned last (struct WorkspaceHeader)."""
    return int(next(reversed(ext._plans.values())).ws[:256].cpu().numpy().view(np.int32)[i])


def launch(ir, prob, dtype, num_cols, bits, kernel=None, loop=None, **kw):
    """Outputs (as bytes) of one launch and whether its plan holds whole rows; ``num_cols``: the number of vertices that the
    descriptor names; ``kernel``: the form that the launch has to take; ``loop``: whether the plan has to choose the loop over
    whole rows."""
    ext = GraphExtension(ir, random_gather=False, **kw)
    non_gather, gathers, index_names = graphs.operator_signature(ir)
    v = [torch.from_numpy(np.ascontiguousarray(prob.values[n].astype(dtype))).cuda() for n in non_gather + gathers]
    ix = [torch.from_numpy(np.ascontiguousarray(prob.indices[n])).cuda() for n in index_names]
    ro = torch.from_numpy(prob.row_offsets.astype(np.int32 if bits == 32 else np.int64)).cuda()
    outs = [torch.full((prob.num_rows, d), -7, dtype=v[0].dtype, device="cuda") for _, d in ext._out_kinds]
    ext.launch_into(v, ix, ro, outs, prob.num_rows, prob.nnz, num_cols)
    assert kernel is None or last_kernel() == kernel
    ext.check()
    assert loop is None or header_word(ext, 39) == loop
    return [o.cpu().numpy().tobytes() for o in outs], ext.planned_whole_rows()


def default_tile(ir, dtype):
    return GraphExtension(ir).symbols(NP2T[dtype]).graph_info.default_tile_items


@pytest.mark.parametrize("gname,dt", GRAPHS)
@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("lengths,tile_items", [([3] * 8003, 0), ([0, 3, 5, 2] * 2900 + [0] * 40, 0), ([2, 1, 4] * 600, 300), ([1] * 31, 0)],
                         ids=["3", "uneven", "small_tiles", "31_rows"])
def test_small_launches_equal_staged_ones(gname, dt, bits, lengths, tile_items):
    """At most one tile a CTA, and two: rows straight from global memory.  Four tiles a CTA and more: stages.  (31 rows are one tile,
    which no grid stages.)"""
    ir, dtype = graphs.ALL_GRAPHS[gname](), np.dtype(dt)
    prob = with_lengths(ir, lengths, 101, dtype)
    tile = tile_items or default_tile(ir, dtype)
    tiles = -(-(prob.num_rows + prob.nnz) // tile)
    kw = {"tile_items": tile_items} if tile_items else {}
    loop = 0 if gname == "ops_zoo" and len(set(lengths)) > 1 else 1       # (a map that divides, lanes that would idle: the other loop)
    small, whole = launch(ir, prob, dtype, prob.num_cols, bits, SMALL, loop, **kw)
    assert whole and (tiles >= 8 or tiles == 1)
    if tiles > 1:
        two, _ = launch(ir, prob, dtype, prob.num_cols, bits, SMALL, loop, max_ctas=-(-tiles // 2), **kw)
        staged, _ = launch(ir, prob, dtype, prob.num_cols, bits, TILE, loop, max_ctas=tiles // 4, **kw)
        one, _ = launch(ir, prob, dtype, prob.num_cols, bits, TILE, loop, max_ctas=1, **kw)
        assert small == staged == two == one
    ref, _, sums = ir_eval.run_graph(ir, prob, dtype, num_threads=4, want_abs_sums=True)
    got, _ = run_gpu(GraphExtension(ir, random_gather=False, **kw), ir, prob, dtype)
    assert_outputs_match(ir, got, ref, sums, dtype, what=f"{gname} small")


@pytest.mark.parametrize("gname,dt", GRAPHS)
@pytest.mark.parametrize("bits", [32, 64])
def test_small_launches_with_several_rows_a_thread(gname, dt, bits):
    """Rows of one edge, about 600 a CTA of 288 threads: the loop asks for the ends of a thread's next row."""
    ir, dtype = graphs.ALL_GRAPHS[gname](), np.dtype(dt)
    prob = with_lengths(ir, [1] * 5990, 107, dtype)
    tiles = -(-(prob.num_rows + prob.nnz) // default_tile(ir, dtype))
    grid = min(tiles, 10)
    assert prob.num_rows / grid > 2 * 288 and tiles <= 2 * grid
    small, whole = launch(ir, prob, dtype, prob.num_cols, bits, SMALL, 1, max_ctas=grid)
    staged, _ = launch(ir, prob, dtype, prob.num_cols, bits, TILE, 1, max_ctas=1)
    assert whole and small == staged


@pytest.mark.parametrize("gname,dt,row_edges", [("spmv", "float64", 12), ("spmv", "float32", 15), ("spring_mass", "float32", 10),
                                                ("swe_delta", "float64", 4)])
@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("lengths,seen", [([3] * 30_000, {0}), ([2] * 15_000 + [6] * 15_000, {0, 1}), ([1] * 15_000 + [7] * 15_000, {1}),
                                          ([7] * 15_000 + [1] * 15_000, {1}), ([3] * 20_000 + [16] * 1000 + [3] * 9000, {1}),
                                          ([0] * 100 + [3] * 30_000 + [0] * 3, {0})],
                         ids=["even", "half_as_many_again", "more", "more_in_front", "one_place", "empty_ends"])
def test_shares_of_very_different_sizes_keep_the_stages(gname, dt, row_edges, bits, lengths, seen):
    """The plan looks at the equal shares of the rows that a small launch would give its CTAs; where one holds more than half as much
    again as the tiles that a CTA has at most, or longer rows than a small launch takes, the kernel runs its loop with stages.  The bits
    are the same either way."""
    ir, dtype = graphs.ALL_GRAPHS[gname](), np.dtype(dt)
    prob = with_lengths(ir, lengths, 109, dtype)
    tile = default_tile(ir, dtype)
    grid = -(-(prob.num_rows + prob.nnz) // tile)                   # a tile a CTA
    share = (-(-prob.num_rows // grid) + 31) // 32 * 32
    sizes = [(len(lengths[r:r + share]), sum(lengths[r:r + share])) for r in range(0, prob.num_rows, share)]
    uneven = int(any(rows + edges > 3 * tile // 2 or edges > row_edges * share for rows, edges in sizes))
    assert uneven in seen
    results = []
    for max_ctas in (0, 1):
        ext = GraphExtension(ir, random_gather=False, max_ctas=max_ctas)
        got, _ = run_gpu(ext, ir, prob, dtype, offsets_dtype=np.int32 if bits == 32 else np.int64)
        ext.check()
        assert ext.planned_whole_rows() and header_word(ext, 39) == 1
        assert last_kernel() == (TILE if max_ctas else SMALL)
        assert header_word(ext, 46) == (0 if max_ctas else uneven)
        results.append([g.tobytes() for g in got])
    assert results[0] == results[1]


@pytest.mark.parametrize("gname,dt", GRAPHS)
@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("ctas", [1, 3, 7])
def test_rounds_equal_runs_of_consecutive_tiles(gname, dt, bits, ctas):
    """A descriptor with many vertices takes tiles in rounds of four a CTA and splits the rest; the results are those of the plain
    order.  40 001 rows of 6 and 7 edges are 140 tiles (2040 items) and more."""
    ir, dtype = graphs.ALL_GRAPHS[gname](), np.dtype(dt)
    prob = with_lengths(ir, [6, 7] * 20_000 + [3], 103, dtype)
    plain, whole = launch(ir, prob, dtype, prob.num_cols, bits, TILE, max_ctas=ctas)
    rounds, _ = launch(ir, prob, dtype, 1 << 27, bits, ROUNDS, max_ctas=ctas)
    assert whole and plain == rounds
    long = with_lengths(ir, [6, 7] * 20_000 + [200], 103, dtype)             # not whole rows: the loop with carries in either
    plain, whole = launch(ir, long, dtype, long.num_cols, bits, TILE, max_ctas=ctas)
    rounds, _ = launch(ir, long, dtype, 1 << 27, bits, ROUNDS, max_ctas=ctas)
    assert not whole and plain == rounds


@pytest.mark.parametrize("dtype,tol", [(torch.float32, 1e-5), (torch.float64, 1e-12)])
@pytest.mark.parametrize("rows", [100_003, 900_007])
def test_warp_kernel_with_few_and_many_chunks_a_warp(dtype, tol, rows):
    """1.6 M and 14 M random edges lie on either side of the small configuration's limit; rows of 0 to 300 edges.  Against sums in
    64 bits, relative to the sums of the terms' magnitudes."""
    g = torch.Generator(device="cuda")
    g.manual_seed(rows)
    ln = torch.randint(0, 32, (rows,), generator=g, device="cuda")
    ln[::5000] = 300
    ro = torch.zeros(rows + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(ln, 0, out=ro[1:])
    e = int(ro[-1])
    cols = torch.randint(0, rows, (e,), generator=g, device="cuda", dtype=torch.int32)
    vals, x = (torch.rand(k, generator=g, device="cuda", dtype=dtype) - 0.5 for k in (e, rows))
    ext = GraphExtension(graphs.spmv_graph(), random_gather=True)
    (y,) = ext.merged_spmv_launch(vals, x, cols, ro.to(torch.int32), rows, rows)
    ext.check()
    of = torch.repeat_interleave(torch.arange(rows, device="cuda"), ln)
    terms = vals.double() * x.double()[cols.long()]
    zero = torch.zeros(rows, dtype=torch.float64, device="cuda")
    err = (y.double() - zero.index_add(0, of, terms)).abs()
    assert bool((err <= tol * zero.index_add(0, of, terms.abs())).all())
    (again,) = ext.merged_spmv_launch(vals, x, cols, ro.to(torch.int32), rows, rows)
    assert torch.equal(y, again)


@pytest.mark.parametrize("rows", [257, 512, 1023, 1024, 1025, (1 << 18) + 3, (1 << 20) - 1, 1 << 20, (1 << 20) + 1])
@pytest.mark.parametrize("n", [1, 8191, 8192, 8193, 5 * 8192 + 77])
def test_ten_bit_digits(rows, n):
    rng = np.random.default_rng(rows + n)
    draws = {"uniform": rng.integers(0, rows, n), "last": np.full(n, rows - 1), "few": rng.choice([0, rows // 2, rows - 1], n)}
    for what, ids in draws.items():
        for dtype in (np.int32, np.int64):
            perm, crow = sort_edges_by_row(torch.from_numpy(ids.astype(dtype)).cuda(), rows)
            assert np.array_equal(perm.cpu().numpy(), np.argsort(ids, kind="stable").astype(np.int32)), what
            assert np.array_equal(crow.cpu().numpy(), np.searchsorted(np.sort(ids), np.arange(rows + 1))), what


def test_offsets_where_few_rows_hold_most_edges():
    """More than 64 edges a row over 1024 rows: bisected; blocks beside them: read once."""
    rows, n = 5000, 300_000
    ids = np.random.default_rng(7).choice([3, 1023, 1024, 2500, 2501, 4999], n, p=[0.3, 0.1, 0.05, 0.25, 0.25, 0.05])
    _, crow = sort_edges_by_row(torch.from_numpy(ids).cuda(), rows)
    assert np.array_equal(crow.cpu().numpy(), np.searchsorted(np.sort(ids), np.arange(rows + 1)))


def test_scratch_for_eight_bit_digits_is_enough():
    """Three arrays of 4 bytes an edge and the counts of 256 digits a tile of 4096: what the sort asked for before it had wider
    digits.  A byte less is refused."""
    lib = load_library()
    n, rows = 30_011, 1 << 20
    ids = np.random.default_rng(9).integers(0, rows, n)
    up = lambda b: -(-b // 256) * 256
    need = 3 * up(4 * n) + up(-(-n // 4096) * 1024) + 1024
    full = ctypes.c_size_t()
    assert lib.flexspmv_sort_rows_bytes(ctypes.c_int64(n), ctypes.byref(full)) == 0 and full.value > need
    d_ids = torch.from_numpy(ids).cuda()
    for size in (need, full.value, need - 1):
        perm = torch.full((n,), -1, dtype=torch.int32, device="cuda")
        crow = torch.empty(rows + 1, dtype=torch.int64, device="cuda")
        scratch, status = torch.empty(full.value, dtype=torch.uint8, device="cuda"), torch.empty(1, dtype=torch.int32, device="cuda")
        ptr = lambda t: ctypes.c_void_p(t.data_ptr())
        code = lib.flexspmv_sort_rows(ptr(d_ids), 64, ctypes.c_int64(n), ctypes.c_int64(rows), ptr(perm), ptr(crow), 64, ptr(scratch),
                                      ctypes.c_size_t(size), ptr(status), None)
        torch.cuda.synchronize()
        if size < need:
            assert code == -3
        else:
            assert code == 0 and np.array_equal(perm.cpu().numpy(), np.argsort(ids, kind="stable").astype(np.int32))


@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("n,rows", [(5, 3), (4097, 1), (20_011, 200), (300_007, 10_007), (600_011, 600_000)])
def test_sorts_behind_one_another_share_scratch(n, rows, captured):
    """The kernels of a sort start while the ones before them drain: sorts of new ids over the same scratch and outputs,
    nothing between them but the stream's order."""
    lib = load_library()
    need = ctypes.c_size_t()
    assert lib.flexspmv_sort_rows_bytes(ctypes.c_int64(n), ctypes.byref(need)) == 0
    rng = np.random.default_rng(n)
    scratch, ids_now = torch.empty(need.value, dtype=torch.uint8, device="cuda"), torch.zeros(n, dtype=torch.int64, device="cuda")
    perm, crow = torch.empty(n, dtype=torch.int32, device="cuda"), torch.empty(rows + 1, dtype=torch.int32, device="cuda")
    status = torch.empty(1, dtype=torch.int32, device="cuda")
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())

    def sort():
        assert lib.flexspmv_sort_rows(ptr(ids_now), 64, ctypes.c_int64(n), ctypes.c_int64(rows), ptr(perm), ptr(crow), 32, ptr(scratch),
                                      ctypes.c_size_t(need.value), ptr(status), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0

    graph = torch.cuda.CUDAGraph()
    if captured:
        with torch.cuda.graph(graph):
            sort()
    ids = [rng.integers(0, rows, n) for _ in range(6)]
    on_device = [torch.from_numpy(i).cuda() for i in ids]
    got = []
    for i in on_device:
        ids_now.copy_(i)
        graph.replay() if captured else sort()
        got.append((perm.clone(), crow.clone()))
    torch.cuda.synchronize()
    assert int(status) == 0
    for i, (p, c) in zip(ids, got):
        assert np.array_equal(p.cpu().numpy(), np.argsort(i, kind="stable").astype(np.int32))
        assert np.array_equal(c.cpu().numpy(), np.searchsorted(np.sort(i), np.arange(rows + 1)))


@pytest.mark.parametrize("rows", [1, 255, 256, 257, 1025, 300_000, 303_104, 303_105, 400_001])
@pytest.mark.parametrize("ids", ["few", "limit", "above", "skewed"])
@pytest.mark.parametrize("offset_bits", [32, 64])
def test_offsets_read_once_or_bisected(rows, ids, offset_bits):
    """Blocks of 256 and of 1024 rows (from two an SM on), at 24 ids a row (read once), one more in a block (bisected) and where
    one block holds most ids; rows without ids at both ends."""
    rng = np.random.default_rng(rows)
    if ids == "few":
        counts = rng.integers(0, 3, rows)
    elif ids == "skewed":
        counts = rng.integers(0, 4, rows)
        counts[rows // 2:rows // 2 + 300] = 2000
    else:
        counts = np.full(rows, 24)
        if ids == "above":
            counts[rows // 3] = 25
    if rows > 2:
        counts[0] = counts[-1] = 0
    of = np.repeat(np.arange(rows), counts)
    n = of.size
    lib = load_library()
    need = ctypes.c_size_t()
    assert lib.flexspmv_sort_rows_bytes(ctypes.c_int64(n), ctypes.byref(need)) == 0
    shuffled = torch.from_numpy(of)[torch.randperm(n, generator=torch.Generator().manual_seed(rows))].cuda()
    perm, scratch = torch.empty(max(n, 1), dtype=torch.int32, device="cuda"), torch.empty(need.value, dtype=torch.uint8, device="cuda")
    got = torch.full((rows + 2,), -1, dtype=torch.int32 if offset_bits == 32 else torch.int64, device="cuda")
    status = torch.empty(1, dtype=torch.int32, device="cuda")
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())
    assert lib.flexspmv_sort_rows(ptr(shuffled), 64, ctypes.c_int64(n), ctypes.c_int64(rows), ptr(perm), ptr(got), offset_bits, ptr(scratch),
                                  ctypes.c_size_t(need.value), ptr(status), None) == 0
    want = np.concatenate([[0], np.cumsum(counts), [-1]])                  # (the word behind the last offset stays)
    assert np.array_equal(got.cpu().numpy(), want) and int(status) == 0


@pytest.mark.parametrize("gname,dt,edges,kernel", [
    ("spmv", "float64", 12, SMALL), ("spmv", "float64", 13, TILE), ("spmv", "float32", 15, SMALL), ("spmv", "float32", 16, TILE),
    ("spring_mass", "float32", 10, SMALL), ("spring_mass", "float64", 11, TILE), ("rusanov", "float32", 6, SMALL),
    ("rusanov", "float32", 7, TILE), ("rusanov", "float64", 4, SMALL), ("rusanov", "float64", 5, TILE), ("swe_delta", "float32", 6, SMALL),
    ("swe_delta", "float64", 5, TILE), ("swe_boundary", "float64", 10, SMALL), ("ops_zoo", "float32", 7, SMALL), ("ops_zoo", "float32", 8, TILE)])
def test_rows_of_small_launches_are_short(gname, dt, edges, kernel):
    ir, dtype = graphs.ALL_GRAPHS[gname](), np.dtype(dt)
    prob = with_lengths(ir, [edges] * 3001, 113, dtype)
    default, _ = launch(ir, prob, dtype, prob.num_cols, 32, kernel)
    staged, _ = launch(ir, prob, dtype, prob.num_cols, 32, TILE, max_ctas=1)
    assert default == staged


@pytest.mark.parametrize("dt,rows_a_cta,kernel", [("float64", 864, SMALL), ("float64", 896, TILE), ("int64", 896, TILE), ("float32", 1728, SMALL),
                                                  ("float32", 1760, TILE)])
def test_small_launches_have_few_rows_a_thread(dt, rows_a_cta, kernel):
    """288 threads a CTA: three rows each of 8-byte values, six of 4-byte ones."""
    ir, dtype = graphs.spmv_graph(), np.dtype(dt)
    prob = with_lengths(ir, [1] * (5 * rows_a_cta - 7), 127, dtype)
    assert 2 * prob.num_rows <= 3 * 5 * 1280
    default, _ = launch(ir, prob, dtype, prob.num_cols, 32, kernel, max_ctas=5)
    staged, _ = launch(ir, prob, dtype, prob.num_cols, 32, TILE, max_ctas=1)
    assert default == staged


@pytest.mark.parametrize("dt", ["float32", "float64", "int64"])
@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("kernel", [WARP, AHEAD])
def test_both_forms_of_the_warp_kernel_match_the_oracle(dt, bits, kernel):
    """Rows over many chunks, runs and CTAs, empty rows, odd chunk sizes, in the form for few chunks a warp (the default grid) and, on one
    to three CTAs, in the one for many.  Integers bit for bit, the same bits twice."""
    ir, dtype = graphs.spmv_graph(), np.dtype(dt)
    offsets = np.int32 if bits == 32 else np.int64
    cases = [((2, 5000, 300_000), 0, 3), ((40_000, 40_000, 120_000), 0, 1), ((97, 97, 100_000), 0, 1), ((3000, 3000, 2000), 7, 1),
             ((300, 300, 40_000), 33, 2), ((60, 60, 250_000), 159, 2), ((1, 1, 90_000), 0, 1), ((90_000, 5, 300), 0, 1)]
    for (rows, vertices, nnz), tile_items, few_ctas in cases:
        prob = problems.random_problem(ir, rows, vertices, nnz, seed=3000 + rows + nnz, dtype=dtype)
        ref, _, sums = ir_eval.run_graph(ir, prob, dtype, num_threads=8, want_abs_sums=True)
        kw = {"tile_items": tile_items} if tile_items else {}
        results = []
        for _ in range(2):
            ext = GraphExtension(ir, random_gather=True, max_ctas=few_ctas if kernel == WARP else 0, **kw)
            got, _ = run_gpu(ext, ir, prob, dtype, offsets_dtype=offsets)
            assert last_kernel() == kernel, (rows, nnz)
            ext.check()
            assert_outputs_match(ir, got, ref, sums, dtype, what=f"warp kernel {kernel} {dt} {rows} x {nnz}")
            results.append([g.tobytes() for g in got])
        assert results[0] == results[1]


@pytest.mark.parametrize("dt,chunks,kernel", [("float64", 439, AHEAD), ("float64", 440, WARP), ("float32", 527, AHEAD), ("float32", 528, WARP)])
def test_chunks_a_warp_choose_the_form(dt, chunks, kernel):
    """One CTA of 20 or 24 warps: up to 22 chunks a warp."""
    ir, dtype = graphs.spmv_graph(), np.dtype(dt)
    prob = problems.random_problem(ir, 500, 500, chunks * 160 - 500, seed=131, dtype=dtype)
    ref, _, sums = ir_eval.run_graph(ir, prob, dtype, num_threads=4, want_abs_sums=True)
    got, _ = run_gpu(GraphExtension(ir, random_gather=True, max_ctas=1), ir, prob, dtype)
    assert last_kernel() == kernel
    assert_outputs_match(ir, got, ref, sums, dtype, what=f"{chunks} chunks")


@pytest.mark.parametrize("gname,dt,record,megabytes", [("spmv", "float64", 8, 40), ("spmv", "float32", 4, 40), ("spring_mass", "float32", 8, 10),
                                                       ("rusanov", "float64", 24, 10)])
def test_the_size_of_the_gathered_vectors_chooses_the_order(gname, dt, record, megabytes):
    ir, dtype = graphs.ALL_GRAPHS[gname](), np.dtype(dt)
    prob = with_lengths(ir, [6, 7] * 10_000, 137, dtype)
    most = (megabytes << 20) // record
    plain, _ = launch(ir, prob, dtype, most, 32, TILE, max_ctas=2)
    rounds, _ = launch(ir, prob, dtype, most + 1, 32, ROUNDS, max_ctas=2)
    assert plain == rounds


@pytest.mark.parametrize("dt", ["float64", "int64", "float32"])
@pytest.mark.parametrize("lengths", [[0, 5, 16] * 1000, [300] * 60, [1] * 500 + [5000] + [0] * 300 + [7] * 200], ids=["short", "several_tiles", "one_long"])
def test_wide_records_in_small_ctas(dt, lengths):
    """Eight-byte values run 64 threads x 4 edges: the default tile and those that a caller may ask for, rows inside a tile and
    over several, the default grid and two CTAs."""
    ir, dtype = graphs.mixed_dims_graph(), np.dtype(dt)
    prob = with_lengths(ir, lengths, 139, dtype)
    ref, _, sums = ir_eval.run_graph(ir, prob, dtype, num_threads=4, want_abs_sums=True)
    for kw in ({}, {"tile_items": 193}, {"tile_items": 256}, {"tile_items": 255, "max_ctas": 2}, {"tile_items": 1, "max_ctas": 50}):
        ext = GraphExtension(ir, **kw)
        got, _ = run_gpu(ext, ir, prob, dtype, offsets_dtype=np.int64 if "max_ctas" in kw else np.int32)
        ext.check()
        assert_outputs_match(ir, got, ref, sums, dtype, what=f"mixed_dims {dt} {kw}")


@pytest.mark.parametrize("dt", ["float64", "float32", "int64"])
@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("lengths", [[5], [4, 5], [3, 4, 5, 6, 7], [0, 10, 5, 5], [1, 9, 4, 5, 5, 0, 6], [7], [6, 7, 7, 5], [0, 14, 6, 8, 3]],
                         ids=["5", "4_5", "3_to_7", "0_10", "1_to_9", "7", "5_to_7", "0_14"])
@pytest.mark.parametrize("rows,kernel", [(9000, SMALL), (600_000, TILE)])
def test_short_rows_in_one_round(dt, bits, lengths, rows, kernel):
    """Four to five edges a row on average, and no row of more, are taken five at a time, and up to seven (4-byte values) seven; the same
    rows in front of others that bring the average out of those ranges are taken four at a time.  The same bits."""
    ir, dtype = graphs.spmv_graph(), np.dtype(dt)
    mine = (lengths * (rows // len(lengths) + 1))[:rows]
    others = [12] * rows
    prob = with_lengths(ir, mine + others, 241, dtype)
    n, e = len(mine), sum(mine)
    assert 4 * n < e <= 7 * n and prob.nnz > 7 * prob.num_rows
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    non_gather, gathers, index_names = graphs.operator_signature(ir)
    x = dev(prob.values[gathers[0]].astype(dtype))
    results = []
    for count, edges in ((n, e), (prob.num_rows, prob.nnz)):
        ext = GraphExtension(ir, random_gather=False)
        y = torch.full((count,), 7, dtype=x.dtype, device="cuda")
        ext.launch_into([dev(prob.values[non_gather[0]][:edges].astype(dtype)), x], [dev(prob.indices[index_names[0]][:edges])],
                        dev(prob.row_offsets[:count + 1].astype(np.int32 if bits == 32 else np.int64)), [y], count, edges, prob.num_cols)
        longest, most = max(lengths), 7 if dt == "float32" else 5
        batch = 4 if count > n or longest > most else 5 if longest <= 5 else 7
        assert load_library().flexspmv_debug_last_row_batch() == batch
        if count == n:
            assert last_kernel() == kernel
        ext.check()
        assert ext.planned_whole_rows()
        results.append(y[:n].cpu().numpy().tobytes())
    assert results[0] == results[1]


@pytest.mark.parametrize("dt,lengths,known,batch", [("float64", [5], None, 5), ("float64", [5], 0, 4), ("float64", [4] * 99 + [5], None, 5), ("float64", [4], None, 4),
                                                    ("float64", [5] * 999 + [6, 4], None, 4), ("float64", [6, 7], None, 4), ("float32", [5] * 9 + [6, 4], None, 7),
                                                    ("float32", [7], None, 7), ("float32", [7] * 999 + [8, 6], None, 4), ("float32", [7, 7, 8], None, 4),
                                                    ("int64", [5], None, 5), ("int64", [6], None, 4)])
def test_the_longest_row_decides_how_many_edges_go_together(dt, lengths, known, batch):
    """Averages at, just above and just below the lines, each with a longest row that a batch holds and with one more; and tiles that go round
    the CTAs take four."""
    ir, dtype = graphs.spmv_graph(), np.dtype(dt)
    prob = with_lengths(ir, lengths * (60_000 // len(lengths)), 263, dtype)
    ext = GraphExtension(ir, random_gather=False, longest_row=known)
    got, _ = run_gpu(ext, ir, prob, dtype)
    ext.check()
    assert load_library().flexspmv_debug_last_row_batch() == batch
    ref, _, sums = ir_eval.run_graph(ir, prob, dtype, num_threads=4, want_abs_sums=True)
    assert_outputs_match(ir, got, ref, sums, dtype, what=f"spmv {dt}")
    launch(ir, prob, dtype, 1 << 27, 32, ROUNDS, max_ctas=4)
    assert load_library().flexspmv_debug_last_row_batch() == 4
