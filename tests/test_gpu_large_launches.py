"""The large configuration of the row-mode graphs (GraphApi::use_big): the sizes on both sides of its rule, tiles of equal number
and of the largest size, both orders of the tiles, plans with and without whole rows -- each against the configuration that a caller
who names a number of CTAs gets, bit for bit where sums run left to right in both, and against the oracle."""
import ctypes

import numpy as np
import pytest
import torch

from flexspmv_b200 import graphs
from flexspmv_b200.binding import GraphExtension, load_library
from oracle import ir_eval
from parity import assert_outputs_match
from test_gpu_launch_sizes import ROUNDS, default_tile, header_word, launch, run_gpu, with_lengths

pytestmark = pytest.mark.gpu

# graph, type, threads and items of each that take rows, edges a row that suit, and rows that are too short and too long
LARGE = [("rusanov", "float64", 736, 4, 3), ("rusanov", "float32", 992, 4, 3), ("swe_delta", "float64", 736, 4, 3),
         ("spring_mass", "float64", 736, 7, 7), ("spring_mass", "float32", 992, 8, 8)]


def sms():
    return torch.cuda.get_device_properties(0).multi_processor_count


def longest_row_of(ext):
    plan = next(reversed(ext._plans.values()))
    out = torch.full((1,), -7, dtype=torch.int32, device="cuda")
    assert load_library().flexspmv_workspace_longest_row(ctypes.c_void_p(plan.ws_ptr), ctypes.c_void_p(out.data_ptr()), None) == 0
    torch.cuda.synchronize()
    assert int(out) == ext._longest_row(plan)
    return int(out)


def small_limit(ir, dtype):
    """Items up to which a launch of short rows takes the kernel without stages: 9 tiles for four CTAs, of which an SM holds three
    or four."""
    resident = 3 if dtype == np.float64 and ir.name != "spring_mass" else 4
    return 9 * sms() * resident * default_tile(ir, dtype) // 4


@pytest.mark.parametrize("gname,dt,threads,ipt,edges", LARGE)
@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("tiles,lengths", [(0, [0]), (1, [0]), (3, [1, -3, 1, 0, 2]), (5, [-1, 1]), (16, [0]), (17, [0])],
                         ids=["small", "above", "uneven", "five", "sixteen", "seventeen"])
def test_large_launches_equal_those_of_the_other_configuration(gname, dt, threads, ipt, edges, bits, tiles, lengths):
    ir, dtype = graphs.ALL_GRAPHS[gname](), np.dtype(dt)
    tile, lengths = threads * ipt - ipt, [edges + more for more in lengths]
    if tiles > 5 and (bits == 64 or (gname, dt) != ("rusanov", "float64")):
        pytest.skip("one graph and width at the large sizes")
    # the last small launch and the first one that is not; up to `tiles` tiles a CTA
    # (Rusanov's first one in fp64 would leave a fifth of its last turn's lanes idle)
    first = 30_000 if (gname, dt) == ("rusanov", "float64") else 4
    items = small_limit(ir, dtype) + (first if tiles else 0) if tiles < 2 else sms() * tile * tiles - 7 + (60 if tiles == 17 else 0)
    rows = items // (sum(lengths) + len(lengths)) * len(lengths) + (len(lengths) if tiles == 1 else 0)
    prob = with_lengths(ir, lengths * (rows // len(lengths)), 211, dtype)
    items = prob.num_rows + prob.nnz
    longest = max(lengths)            # named, so that the rows' evenness does not come into it
    ext = GraphExtension(ir, random_gather=False, longest_row=longest)
    run_gpu(ext, ir, prob, dtype, offsets_dtype=np.int32 if bits == 32 else np.int64)
    ext.check()
    each, took = -(-items // (sms() * tile)), header_word(ext, 10)
    if tiles == 0:
        assert took == default_tile(ir, dtype)
        return
    assert took == (-(-items // (sms() * each)) if each <= 16 else tile)
    large, whole = launch(ir, prob, dtype, prob.num_cols, bits, longest_row=longest)
    named, also = launch(ir, prob, dtype, prob.num_cols, bits, max_ctas=3 * sms())
    assert whole and also and large == named
    rounds, _ = launch(ir, prob, dtype, 1 << 27, bits, ROUNDS, longest_row=longest)           # the same tiles going round the CTAs
    assert rounds == large
    if tiles == 3:
        ref, _, sums = ir_eval.run_graph(ir, prob, dtype, num_threads=4, want_abs_sums=True)
        got, _ = run_gpu(ext, ir, prob, dtype)
        assert_outputs_match(ir, got, ref, sums, dtype, what=f"{gname} large")


@pytest.mark.parametrize("gname,dt,threads,ipt,edges", LARGE)
@pytest.mark.parametrize("bits", [32, 64])
def test_large_launches_without_whole_rows(gname, dt, threads, ipt, edges, bits):
    """A row of 40 edges, one of 900 and one of 20 000 among rows of three: the loop with carries, which large tiles make slower.  Both
    kinds give the oracle's sums; the plan's look at the rows brings the usual one."""
    ir, dtype = graphs.ALL_GRAPHS[gname](), np.dtype(dt)
    rows = 3 * small_limit(ir, dtype) // (2 * edges + 2) + 1000
    lengths = np.full(rows, edges)
    lengths[[100, rows // 2, rows - 7]] = [40, 900, 20_000]
    prob = with_lengths(ir, lengths.tolist(), 223, dtype)
    ref, _, sums = ir_eval.run_graph(ir, prob, dtype, num_threads=4, want_abs_sums=True)
    for longest_row in (None, 0, 32):
        ext = GraphExtension(ir, random_gather=False, longest_row=longest_row)
        got, _ = run_gpu(ext, ir, prob, dtype, offsets_dtype=np.int32 if bits == 32 else np.int64)
        ext.check()
        assert not ext.planned_whole_rows() and longest_row_of(ext) == 0
        assert (header_word(ext, 10) > 3 * default_tile(ir, dtype) // 2) == (longest_row == 32)
        assert_outputs_match(ir, got, ref, sums, dtype, what=f"{gname} large, long rows")


@pytest.mark.parametrize("gname,dt,held", [("rusanov", "float64", {2: 0, 3: 1, 4: 1, 5: 0}), ("rusanov", "float32", {2: 0, 3: 1, 4: 1, 5: 0}),
                                           ("swe_delta", "float64", {2: 0, 3: 1, 4: 1, 5: 0}), ("spring_mass", "float64", {5: 0, 6: 1, 8: 1, 9: 0}),
                                           ("spring_mass", "float32", {6: 0, 7: 1, 8: 1, 9: 0})])
def test_rows_of_which_the_large_tiles_hold_too_few_or_too_many(gname, dt, held):
    """Seven (words of four edges: 8.5) to eleven rows a tile for ten threads."""
    ir, dtype = graphs.ALL_GRAPHS[gname](), np.dtype(dt)
    for edges, large in held.items():
        rows = 2 * (small_limit(ir, dtype) + 4000) // (edges + 1)
        prob = with_lengths(ir, [edges] * rows, 227, dtype)
        ext = GraphExtension(ir, random_gather=False)
        run_gpu(ext, ir, prob, dtype)
        assert (header_word(ext, 10) > default_tile(ir, dtype)) == large, edges


@pytest.mark.parametrize("gname,dt,lengths,tiles,suits", [
    ("spring_mass", "float32", [8], 3.0, True), ("spring_mass", "float32", [8] * 9999 + [32], 3.0, True), ("spring_mass", "float32", [8] * 9999 + [33], 3.0, False),
    ("spring_mass", "float32", [7, 8, 9], 3.0, True), ("spring_mass", "float32", [7] * 9999 + [28], 3.0, True), ("spring_mass", "float32", [7] * 9999 + [29], 3.0, False),
    ("spring_mass", "float64", [8], 3.5, True), ("spring_mass", "float64", [8] * 9600 + [9] * 32, 3.5, True), ("spring_mass", "float64", [8] * 63 + [9], 3.5, False),
    ("spring_mass", "float64", [6, 10], 3.5, False), ("rusanov", "float64", [3] * 999 + [12], 2.9, True), ("rusanov", "float64", [3] * 999 + [13], 2.9, False),
    ("rusanov", "float64", [0, 6, 3], 2.9, True), ("rusanov", "float32", [0, 6, 3], 3.0, True), ("swe_delta", "float64", [2, 5], 3.0, True),
    ("swe_delta", "float64", [2, 4], 17.0, True), ("swe_delta", "float64", [3] * 19 + [2], 17.0, False), ("rusanov", "float32", [3] * 99 + [2], 17.0, True),
    ("rusanov", "float32", [3] * 19 + [2], 17.0, False)])
@pytest.mark.parametrize("bits", [32, 64])
def test_rows_that_suit_large_tiles(gname, dt, lengths, tiles, suits, bits):
    """Whole rows, none of more than four times the mean and no more of them a tile than threads; in 8-byte values graphs that read their
    edge tensors in place take rows of one length only.  (``tiles`` a CTA, of which the last part is the margin.)"""
    ir, dtype = graphs.ALL_GRAPHS[gname](), np.dtype(dt)
    _, _, threads, ipt, _ = next(c for c in LARGE if c[:2] == (gname, dt))
    times = int((sms() * (threads - 1) * ipt * tiles - 50) / (sum(lengths) + len(lengths)))
    prob = with_lengths(ir, lengths * times, 251, dtype)
    ext = GraphExtension(ir, random_gather=False)
    run_gpu(ext, ir, prob, dtype, offsets_dtype=np.int32 if bits == 32 else np.int64)
    ext.check()
    assert ext.planned_whole_rows() == (max(lengths) <= 32) and (header_word(ext, 10) > 3 * default_tile(ir, dtype) // 2) == suits
    assert next(reversed(ext._plans.values())).desc.reserved >> 8 == (max(lengths) if suits else 0)


@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("skip", [0, 1, 2, 3, 4])
@pytest.mark.parametrize("last", [8, 9, 10, 11])
def test_words_of_four_edges_at_odd_places(bits, skip, last):
    """Rows that begin and end at any edge of a word of four, a last word that the arrays do not fill, edge tensors at any multiple of
    four bytes (an operator takes views), against the configuration that reads edge by edge."""
    ir, dtype = graphs.spring_mass_graph(), np.dtype("float32")
    lengths = [8, 7, 9, 8, 5, 11, 0, 16] * ((small_limit(ir, dtype) + 5000) // 72) + [last]
    prob = with_lengths(ir, lengths, 229, dtype)
    non_gather, gathers, index_names = graphs.operator_signature(ir)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()

    def shifted(a):
        t = torch.full((a.size + skip,), float("nan"), device="cuda")
        t[skip:] = dev(a.astype(np.float32))
        return t[skip:]
    values = [shifted(prob.values[n]) for n in non_gather] + [dev(prob.values[n].astype(np.float32)) for n in gathers]
    indices = [dev(prob.indices[n]) for n in index_names]
    ro = dev(prob.row_offsets.astype(np.int32 if bits == 32 else np.int64))
    outs = []
    for max_ctas in (0, 4 * sms()):
        ext = GraphExtension(ir, max_ctas=max_ctas, longest_row=max(lengths))
        out = torch.full((prob.num_rows, 2), float("nan"), device="cuda")
        ext.launch_into(values, indices, ro, [out], prob.num_rows, prob.nnz, prob.num_cols)
        ext.check()
        assert (header_word(ext, 10) > default_tile(ir, dtype)) == (max_ctas == 0)
        outs.append(out.cpu().numpy().tobytes())
    assert outs[0] == outs[1]


@pytest.mark.parametrize("dt,tile", [("float64", 352 * 8), ("float32", 352 * 10)])
@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("lengths,large", [([27], True), ([21], True), ([32], True), ([20], False), ([33], False), ([30, 0, 32, 9, 31, 32, 28, 10], True),
                                           ([27] * 5000 + [40], True), ([25] * 3000 + [900, 0, 0], True)],
                         ids=["27", "21", "32", "20", "33", "uneven", "one_of_40", "long"])
def test_longer_rows_of_spmv(dt, tile, bits, lengths, large):
    """21 to 32 edges a row on average: batches of nine in two CTAs of 12 warps, unless a row is longer than 32."""
    ir, dtype = graphs.spmv_graph(), np.dtype(dt)
    times = int(2 * sms() * tile * 1.3 / (sum(lengths) + len(lengths))) + 1
    prob = with_lengths(ir, lengths * times, 233, dtype)
    items = prob.num_rows + prob.nnz
    each, longest = -(-items // (2 * sms() * tile)), max(lengths) if max(lengths) <= 32 else 0
    ref, _, sums = ir_eval.run_graph(ir, prob, dtype, num_threads=4, want_abs_sums=True)
    for known in (0, 32, None):
        ext = GraphExtension(ir, random_gather=False, longest_row=known)
        got, _ = run_gpu(ext, ir, prob, dtype, offsets_dtype=np.int32 if bits == 32 else np.int64)
        ext.check()
        assert longest_row_of(ext) == longest
        takes = large and (longest > 0 if known is None else known > 0)
        assert header_word(ext, 10) == (-(-items // (2 * sms() * each)) if takes else default_tile(ir, dtype))
        assert_outputs_match(ir, got, ref, sums, dtype, what=f"spmv {dt}")
    if large and max(lengths) <= 32:
        named, whole = launch(ir, prob, dtype, prob.num_cols, bits, max_ctas=4 * sms())
        rounds, _ = launch(ir, prob, dtype, 1 << 27, bits, ROUNDS)
        assert whole and [g.tobytes() for g in got] == named == rounds


@pytest.mark.parametrize("dt,tile", [("float64", 352 * 8), ("float32", 352 * 10)])
def test_a_tile_a_cta_of_longer_rows_keeps_the_other_configuration(dt, tile):
    ir, dtype = graphs.spmv_graph(), np.dtype(dt)
    for more, large in ((0, False), (28, True)):
        prob = with_lengths(ir, [27] * ((2 * sms() * tile + more) // 28), 239, dtype)
        ext = GraphExtension(ir, random_gather=False)
        run_gpu(ext, ir, prob, dtype)
        assert (header_word(ext, 10) != default_tile(ir, dtype)) == large


@pytest.mark.parametrize("gname,dt,edges,items", [("spring_mass", "float64", 8, (1_900_000, 2_250_000, 2_400_000, 3_010_000, 3_700_000)),
                                                  ("rusanov", "float64", 3, (1_320_000, 1_410_000)), ("swe_delta", "float64", 3, (1_320_000, 1_410_000)), ("spring_mass", "float32", 8, (2_800_000,))])
def test_last_turns_that_leave_warps_idle(gname, dt, edges, items):
    """215 of 1000 lanes without a row over up to four turns of a CTA's warps: 8-byte values of graphs that stage their edge tensors keep
    small CTAs.  The same bits in either form."""
    ir, dtype = graphs.ALL_GRAPHS[gname](), np.dtype(dt)
    _, _, threads, ipt, _ = next(c for c in LARGE if c[:2] == (gname, dt))
    for n in items:
        prob = with_lengths(ir, [edges] * (n // (edges + 1)), 257, dtype)
        ext = GraphExtension(ir, random_gather=False)
        got, _ = run_gpu(ext, ir, prob, dtype)
        ext.check()
        tiles = -(-n // (sms() * (threads - 1) * ipt))
        turns = -(-tiles * (-(-prob.num_rows // (32 * sms() * tiles))) // (threads // 32))
        full = gname == "spring_mass" or 1000 * prob.num_rows >= 785 * 32 * sms() * turns * (threads // 32)
        assert (header_word(ext, 10) > 3 * default_tile(ir, dtype) // 2) == full
        assert [g.tobytes() for g in got] == launch(ir, prob, dtype, prob.num_cols, 32, max_ctas=3 * sms())[0]
