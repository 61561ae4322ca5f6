"""The large configuration of the row-mode graphs (GraphApi::use_big): the sizes on both sides of its rule, tiles of equal number
and of the largest size, both orders of the tiles, plans with and without whole rows -- each against the configuration that a caller
who names a number of CTAs gets, bit for bit where sums run left to right in both, and against the oracle."""
import numpy as np
import pytest
import torch

from flexspmv_b200 import graphs
from flexspmv_b200.binding import GraphExtension
from oracle import ir_eval
from parity import assert_outputs_match
from test_gpu_launch_sizes import ROUNDS, default_tile, header_word, launch, run_gpu, with_lengths

pytestmark = pytest.mark.gpu

LARGE = [("rusanov", "float64", 736), ("rusanov", "float32", 992), ("swe_delta", "float64", 736)]


def sms():
    return torch.cuda.get_device_properties(0).multi_processor_count


def small_limit(ir, dtype):
    """Items up to which a launch of short rows takes the kernel without stages: 9 tiles for four CTAs, of which an SM holds three
    or four."""
    return 9 * sms() * (3 if dtype == np.float64 else 4) * default_tile(ir, dtype) // 4


@pytest.mark.parametrize("gname,dt,threads", LARGE)
@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("tiles,lengths", [(0, [3]), (1, [3]), (3, [4, 0, 4, 3, 5]), (5, [2, 4]), (16, [3]), (17, [3])],
                         ids=["small", "above", "uneven", "five", "sixteen", "seventeen"])
def test_large_launches_equal_those_of_the_other_configuration(gname, dt, threads, bits, tiles, lengths):
    ir, dtype = graphs.ALL_GRAPHS[gname](), np.dtype(dt)
    tile = threads * 4 - 4
    if tiles > 5 and (bits == 64 or (gname, dt) != ("rusanov", "float64")):
        pytest.skip("one graph and width at the large sizes")
    # the last small launch and the first one that is not; up to `tiles` tiles a CTA
    items = small_limit(ir, dtype) + (4 if tiles else 0) if tiles < 2 else sms() * tile * tiles - 7 + (60 if tiles == 17 else 0)
    rows = items // (sum(lengths) // len(lengths) + 1) // len(lengths) * len(lengths)
    prob = with_lengths(ir, lengths * (rows // len(lengths)), 211, dtype)
    items = prob.num_rows + prob.nnz
    ext = GraphExtension(ir, random_gather=False)
    run_gpu(ext, ir, prob, dtype, offsets_dtype=np.int32 if bits == 32 else np.int64)
    ext.check()
    each, took = -(-items // (sms() * tile)), header_word(ext, 10)
    if tiles == 0:
        assert took == default_tile(ir, dtype)
        return
    assert took == (-(-items // (sms() * each)) if each <= 16 else tile)
    large, whole = launch(ir, prob, dtype, prob.num_cols, bits)
    named, also = launch(ir, prob, dtype, prob.num_cols, bits, max_ctas=3 * sms())
    assert whole and also and large == named
    rounds, _ = launch(ir, prob, dtype, 1 << 27, bits, ROUNDS)           # the same tiles going round the CTAs
    assert rounds == large
    if tiles == 3:
        ref, _, sums = ir_eval.run_graph(ir, prob, dtype, num_threads=4, want_abs_sums=True)
        got, _ = run_gpu(ext, ir, prob, dtype)
        assert_outputs_match(ir, got, ref, sums, dtype, what=f"{gname} large")


@pytest.mark.parametrize("gname,dt,threads", LARGE)
@pytest.mark.parametrize("bits", [32, 64])
def test_large_launches_without_whole_rows(gname, dt, threads, bits):
    """A row of 40 edges, one of 900 and one of 20 000 among rows of three: the loop with carries, in tiles of both kinds."""
    ir, dtype = graphs.ALL_GRAPHS[gname](), np.dtype(dt)
    rows = small_limit(ir, dtype) // 4
    lengths = np.full(rows, 3)
    lengths[[100, rows // 2, rows - 7]] = [40, 900, 20_000]
    prob = with_lengths(ir, lengths.tolist(), 223, dtype)
    ext = GraphExtension(ir, random_gather=False)
    got, _ = run_gpu(ext, ir, prob, dtype, offsets_dtype=np.int32 if bits == 32 else np.int64)
    ext.check()
    assert not ext.planned_whole_rows() and header_word(ext, 10) > 3 * default_tile(ir, dtype) // 2
    ref, _, sums = ir_eval.run_graph(ir, prob, dtype, num_threads=4, want_abs_sums=True)
    assert_outputs_match(ir, got, ref, sums, dtype, what=f"{gname} large, long rows")


@pytest.mark.parametrize("gname,dt,threads", LARGE)
def test_rows_of_which_the_large_tiles_hold_too_few_or_too_many(gname, dt, threads):
    """Seven to eleven rows a tile for ten threads: three or four edges a row (of 4 items a thread)."""
    ir, dtype = graphs.ALL_GRAPHS[gname](), np.dtype(dt)
    for edges, large in ((2, False), (3, True), (4, True), (5, False)):
        rows = (small_limit(ir, dtype) + 4000) // (edges + 1)
        prob = with_lengths(ir, [edges] * rows, 227, dtype)
        ext = GraphExtension(ir, random_gather=False)
        run_gpu(ext, ir, prob, dtype)
        assert (header_word(ext, 10) > default_tile(ir, dtype)) == large, edges
