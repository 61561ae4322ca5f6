"""The shallow-water step with the stage arithmetic behind the flux sums (one launch a stage) against the same step as
three launches a stage: the same operations in the same order, so the same bits."""
import numpy as np
import pytest
import torch

from flexspmv_b200 import graphs, problems
from flexspmv_b200.binding import FlexSpmvError, GraphExtension, load_builtin, load_library
from flexspmv_b200.shallow_water import ShallowWaterStep

pytestmark = pytest.mark.gpu
TILE, SMALL, ROUNDS = 1, 2, 3      # FLEXSPMV_KERNEL_* of include/flexspmv.h


def mesh_of(n, dtype, split_walls):
    m = {k: v for k, v in problems.swe_model_inputs(n).items() if k != "row_offsets"}
    if split_walls == "everywhere":      # 1 to 3 records on most cells, none on some, up to 96 in a group of 32 cells
        cells = m["h"].size
        counts = np.random.default_rng(5).choice([0, 1, 2, 3], cells, p=[0.1, 0.2, 0.2, 0.5])
        m["bcells"] = np.repeat(np.arange(cells), counts).astype(m["bcells"].dtype)
        m["bsx"], m["bsy"] = np.random.default_rng(7).uniform(-1e-3, 1e-3, (2, m["bcells"].size))
    elif split_walls:      # a wall record per face: cells with several come several times, ascending
        keep = np.repeat(np.arange(m["bcells"].size), np.where(np.arange(m["bcells"].size) % 3 == 0, 3, 1))
        m["bcells"] = m["bcells"][keep]
        m["bsx"], m["bsy"] = 0.3 * m["bsx"][keep], 0.7 * m["bsy"][keep]
    cast = lambda v: v.astype(dtype) if v.dtype.kind == "f" else v
    return {k: torch.from_numpy(np.ascontiguousarray(cast(v))).cuda() for k, v in m.items()}


@pytest.mark.parametrize("n", [1, 3, 16, 33, 97])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("split_walls", [False, True, "everywhere"])
def test_fused_stage_equals_three_launches(n, dtype, split_walls):
    dt = 0.05 / n
    a, b = mesh_of(n, dtype, split_walls), mesh_of(n, dtype, split_walls)
    fused = ShallowWaterStep(a, dt=dt)
    apart = ShallowWaterStep(b, dt=dt, delta_ext=load_builtin("swe_delta"), boundary_ext=load_builtin("swe_boundary"))
    assert apart._fused is None
    if n >= 16:
        assert fused._fused is not None      # a tile of a few cells leaves most of a warp idle: either way then
        fused.capture()
    for k in range(3):
        fused.replay() if n >= 16 else fused.forward()
        apart.forward()
    torch.cuda.synchronize()
    for name in ("h", "uh", "vh"):
        assert torch.isfinite(a[name]).all()
        assert torch.equal(a[name], b[name]), name


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_the_time_step_may_change_between_eager_steps(dtype):
    """A program that sets ``dt`` from its state: every step takes the present one, in either form."""
    a, b = mesh_of(33, dtype, False), mesh_of(33, dtype, False)
    fused = ShallowWaterStep(a, dt=1e-3)
    apart = ShallowWaterStep(b, dt=1e-3, delta_ext=load_builtin("swe_delta"), boundary_ext=load_builtin("swe_boundary"))
    assert fused._fused is not None and apart._fused is None
    for dt in (None, 2e-3, 0.5e-3, 0.5e-3, 1e-3):
        start = a["h"].clone()
        for step in (fused, apart):
            if dt is not None:
                step.dt = dt
            step.forward()
        assert not torch.equal(a["h"], start)
        for name in ("h", "uh", "vh"):
            assert torch.isfinite(a[name]).all() and torch.equal(a[name], b[name]), (dt, name)
    fused.capture()                      # the captured step keeps the time step it was captured with
    fused.dt = 5e-3
    fused.replay()
    apart.forward()
    for name in ("h", "uh", "vh"):
        assert torch.equal(a[name], b[name]), name


def mesh_with_a_long_row(n):
    m = mesh_of(n, np.float64, False)
    src, dst = m["src"], m["dst"]
    many = torch.full((40,), 5, dtype=torch.int32, device="cuda")          # 40 more edges into cell 7
    order = torch.argsort(torch.cat([dst, many + 2]).long(), stable=True)
    for k, extra in (("src", many), ("dst", many + 2)):
        m[k] = torch.cat([m[k], extra])[order].contiguous()
    for k in ("alpha", "sx", "sy"):
        m[k] = torch.cat([m[k], torch.full((40,), 0.25, dtype=torch.float64, device="cuda") * (0.0 if k != "alpha" else 1.0)])[order].contiguous()
    return m


def test_a_cell_with_many_edges_takes_three_launches():
    m = mesh_with_a_long_row(24)
    step = ShallowWaterStep(m, dt=1e-3)
    assert step._fused is None
    step.forward()
    torch.cuda.synchronize()
    assert torch.isfinite(m["h"]).all()


@pytest.mark.parametrize("max_ctas", [0, 1])      # one tile a CTA, and more tiles than a CTA has stages
def test_the_epilogue_refuses_a_plan_without_whole_rows(max_ctas):
    """The launch leaves at the header, before any copy: the status is "not planned" (no wait ran out), nothing is written."""
    m = mesh_with_a_long_row(48)
    nc, ne = m["h"].numel(), m["src"].numel()
    ext = GraphExtension(graphs.swe_delta_graph(), symbol_prefix="swe_delta_rk", max_ctas=max_ctas)
    ro = torch.searchsorted(m["dst"], torch.arange(nc + 1, dtype=torch.int32, device="cuda")).to(torch.int32)
    walls = torch.searchsorted(m["bcells"], torch.arange(0, nc + 32, 32, dtype=torch.int32, device="cuda")).to(torch.int32)
    state = [m[k] for k in ("h", "uh", "vh")]
    before = [t.clone() for t in state]
    acc, out = ([torch.full((nc,), float("nan"), dtype=torch.float64, device="cuda") for _ in range(3)] for _ in range(2))
    coef = torch.tensor([1e-3, 1e-3, 0.0, 1.0], dtype=torch.float64)
    values = [m["alpha"], m["sx"], m["sy"]] + state + [m["area"], m["bsx"], m["bsy"], walls, m["bcells"]] + state + acc + [coef]
    launch = ext.prepare(values, [m["src"], m["dst"]], ro, out, nc, ne, nc)
    assert not ext.planned_whole_rows()
    launch.launch()
    with pytest.raises(FlexSpmvError, match="status -7"):
        ext.check()
    assert all(torch.equal(a, b) for a, b in zip(state, before))
    assert all(torch.isnan(t).all() for t in acc + out)


def run_stage(m, start, sums, bits, first, last, max_ctas, vertices=None, tiles=None):
    """One stage through the C ABI: the kernel that the launch took, state, sums and next state as bytes.  ``tiles``: takes the items of
    the plan's tiles."""
    nc, ne, V = m["h"].numel(), m["src"].numel(), m["h"].dtype
    ro = torch.searchsorted(m["dst"], torch.arange(nc + 1, dtype=torch.int32, device="cuda")).to(torch.int32 if bits == 32 else torch.int64)
    walls = torch.searchsorted(m["bcells"], torch.arange(0, nc + 32, 32, dtype=torch.int32, device="cuda")).to(torch.int32)
    coef = torch.tensor([1e-3, 2e-3, first, last], dtype=V)
    ext = GraphExtension(graphs.swe_delta_graph(), symbol_prefix="swe_delta_rk", max_ctas=max_ctas)
    state, acc = [t.clone() for t in start], [t.clone() for t in sums]
    stage = [t.clone() for t in start]            # what the fluxes are taken of
    out = [torch.full((nc,), float("nan"), dtype=V, device="cuda") for _ in range(3)]
    values = [m["alpha"], m["sx"], m["sy"]] + stage + [m["area"], m["bsx"], m["bsy"], walls, m["bcells"]] + state + acc + [coef]
    launch = ext.prepare(values, [m["src"], m["dst"]], ro, out, nc, ne, vertices or nc)
    assert ext.planned_whole_rows()
    launch.launch()
    kernel = load_library().flexspmv_debug_last_kernel()
    ext.check()
    if tiles is not None:
        tiles.append(int(launch._keep[-1][:256].cpu().numpy().view(np.int32)[10]))
    assert all(torch.equal(a, b) for a, b in zip(stage, start))
    return kernel, [t.cpu().numpy().tobytes() for t in state + acc + out]


def stage_inputs(dtype, split_walls, n=64):
    m = mesh_of(n, dtype, split_walls)
    g = torch.Generator(device="cuda")
    g.manual_seed(11)
    rand = lambda: torch.rand(m["h"].numel(), generator=g, device="cuda", dtype=m["h"].dtype)
    return m, [m[k] + 0.01 * rand() for k in ("h", "uh", "vh")], [rand() for _ in range(3)]


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("split_walls", [False, True, "everywhere"])
def test_every_form_of_the_stage_gives_the_same_bits(dtype, bits, split_walls):
    """One stage in place (the first, a middle and the last of a step) straight from global memory (the default grid), through stages
    (one CTA and five) and with tiles going round the CTAs (a descriptor that names many vertices)."""
    m, start, sums = stage_inputs(dtype, split_walls)
    for first, last in ((1.0, 0.0), (0.0, 0.0), (0.0, 1.0)):
        results = []
        for max_ctas, vertices, kernel in ((0, None, SMALL), (1, None, TILE), (5, None, TILE), (1, 1 << 27, ROUNDS), (5, 1 << 27, ROUNDS)):
            taken, got = run_stage(m, start, sums, bits, first, last, max_ctas, vertices)
            assert taken == kernel
            results.append(got)
        assert all(r == results[0] for r in results[1:]), (first, last)


@pytest.mark.parametrize("dtype,max_ctas,kernel", [(np.float64, 21, SMALL), (np.float64, 23, TILE), (np.float32, 13, SMALL)])
def test_a_second_cell_a_thread_against_a_second_tile(dtype, max_ctas, kernel):
    """8192 cells, in fp64 43 tiles: where a thread has two cells and a CTA of 23 has two tiles the stages are kept, where one of 21 has
    three they are not.  In fp32 they are not kept either way."""
    m, start, sums = stage_inputs(dtype, False)
    taken, got = run_stage(m, start, sums, 32, 0.0, 0.0, max_ctas)
    assert taken == kernel and got == run_stage(m, start, sums, 32, 0.0, 0.0, 1)[1]


@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("split_walls", [False, "everywhere"])
def test_stages_in_large_tiles(bits, split_walls):
    """fp64 on 231 200 cells: large tiles, in a CTA's own run and going round the CTAs one by one, against the usual ones (a descriptor that names
    the CTAs)."""
    m, start, sums = stage_inputs(np.float64, split_walls, 340)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for first, last in ((1.0, 0.0), (0.0, 0.0), (0.0, 1.0)):
        results, tiles = [], []
        for max_ctas, vertices, kernel in ((0, None, TILE), (0, 1 << 27, ROUNDS), (3 * sms, None, TILE), (3 * sms, 1 << 27, TILE)):
            taken, got = run_stage(m, start, sums, bits, first, last, max_ctas, vertices, tiles)
            assert taken == kernel
            results.append(got)
        assert min(tiles[:2]) > 2 * max(tiles[2:])
        assert all(r == results[0] for r in results[1:]), (first, last)


@pytest.mark.parametrize("split_walls", [False, "everywhere"])
def test_a_step_in_large_tiles_that_go_round(split_walls):
    """460 800 cells, whose gathered states are beyond 10 MB: the kernel that large meshes take, against three launches a stage."""
    a, b = mesh_of(480, np.float64, split_walls), mesh_of(480, np.float64, split_walls)
    fused = ShallowWaterStep(a, dt=1e-5)
    apart = ShallowWaterStep(b, dt=1e-5, delta_ext=load_builtin("swe_delta"), boundary_ext=load_builtin("swe_boundary"))
    assert fused._fused is not None and fused._step is None and apart._fused is None
    for _ in range(2):
        fused.forward()
        assert load_library().flexspmv_debug_last_kernel() == ROUNDS
        apart.forward()
    assert int(fused._fused[0]._keep[-1][:256].cpu().numpy().view(np.int32)[10]) > 2000          # items a tile; 765 in the usual ones
    fused.check()
    for name in ("h", "uh", "vh"):
        assert torch.isfinite(a[name]).all() and torch.equal(a[name], b[name]), name
