"""A whole step of the shallow-water model in one cooperative launch against the launches of a stage each: the same bits."""
import ctypes

import numpy as np
import pytest
import torch

from flexspmv_b200 import graphs
from flexspmv_b200.binding import FlexSpmvError, GraphExtension, load_library
from flexspmv_b200.shallow_water import ShallowWaterStep
from test_gpu_swe_fused import mesh_of

pytestmark = pytest.mark.gpu
STEP = 7            # FLEXSPMV_KERNEL_STEP of include/flexspmv.h
STATE = ("h", "uh", "vh")


def sms():
    return torch.cuda.get_device_properties(0).multi_processor_count


def both(mesh, steps=2, dt=1e-4):
    """The state after some steps in one launch each, and in four; what ran last in the first form."""
    a, b = mesh, {k: v.clone() for k, v in mesh.items()}
    one, four = ShallowWaterStep(a, dt=dt), ShallowWaterStep(b, dt=dt)
    assert one._step is not None and four._fused is not None
    four._step = None
    for _ in range(steps):
        one.forward()
        kernel = load_library().flexspmv_debug_last_kernel()
        four.forward()
    torch.cuda.synchronize()
    return a, b, kernel


@pytest.mark.parametrize("n,walls", [(16, True), (33, "everywhere"), (97, False), (150, True), (200, "everywhere"), (270, False), (330, True)])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_one_launch_equals_four(n, walls, dtype):
    """One cell a thread and several rounds, in CTAs of both sizes; cells with no, one and several wall records."""
    a, b, kernel = both(mesh_of(n, dtype, walls), dt=0.01 / n)
    assert kernel == STEP
    for k in STATE:
        assert torch.isfinite(a[k]).all() and torch.equal(a[k], b[k]), k


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_edges_that_a_cta_cannot_keep(dtype, monkeypatch):
    """Cells of 25 edges side by side: their CTAs have more edges than shared memory was claimed for, and read the others in place.
    (Four launches are faster there, and are what such a mesh takes.)"""
    m = heavy_cells(mesh_of(160, dtype, True), torch.arange(20_000, 21_000), 22)
    assert ShallowWaterStep(m, dt=1e-4)._step is None
    monkeypatch.setattr(ShallowWaterStep, "_shares_are_even", lambda *a: True)
    a, b, kernel = both(m, dt=1e-4)
    assert kernel == STEP
    for k in STATE:
        assert torch.isfinite(a[k]).all() and torch.equal(a[k], b[k]), k


@pytest.mark.parametrize("n,cells,extra,even", [(64, 0, 0, True), (64, 1, 3, True), (64, 1, 4, False), (160, 1, 22, True), (330, 50, 22, True), (330, 700, 5, False)])
def test_cells_that_hold_the_others_up(n, cells, extra, even):
    """What decides is measured in ``_shares_are_even``; the step has the same bits in either form."""
    m = mesh_of(n, np.float64, True)
    if cells:
        m = heavy_cells(m, torch.arange(n * n, n * n + cells), extra)
    b = {k: v.clone() for k, v in m.items()}
    step, four = ShallowWaterStep(m, dt=1e-4), ShallowWaterStep(b, dt=1e-4)
    assert four._fused is not None and (step._step is not None) == even
    four._step = None
    step.forward()
    assert (load_library().flexspmv_debug_last_kernel() == STEP) == even
    four.forward()
    for k in STATE:
        assert torch.isfinite(m[k]).all() and torch.equal(m[k], b[k]), k


def heavy_cells(m, at, extra):
    """The mesh with ``extra`` more edges into each of the cells ``at``."""
    cells = m["h"].numel()
    many = at.to(torch.int32).repeat_interleave(extra).cuda()
    src = torch.randint(0, cells, (many.numel(),), generator=torch.Generator().manual_seed(3)).to(torch.int32).cuda()
    order = torch.argsort(torch.cat([m["dst"], many]).long(), stable=True)
    for k, extra in (("src", src), ("dst", many)):
        m[k] = torch.cat([m[k], extra])[order].contiguous()
    for k, c in (("alpha", 0.5), ("sx", 1e-7), ("sy", -2e-7)):
        m[k] = torch.cat([m[k], torch.full((many.numel(),), c, dtype=m[k].dtype, device="cuda")])[order].contiguous()
    return m


@pytest.mark.parametrize("n,fits", [(380, True), (400, False)])
def test_meshes_that_do_not_fit_take_four_launches(n, fits):
    """About 1980 cells of three edges an SM in fp64."""
    step = ShallowWaterStep(mesh_of(n, np.float64, False), dt=1e-5)
    assert step._fused is not None and (step._step is not None) == fits
    step.forward()
    assert (load_library().flexspmv_debug_last_kernel() == STEP) == fits


def bind(m, bits, max_ctas=0):
    """The step through the operator object with 32- or 64-bit offsets; scratch filled with NaN."""
    nc, ne, V = m["h"].numel(), m["src"].numel(), m["h"].dtype
    ro = torch.searchsorted(m["dst"], torch.arange(nc + 1, dtype=torch.int32, device="cuda")).to(torch.int32 if bits == 32 else torch.int64)
    walls = torch.searchsorted(m["bcells"], torch.arange(0, nc + 32, 32, dtype=torch.int32, device="cuda")).to(torch.int32)
    state = [m[k] for k in STATE]
    nan = lambda k: [torch.full((nc,), float("nan"), dtype=V, device="cuda") for _ in range(k)]
    coef = torch.tensor([[5e-5, 2e-5, 1, 0], [5e-5, 2e-5, 0, 0], [1e-4, 2e-5, 0, 0], [0, 2e-5, 0, 1]], dtype=V)
    values = [m["alpha"], m["sx"], m["sy"]] + state + [m["area"], m["bsx"], m["bsy"], walls, m["bcells"]] + state + nan(3) + [coef]
    ext = GraphExtension(graphs.swe_delta_graph(), symbol_prefix="swe_delta_rk", max_ctas=max_ctas)
    return ext, ext.prepare_step(values, [m["src"], m["dst"]], ro, nan(6), nc, ne, nc)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_offsets_of_either_width(dtype):
    a, b = mesh_of(70, dtype, True), mesh_of(70, dtype, True)
    for m, bits in ((a, 32), (b, 64)):
        ext, step = bind(m, bits)
        step.launch()
        ext.check()
    for k in STATE:
        assert torch.isfinite(a[k]).all() and torch.equal(a[k], b[k]), k


def test_a_barrier_that_stays_shut_runs_out():
    """A CTA that never arrives (testing aid): the others wait for a second, the status says so, the context stays usable, a later launch
    on the workspace writes nothing, and a newly planned one runs."""
    m = mesh_of(64, np.float64, False)
    before = {k: m[k].clone() for k in STATE}
    ext, step = bind(m, 32)
    lib, ws = load_library(), step._keep[-1]
    lib.flexspmv_debug_withhold_stage.restype = ctypes.c_int
    assert lib.flexspmv_debug_withhold_stage(ctypes.c_void_p(ws.data_ptr()), ctypes.c_uint32(1), None) == 0
    torch.cuda.synchronize()
    step.launch()
    with pytest.raises(FlexSpmvError, match="status -6"):
        ext.check()
    assert all(torch.equal(m[k], before[k]) for k in STATE)
    step._plan._flag_view[0] = 0                 # as if the host had not noticed
    step.launch()
    torch.cuda.synchronize()
    assert all(torch.equal(m[k], before[k]) for k in STATE)
    ext, step = bind(m, 32)
    step.launch()
    ext.check()
    assert not torch.equal(m["h"], before["h"]) and torch.isfinite(m["h"]).all()


def test_replays_after_a_run_out_raise():
    """The launches of a captured step return at once on a workspace whose status is raised; the host has the status word and says so,
    in ``replay`` and in ``check``."""
    m = mesh_of(64, np.float64, False)
    step = ShallowWaterStep(m, dt=1e-4)
    assert step._step is not None
    step.capture()
    step.replay()
    step.check()
    before = {k: m[k].clone() for k in STATE}
    lib = load_library()
    assert lib.flexspmv_debug_withhold_stage(ctypes.c_void_p(step._step._keep[-1].data_ptr()), ctypes.c_uint32(1), None) == 0
    torch.cuda.synchronize()
    step.replay()
    with pytest.raises(FlexSpmvError, match="check.*status -6"):
        step.check()
    for call in (step.replay, step.forward):
        with pytest.raises(FlexSpmvError, match="status -6"):
            call()
    assert all(torch.equal(m[k], before[k]) for k in STATE)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_the_time_step_reaches_both_forms(dtype):
    """``dt`` set after binding: the four launches of a step whose one launch is left out take it too."""
    a, b = mesh_of(40, dtype, True), mesh_of(40, dtype, True)
    one, four = ShallowWaterStep(a, dt=1e-3), ShallowWaterStep(b, dt=1e-3)
    assert one._step is not None
    four._step = None
    for dt in (1e-3, 2e-3, 0.5e-3):
        one.dt = four.dt = dt
        one.forward()
        four.forward()
        for k in STATE:
            assert torch.isfinite(a[k]).all() and torch.equal(a[k], b[k]), (dt, k)


@pytest.mark.parametrize("captured", [False, True])
def test_a_refused_launch_is_four_launches(captured):
    """A context with fewer SMs than the device refuses the cooperative launch (here: in its place a function that answers so)."""
    a, b = mesh_of(40, np.float64, True), mesh_of(40, np.float64, True)
    refused, other = ShallowWaterStep(a, dt=1e-3), ShallowWaterStep(b, dt=1e-3)
    asked = []
    refused._step._fn = lambda *args: asked.append(1) or -4
    if captured:
        refused.capture()
    for _ in range(2):
        refused.replay() if captured else refused.forward()
        other.forward()
    assert len(asked) == 1 and refused._step is None
    refused.check()
    for k in STATE:
        assert torch.isfinite(a[k]).all() and torch.equal(a[k], b[k]), k


@pytest.mark.parametrize("max_ctas", [1, 5, 33, 1000])
def test_the_descriptor_caps_the_ctas(max_ctas):
    a, b = mesh_of(30, np.float64, True), mesh_of(30, np.float64, True)
    (ext, capped), (_, usual) = bind(a, 32, max_ctas), bind(b, 32)
    for step in (capped, usual):
        step.launch()
    ext.check()
    assert capped.rows_a_cta == -(-(-(-1800 // min(max_ctas, 57, sms()))) // 32) * 32
    for k in STATE:
        assert torch.isfinite(a[k]).all() and torch.equal(a[k], b[k]), k


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_a_first_state_of_its_own(dtype):
    """The first stage's fluxes may be evaluated at other arrays than the ones that are advanced, as in four launches."""
    results = []
    for whole in (True, False):
        m = mesh_of(50, dtype, True)
        x = [m[k] + 0.01 * (i + 1) for i, k in enumerate(STATE)]
        m["h"], first = m["h"].clone(), [m[k] * 1.01 for k in STATE]
        nc, ne, V = m["h"].numel(), m["src"].numel(), m["h"].dtype
        ro = torch.searchsorted(m["dst"], torch.arange(nc + 1, dtype=torch.int32, device="cuda")).to(torch.int32)
        walls = torch.searchsorted(m["bcells"], torch.arange(0, nc + 32, 32, dtype=torch.int32, device="cuda")).to(torch.int32)
        stage, other, acc = ([torch.zeros(nc, dtype=V, device="cuda") for _ in range(3)] for _ in range(3))
        coef = torch.tensor([[5e-5, 2e-5, 1, 0], [5e-5, 2e-5, 0, 0], [1e-4, 2e-5, 0, 0], [0, 2e-5, 0, 1]], dtype=V)
        ext = GraphExtension(graphs.swe_delta_graph(), symbol_prefix="swe_delta_rk")
        values = lambda src, c: [m["alpha"], m["sx"], m["sy"]] + src + [m["area"], m["bsx"], m["bsy"], walls, m["bcells"]] + x + acc + [c]
        if whole:
            ext.prepare_step(values(first, coef), [m["src"], m["dst"]], ro, stage + other, nc, ne, nc).launch()
        else:
            for k in range(4):
                src, dst = first if k == 0 else (stage if k % 2 else other), other if k % 2 else stage
                ext.prepare(values(src, coef[k]), [m["src"], m["dst"]], ro, dst, nc, ne, nc).launch()
        ext.check()
        results.append(x)
    for a, b in zip(*results):
        assert torch.isfinite(a).all() and torch.equal(a, b)


@pytest.mark.parametrize("n", [60, 200])      # CTAs of which an SM holds two, and one
@pytest.mark.parametrize("captured", [False, True])
def test_two_models_on_two_streams(n, captured):
    """Whole-step launches of two models that meet on the chip: each waits for room for all of its CTAs, none for the other's."""
    meshes = [mesh_of(n, np.float64, True) for _ in range(3)]
    meshes[1]["h"] += 0.01
    start = {k: meshes[1][k].clone() for k in STATE}
    models = [ShallowWaterStep(m, dt=1e-5) for m in meshes[:2]]
    assert all(model._step is not None for model in models)
    if captured:
        for model in models:
            model.capture()
    streams = [torch.cuda.Stream() for _ in models]
    torch.cuda.synchronize()
    for _ in range(40):
        for model, stream in zip(models, streams):
            with torch.cuda.stream(stream):
                model.replay() if captured else model.forward()
    for model in models:
        model.check()
    alone = ShallowWaterStep(meshes[2], dt=1e-5)
    for m, state in ((meshes[0], None), (meshes[1], start)):
        if state is not None:
            for k in STATE:
                meshes[2][k].copy_(state[k])
        for _ in range(40):
            alone.forward()
        torch.cuda.synchronize()
        for k in STATE:
            assert torch.isfinite(m[k]).all() and torch.equal(m[k], meshes[2][k]), k


def test_launches_of_different_grids_on_one_workspace():
    """A descriptor's max_ctas may change from launch to launch: the barrier's counter, which stays in the workspace, does not know grids."""
    a, b = mesh_of(30, np.float64, True), mesh_of(30, np.float64, True)
    (ext, changing), (_, usual) = bind(a, 32), bind(b, 32)
    for max_ctas in (5, 0, 33, 1, 100, 0, 7, 7, 0):
        changing._desc.max_ctas = max_ctas
        changing.launch()
        usual.launch()
        ext.check()
    for k in STATE:
        assert torch.isfinite(a[k]).all() and torch.equal(a[k], b[k]), k
