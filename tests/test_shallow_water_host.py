"""Host side of the shallow-water step, without a GPU."""
import ctypes

import pytest

from flexspmv_b200 import shallow_water
from flexspmv_b200.binding import Desc, FlexSpmvError, PreparedLaunch, load_library


class FakePlan:
    def __init__(self):
        self._flag_view = [0]

    def status(self):
        return self._flag_view[0]


class FakeGraph:
    replays = 0

    def replay(self):
        self.replays += 1


def bare_launch(plan):
    launch = PreparedLaunch.__new__(PreparedLaunch)
    launch.ext = type("Ext", (), {"lib": load_library()})
    launch._plan = plan
    return launch


def bare_step(**attributes):
    step = shallow_water.ShallowWaterStep.__new__(shallow_water.ShallowWaterStep)
    step.__dict__.update(_step=None, _fused=None, _graph=FakeGraph(), **attributes)
    return step


@pytest.mark.parametrize("form", ["one", "four", "twelve"])
def test_replay_raises_where_an_earlier_step_failed(form):
    plan = FakePlan()
    step = bare_step()
    if form == "twelve":
        step._on_state, step._on_stage = (bare_launch(FakePlan()), bare_launch(FakePlan())), (bare_launch(FakePlan()), bare_launch(plan))
    else:
        step._fused = [bare_launch(plan) for _ in range(4)]
        if form == "one":
            step._step = bare_launch(plan)          # a launch on the four ones' plan
    step.replay()
    assert step._graph.replays == 1
    plan._flag_view[0] = -6
    with pytest.raises(FlexSpmvError, match="replay.*status -6"):
        step.replay()
    assert step._graph.replays == 1


@pytest.mark.parametrize("status,launches", [(-4, 4), (-3, 0), (1, 0)])
def test_only_a_launch_that_does_not_fit_is_replaced_by_four(status, launches):
    """FLEXSPMV_ERR_TOO_LARGE of the whole step; other errors are raised."""
    made = []

    class Refused:
        def launch(self):
            raise FlexSpmvError("refused", status)

    class Stage:
        def launch(self):
            made.append(1)

    step = bare_step(dt=1.0, _coef_dt=1.0)
    step._step, step._fused = Refused(), [Stage() for _ in range(4)]
    if launches:
        step.forward()
        assert step._step is None
    else:
        with pytest.raises(FlexSpmvError, match="refused"):
            step.forward()
    assert len(made) == launches


@pytest.mark.parametrize("cells,max_ctas,fits", [(40_000, 0, 1), (40_000, 1000, 1), (40_000, 21, 1), (40_000, 19, 0), (1900, 1, 1), (2100, 1, 0)])
def test_a_cap_on_the_ctas_leaves_each_more_cells(cells, max_ctas, fits):
    """About 1980 cells of three edges a CTA in fp64."""
    d = Desc(cells, 3 * cells, cells, 32, 0, max_ctas, 0)
    assert bool(load_library().flexspmv_swe_delta_rk_f64_step_fits(ctypes.byref(d))) == bool(fits)


def test_the_cells_of_a_cta():
    """step_fits: whole warps of cells, over 148 SMs where there is no device to ask."""
    for cells, max_ctas, share in ((101, 4, 32), (101, 1, 128), (1900, 1, 1920)):
        d = Desc(cells, 3 * cells, cells, 64, 0, max_ctas, 0)
        assert load_library().flexspmv_swe_delta_rk_f32_step_fits(ctypes.byref(d)) == share


@pytest.mark.parametrize("cells,most,longest,even", [(64, 192, 3, True), (64, 288, 6, True), (64, 289, 6, False), (64, 192, 7, False), (32, 96, 4, True),
                                                     (32, 96, 5, False), (160, 480, 10, True), (160, 480, 11, False), (320, 960, 32, True), (320, 1441, 4, False)])
def test_shares_of_cells(cells, most, longest, even):
    """On a mesh of 9000 cells with three edges each."""
    assert shallow_water.shares_are_even(cells, 9000, 27000, most, longest) == even


@pytest.mark.parametrize("dtype,size", [("f32", 4), ("f64", 8)])
def test_the_whole_step_refuses_arrays_that_overlap(dtype, size):
    """Checked before anything is enqueued, so that addresses which nothing reads will do.  -2: the arrays pass, the row offsets' address
    does not."""
    lib, cells = load_library(), 1000
    d = Desc(cells, 3 * cells, cells, 32, 0, 0, 0)
    need = ctypes.c_size_t()
    assert getattr(lib, f"flexspmv_swe_delta_rk_{dtype}_workspace_bytes")(ctypes.byref(d), ctypes.byref(need)) == 0
    step = getattr(lib, f"flexspmv_swe_delta_rk_{dtype}_step")
    far, coef = 1 << 20, (ctypes.c_double * 16)()

    def call(**places):
        at = {f"v{i}": far * (1 + i) for i in range(18)}
        at.update({f"o{i}": far * (31 + i) for i in range(6)}, v11=far * 4, v12=far * 5, v13=far * 6, v17=ctypes.addressof(coef))
        at.update(places)
        values = (ctypes.c_void_p * 18)(*[at[f"v{i}"] for i in range(18)])
        outputs = (ctypes.c_void_p * 6)(*[at[f"o{i}"] for i in range(6)])
        indices = (ctypes.c_void_p * 2)(far * 40, far * 41)
        return step(ctypes.byref(d), values, indices, ctypes.c_void_p(8), outputs, ctypes.c_void_p(far), need, None)

    last = (cells - 1) * size
    assert call() == -2
    for accepted in ({"v11": far * 50, "v12": far * 51, "v13": far * 52}, {"v14": far * 31}, {"o0": far * 20, "o1": far * 20 + cells * size},
                     {"v11": far * 50, "v12": far * 51, "v13": far * 52, "o3": far * 4}):
        assert call(**accepted) == -2
    for refused in ({"o0": far * 4}, {"o5": far * 5}, {"o1": far * 4 + last}, {"o3": far * 31}, {"o2": far * 16}, {"v15": far * 17}, {"v16": far * 6 + last},
                    {"v12": far * 4}, {"v11": far * 50, "v12": far * 51, "v13": far * 52, "o0": far * 4}):
        assert call(**refused) == -1, refused
