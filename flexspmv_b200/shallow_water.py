"""One time step of the reference's shallow-water model on the fused operators.

The reference model (shallow_water_equation/swe_main.py:12-146) is an ``easier`` module whose ``forward``
is a classical Runge-Kutta step; each of its four ``delta`` evaluations gathers h, uh, vh over the edges
(``gather_src`` / ``gather_dst``), blends them to face values, and scatters three flux sums per cell
(``scatter``) plus two wall terms on the boundary cells (``scatter_b``).  The reference replaces those
fused regions by generated operators and leaves the per-cell arithmetic to torch (about 60 element-wise
kernels per step).  ``ShallowWaterStep`` runs a stage as ONE launch: the ``swe_delta`` graph's kernel with the
stage's per-cell arithmetic -- wall terms, ``-(...)/area``, the Runge-Kutta update -- as what it does with a
cell's finished flux sums (csrc/flex_swe_rk.cuh), bound once with ``GraphExtension.prepare``.  Meshes whose
cells are too irregular for that kernel (a cell with more than 32 edges), and steps with operator objects of the
caller's, run a stage as three launches with the same results, bit for bit: ``swe_delta``, ``swe_boundary``,
``flexspmv_swe_rk_stage``.  Meshes that fit the chip (about 290 000 cells in fp64) run all four stages in one cooperative
launch (csrc/flex_swe_step.cuh), again with the same bits.  ``capture()`` records the whole step (1 launch, 4, or 12) into one
CUDA graph.

Edges must be sorted by destination cell and ``bcells`` ascending: both Reducers then see sorted indices,
which is what the merge-path kernels need (python_wrapper/dynamic_replace_submodule.py:20-41 makes the
same assumption when it converts COO rows to CSR offsets).
"""
from __future__ import annotations

from typing import Dict, Optional

import ctypes

import torch

from .binding import FlexSpmvError, GraphExtension, check, load_builtin
from .graphs import swe_delta_graph
from .python_wrapper.dynamic_replace_submodule import coo_rows_to_csr_ptr

_ERR_TOO_LARGE = -4          # FLEXSPMV_ERR_TOO_LARGE of include/flexspmv.h


def shares_are_even(cells: int, num_cells: int, num_edges: int, most: int, longest: int) -> bool:
    """No share of ``cells`` consecutive cells with more than half as many edges again as the mean, and no cell with more edges than
    its share hides (see ``ShallowWaterStep._shares_are_even``)."""
    if 2 * most * num_cells > 3 * cells * num_edges:
        return False
    return cells >= 320 or longest <= -(-num_edges // num_cells) * (1 + cells / 64)


class ShallowWaterStep:
    def __init__(self, mesh: Dict[str, torch.Tensor], dt: float = 0.005,
                 delta_ext: Optional[GraphExtension] = None, boundary_ext: Optional[GraphExtension] = None):
        """``mesh``: CUDA tensors named as the reference module's attributes -- src, dst (int32, sorted by dst),
        bcells (int32, ascending), alpha, sx, sy (per edge), bsx, bsy (per boundary cell), area, h, uh, vh (per
        cell).  h, uh, vh are advanced in place."""
        self.dt = float(dt)
        m = self.m = mesh
        dev = m["h"].device
        self.nc = int(m["h"].numel())
        self.ne = int(m["src"].numel())
        self.nbc = int(m["bcells"].numel())
        own = delta_ext is not None or boundary_ext is not None
        self.delta_ext = delta_ext or load_builtin("swe_delta")
        self.boundary_ext = boundary_ext or load_builtin("swe_boundary")
        self.ro = coo_rows_to_csr_ptr(m["dst"], self.nc)
        if self.ne < 2 ** 31 - self.nc:
            self.ro = self.ro.to(torch.int32)             # half the bytes to stream per stage
        self.ro_b = coo_rows_to_csr_ptr(m["bcells"], self.nc)
        dt_ = m["h"].dtype
        new = lambda k: [torch.empty(self.nc, dtype=dt_, device=dev) for _ in range(k)]
        self.stage = new(3)                               # the state the next delta is evaluated at
        self.acc = new(3)                                 # running sum of the increments
        self._graph: Optional[torch.cuda.CUDAGraph] = None
        self._step = None
        self._fused = None if own else self._bind_fused(new)
        if self._fused is not None:
            return
        self.red, self.red_b = new(3), new(2)             # the reducers' outputs
        self._on_state = self._bind(m["h"], m["uh"], m["vh"])
        self._on_stage = self._bind(*self.stage)
        ptrs = lambda ts: (ctypes.c_void_p * len(ts))(*[t.data_ptr() for t in ts])
        self._p_red, self._p_red_b, self._p_acc, self._p_stage = ptrs(self.red), ptrs(self.red_b), ptrs(self.acc), ptrs(self.stage)
        self._p_x = ptrs([m["h"], m["uh"], m["vh"]])
        self.delta_ext.lib.flexspmv_swe_rk_stage.restype = ctypes.c_int

    def _coefficients(self):
        """(c, first, last) of the four stages at the present ``dt``: the next state is x + c d, the last one adds dt / 6
        of the sum."""
        return ((0.5 * self.dt, 1, 0), (0.5 * self.dt, 0, 0), (self.dt, 0, 0), (0.0, 0, 1))

    def _set_coefficients(self):
        self._coef_dt = float(self.dt)
        self._coef.copy_(torch.tensor([[c, self._coef_dt / 6, first, last] for c, first, last in self._coefficients()], device="cpu",
                                      dtype=self._coef.dtype))

    def _bind_fused(self, new):
        """The four launches of a step, or None when the mesh was not planned with whole rows.  A stage reads one
        state and writes the next, and neighbours read what a cell wrote, so the states alternate between two sets
        of arrays."""
        m, dt_ = self.m, self.m["h"].dtype
        ext = GraphExtension(swe_delta_graph(), symbol_prefix="swe_delta_rk")
        cells = m["bcells"].to(torch.int32).contiguous()
        starts = torch.arange(0, self.nc + 32, 32, device=cells.device, dtype=torch.int32)
        self._wall_start = torch.searchsorted(cells, starts, right=False).to(torch.int32)
        other = new(3)
        state = [m["h"], m["uh"], m["vh"]]
        launches = []
        # a row for each stage, in host memory that is read when a launch is made; both forms of the step read the same rows
        self._coef = torch.empty(4, 4, dtype=dt_, device="cpu")
        self._set_coefficients()
        for k in range(4):
            src = state if k == 0 else (self.stage if k % 2 else other)
            dst = other if k % 2 else self.stage          # the last stage writes the state itself
            values = [m["alpha"], m["sx"], m["sy"]] + src + [m["area"], m["bsx"], m["bsy"], self._wall_start, cells] + state + self.acc + [self._coef[k]]
            launches.append(ext.prepare(values, [m["src"], m["dst"]], self.ro, dst, self.nc, self.ne, self.nc))
            if k == 0:
                longest = ext.longest_row_of(launches[0])
                if longest == 0 and not ext.planned_whole_rows():       # (a mesh without edges has whole rows, too)
                    return None
        # meshes that fit the chip in even shares: the four stages in one launch (csrc/flex_swe_step.cuh)
        values = [m["alpha"], m["sx"], m["sy"]] + state + [m["area"], m["bsx"], m["bsy"], self._wall_start, cells] + state + self.acc + [self._coef]
        step = ext.prepare_step(values, [m["src"], m["dst"]], self.ro, self.stage + other, self.nc, self.ne, self.nc)
        if step is not None and self._shares_are_even(step.rows_a_cta, longest):
            self._step = step
        return launches

    def _shares_are_even(self, cells: int, longest: int) -> bool:
        """Whether the whole-step launch is the faster form with ``cells`` consecutive cells a CTA and ``longest`` edges in a cell at most (one
        look at the row offsets when the model is bound).  Its stages wait for the CTA with the most edges, and a cell's edges are a chain of gathers that takes
        0.23 us an edge and step of each stage, 0.14 in the four launches; with more cells a CTA there is other work to hide it.
        us a step, one launch / four, fp64, n x n squares: 330^2 with 1000 cells of 25 edges side by side 457 / 92, 700 of 8 (the
        largest share 1.8 times the mean) 64 / 60, half of the cells with 6 (1.3) 39 / 53 on 260^2; one cell of 25 on 64^2 (64 a CTA)
        41 / 37, on 101^2 (160) 37 / 35, on 160^2 (352) 37 / 43; of 12 on 64^2 29 / 25, on 101^2 25 / 29; six cells of 5 on 40^2 (32)
        25 / 23.  fp32 alike (330^2 174 / 56; one of 25 on 64^2 35 / 29)."""
        begins = self.ro[:self.nc:cells].tolist()
        most = max(e - b for b, e in zip(begins, begins[1:] + [self.ne]))
        return shares_are_even(cells, self.nc, self.ne, most, longest)

    def _bind(self, h, uh, vh):
        m = self.m
        d = self.delta_ext.prepare([m["alpha"], m["sx"], m["sy"], h, uh, vh], [m["src"], m["dst"]], self.ro,
                                   self.red, self.nc, self.ne, self.nc)
        b = self.boundary_ext.prepare([m["bsx"], m["bsy"], h], [m["bcells"]], self.ro_b, self.red_b, self.nc,
                                      self.nbc, self.nc)
        return d, b

    def _stage(self, c: float, first: bool, last: bool) -> None:
        fn = self.delta_ext.lib.flexspmv_swe_rk_stage
        st = fn(ctypes.c_int32(self.m["h"].element_size()), self._p_red, self._p_red_b,
                ctypes.c_void_p(self.m["area"].data_ptr()), self._p_x, self._p_acc, self._p_stage,
                ctypes.c_double(c), ctypes.c_double(self.dt / 6), ctypes.c_int64(self.nc),
                ctypes.c_int32(int(first)), ctypes.c_int32(int(last)),
                ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        check(self.delta_ext.lib, st, "swe_rk_stage")

    def forward(self) -> None:
        """swe_main.py:121-146: four delta evaluations (:86-119), each followed by its stage update.  ``dt`` may be set
        between calls (a step captured by ``capture`` keeps the one it was captured with)."""
        if self._fused is not None:
            if float(self.dt) != self._coef_dt:
                self._set_coefficients()
            if self._step is not None:
                try:
                    return self._step.launch()
                except FlexSpmvError as error:
                    if error.status != _ERR_TOO_LARGE:
                        raise
                    self._step = None            # the context does not hold all of its CTAs at once; nothing was enqueued
            for launch in self._fused:
                launch.launch()
            return
        for k, (c, first, last) in enumerate(self._coefficients()):
            bound = self._on_state if k == 0 else self._on_stage
            bound[0].launch()
            bound[1].launch()
            self._stage(c, first=bool(first), last=bool(last))

    __call__ = forward

    # -- CUDA graph --------------------------------------------------------------------------------------
    def capture(self) -> None:
        """Records one step into a CUDA graph (after one eager step on a side stream to warm the allocator);
        ``replay()`` then advances the state by one step per call.  The warm-up step is undone."""
        saved = [self.m[k].clone() for k in ("h", "uh", "vh")]
        side = torch.cuda.Stream()          # warm-up and capture on one stream: the prepared launches are
        side.wait_stream(torch.cuda.current_stream())   # already ordered after their plans there
        with torch.cuda.stream(side):
            self.forward()
            for k, v in zip(("h", "uh", "vh"), saved):
                self.m[k].copy_(v)
        side.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=side):
            self.forward()
        self._graph = g

    def replay(self) -> None:
        """One captured step.  Raises FlexSpmvError, as ``forward`` does, where an earlier one failed on the device: the launches
        of a graph leave a workspace whose status is raised without doing anything, and the state would stand still."""
        if self._graph is None:
            raise RuntimeError("capture() first")
        self._raise_if_failed("replay")
        self._graph.replay()

    # -- errors --------------------------------------------------------------------------------------------
    def _raise_if_failed(self, what: str) -> None:
        launches = self._fused if self._fused is not None else self._on_state + self._on_stage
        for launch in launches:             # (those of one plan share its status, the whole step's launch among them)
            if launch.failed():
                launch.raise_if_failed(what)

    def check(self) -> None:
        """Waits for the steps enqueued so far and raises FlexSpmvError if one of them gave up on the device (a bounded wait
        ran out).  The state is undefined then: cells may be at different stages of a step."""
        torch.cuda.synchronize(self.m["h"].device)
        self._raise_if_failed("check")


def assemble_shallow_water(mesh: Dict[str, torch.Tensor]) -> Dict[str, torch.Tensor]:
    """The reference's mesh assembler (``assemble_shallow_water``, shallow_water_equation/assemble_shallow_water.py:
    251-291) on the fused operators, with tensors where the reference reads and writes HDF5 data sets.

    ``mesh``: CUDA tensors named as the mesh file's data sets -- points (np, 2) float64, cells (nc, 3), src, dst (ne,),
    bcells (nbc,), bpoints (nbc, 2), all integer.  Returns what the reference saves: src_p0..2, dst_p0..2, cells_p0..2,
    bp0..1 (int64) and x, y, area, sx, sy, bsx, bsy, h, alpha (float64).  Four launches: the components collector's
    gathers (``swe_components``), then the initializer's per-edge, per-cell and boundary parts (``swe_init_edges``,
    ``swe_init_cells``, ``swe_init_boundary``); the column slices the collector also copies (:74-78) are torch slices.
    """
    points = mesh["points"].contiguous()
    dev = points.device
    cells = mesh["cells"].to(torch.int64).contiguous()
    nc, ne, nbc, npnt = int(cells.shape[0]), int(mesh["src"].numel()), int(mesh["bcells"].numel()), int(points.shape[0])
    i32 = lambda t: t.to(torch.int32).contiguous()
    dummy = torch.zeros(1, dtype=torch.int32, device=dev)      # row_end_offsets of a graph without a reducer
    out: Dict[str, torch.Tensor] = {}

    # ShallowWaterMeshComponentsCollector.forward (:62-78)
    comp = [torch.zeros(ne, dtype=torch.int64, device=dev) for _ in range(6)]
    load_builtin("swe_components").launch_into(comp + [cells], [i32(mesh["src"]), i32(mesh["dst"])], dummy, [], 0, ne, nc)
    for i in range(3):
        out[f"src_p{i}"], out[f"dst_p{i}"] = comp[i], comp[3 + i]
        out[f"cells_p{i}"] = cells[:, i].clone()
    bpoints = mesh["bpoints"].to(torch.int64)
    for i in range(2):
        out[f"bp{i}"] = bpoints[:, i].clone()

    # ShallowWaterInitializer.forward (:178-248)
    f64 = lambda n_: torch.zeros(n_, dtype=torch.float64, device=dev)
    for k in ("sx", "sy", "alpha"):
        out[k] = f64(ne)
    load_builtin("swe_init_edges").launch_into([out["sx"], out["sy"], out["alpha"], points],
                                               [i32(c) for c in comp], dummy, [], 0, ne, npnt)
    for k in ("area", "x", "y", "h"):
        out[k] = f64(nc)
    load_builtin("swe_init_cells").launch_into([out["area"], out["x"], out["y"], out["h"], points],
                                               [i32(out[f"cells_p{i}"]) for i in range(3)], dummy, [], 0, nc, npnt)
    centroid = torch.stack([out["x"], out["y"]], dim=1).contiguous()
    out["bsx"], out["bsy"] = f64(nbc), f64(nbc)
    load_builtin("swe_init_boundary").launch_into([out["bsx"], out["bsy"], points, centroid],
                                                  [i32(out["bp0"]), i32(out["bp1"]), i32(mesh["bcells"])], dummy, [], 0, nbc, npnt)
    return out
