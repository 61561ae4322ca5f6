"""The operator the reference's runtime wrapper calls: ``ext.merged_spmv_launch(*args)``.

The reference JIT-builds one pybind11 torch extension per fused graph whose single function
``merged_spmv_launch`` (cuda_template/merged_binding_template.cu:73-80) takes, positionally
(codegen/merged_gen_binding.py:65-78): the non-gather value inputs, the gather value inputs, one int32
index tensor per selector target, ``row_end_offsets`` (leading 0 included), ``num_rows``,
``num_cols`` -- and returns a tuple of freshly allocated outputs (or None when the graph has none).
``GraphExtension`` is that object for this library: same function name, argument order, keyword
names, checks and return convention; behind it a ctypes call into the C ABI of
libflexspmv_b200.so (include/flexspmv.h) on torch's current CUDA stream.  PyTorch provides device
memory and the stream, nothing else.

Differences from the reference binding, all on the host side of the same contract:
  * outputs are ``torch.empty`` (the kernels write every element; the reference needs torch::zeros
    because it accumulates with atomicAdd), scratch comes from torch's caching allocator instead of a
    per-call cudaMalloc/cudaFree (cuda_template/merged_binding_template.cu:42-49);
  * the merge-path partition is planned once per (row_end_offsets tensor, version, stream) and cached;
  * int64 ``row_end_offsets`` are accepted as they are (the reference casts to int32);
  * an unsupported dtype raises (the reference prints to stderr and falls off the end of a non-void
    function, cuda_template/merged_binding_template.cu:65-68);
  * a kernel that gives up (a bounded device-side wait ran out, or the workspace was not planned for the
    problem) stores its status in a page-locked host int registered with the workspace: the next call on
    that workspace, or ``ext.check()``, raises FlexSpmvError.  The launch path itself never synchronises;
    FLEXSPMV_CHECK_STATUS=1 makes every call synchronise and check.  After such an error the outputs of the
    failed launch are undefined.

There is no CPU path: a missing library or a CPU tensor is an error.
"""
from __future__ import annotations

import ctypes
import os
import time
from collections import OrderedDict
from typing import Dict, List, Optional, Sequence, Tuple

import torch

from .graphs import GraphIR, dim_of, operator_signature

_PKG = os.path.dirname(os.path.abspath(__file__))
DEFAULT_LIB = os.path.join(_PKG, "lib", "libflexspmv_b200.so")

_SFX = {torch.float32: "f32", torch.float64: "f64", torch.int64: "i64"}


class Desc(ctypes.Structure):
    _fields_ = [("num_rows", ctypes.c_int64), ("num_edges", ctypes.c_int64), ("num_vertices", ctypes.c_int64),
                ("offset_bits", ctypes.c_int32), ("tile_items", ctypes.c_int32), ("max_ctas", ctypes.c_int32),
                ("reserved", ctypes.c_int32)]


class GraphInfo(ctypes.Structure):
    _fields_ = [(n, ctypes.c_int32) for n in
                ("num_values", "num_indices", "num_outputs", "has_reducer", "value_bytes", "default_tile_items",
                 "block_threads", "items_per_thread", "stages", "smem_bytes", "acc_dim", "reserved")]


class FlexSpmvError(RuntimeError):
    """``status``: the library's status behind the error, 0 where there is none."""

    def __init__(self, message: str = "", status: int = 0):
        super().__init__(message)
        self.status = status


_libs: Dict[str, ctypes.CDLL] = {}


def load_library(path: Optional[str] = None) -> ctypes.CDLL:
    """dlopen the C-ABI library; raises when it is missing (no fallback of any kind)."""
    path = os.path.abspath(path or os.environ.get("FLEXSPMV_LIB", DEFAULT_LIB))
    if path not in _libs:
        if not os.path.exists(path):
            raise FlexSpmvError(f"{path} not found: build it with `python -m flexspmv_b200.build` "
                                "(there is no CPU or eager fallback)")
        lib = ctypes.CDLL(path)
        lib.flexspmv_error_string.restype = ctypes.c_char_p
        lib.flexspmv_error_string.argtypes = [ctypes.c_int]
        lib.flexspmv_plan_launches.restype = ctypes.c_int64
        _libs[path] = lib
    return _libs[path]


def check(lib, status: int, what: str):
    if status != 0:
        raise FlexSpmvError(f"{what} failed: {lib.flexspmv_error_string(status).decode()} (status {status})", status)


_CHECK_EVERY_CALL = os.environ.get("FLEXSPMV_CHECK_STATUS", "0") == "1"


class _Plan:
    """One planned workspace: the scratch tensor, its size, the tensors whose addresses it depends on, and
    the page-locked ints, to the first of which the kernels copy their error status."""
    __slots__ = ("ws", "nbytes", "keep", "flag", "_flag_view", "desc", "ws_ptr")

    def __init__(self, ws, nbytes, keep, desc):
        self.ws, self.nbytes, self.keep = ws, nbytes, keep
        self.desc, self.ws_ptr = desc, ws.data_ptr()
        self.flag = torch.zeros(2, dtype=torch.int32).pin_memory()          # the status, and the longest row once the plan is complete
        self._flag_view = self.flag.numpy()

    def status(self) -> int:
        return int(self._flag_view[0])


def _raise_if_failed(lib, plan: "_Plan", what: str):
    st = plan.status()
    if st != 0:
        raise FlexSpmvError(f"{what}: an earlier launch on this workspace failed on the device: "
                            f"{lib.flexspmv_error_string(st).decode()} (status {st}); its outputs are undefined", st)


def _stream_ptr() -> ctypes.c_void_p:
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


# The call path asks for the current device and stream on every launch; these are the plain integers behind
# torch.cuda.current_device() and torch.cuda.current_stream(index).cuda_stream, without the Stream object that the
# latter builds each time (CUDA is initialised by then: the arguments are CUDA tensors).  They are torch's own internals,
# which a torch without CUDA or a later one may not have: then the public functions serve.
_current_device = getattr(torch._C, "_cuda_getDevice", None) or torch.cuda.current_device
_raw_stream = getattr(torch._C, "_cuda_getCurrentRawStream", None) or (lambda index: torch.cuda.current_stream(index).cuda_stream)

# flexspmv_<graph>_launch(desc, values, indices, row_offsets, outputs, workspace, workspace_bytes, stream): with the
# argument types declared ctypes converts plain integers itself, without a wrapper object per pointer
_LAUNCH = ctypes.CFUNCTYPE(ctypes.c_int, *([ctypes.c_void_p] * 6), ctypes.c_size_t, ctypes.c_void_p)


def _pointers(tensors):
    """C array of the tensors' addresses (at least one slot)."""
    return (ctypes.c_void_p * (len(tensors) or 1))(*[t.data_ptr() for t in tensors])


class _Symbols:
    def __init__(self, lib, sym: str):
        def fn(name):
            try:
                f = getattr(lib, f"flexspmv_{sym}_{name}")
            except AttributeError as e:
                raise FlexSpmvError(f"library has no graph '{sym}' (symbol flexspmv_{sym}_{name})") from e
            f.restype = ctypes.c_int
            return f
        self.info, self.workspace_bytes, self.plan = fn("info"), fn("workspace_bytes"), fn("plan_indexed")
        self.plan_windows, self.uses_longest_row = fn("plan_windows"), fn("uses_longest_row")
        fn("launch")
        self.launch, self.device_status = _LAUNCH((f"flexspmv_{sym}_launch", lib)), fn("device_status")
        gi = GraphInfo()
        check(lib, self.info(ctypes.byref(gi)), f"{sym}_info")
        self.graph_info = gi
        self.also, self.name = fn, lambda what: f"flexspmv_{sym}_{what}"


class GraphExtension:
    """Drop-in for the module object ``torch.utils.cpp_extension.load`` returns in the reference flow
    (test_full/easier_full.py:359-373): exposes ``merged_spmv_launch``."""

    PLAN_CACHE_ENTRIES = 8

    def __init__(self, ir: GraphIR, lib_path: Optional[str] = None, symbol_prefix: Optional[str] = None,
                 tile_items: int = 0, max_ctas: int = 0, gather_windows: Optional[bool] = None,
                 random_gather: Optional[bool] = None, longest_row: Optional[int] = None):
        """``longest_row``: the edges of the longest row where the caller knows that all tiles hold whole rows (include/flexspmv.h,
        FLEXSPMV_LONGEST_ROW), 0 = unknown.  None = asked of the plan where launches of the size go by it (one device-to-host read,
        at plan time only; not while the stream is captured).

        ``random_gather``: run the kernel for matrices whose columns have no locality (include/flexspmv.h,
        FLEXSPMV_FLAG_RANDOM_GATHER), for graphs built with it.  None = decide per matrix the first time it is
        planned, from a sample of its index array (one device-to-host read, at plan time only): the flag is set
        when 32 consecutive edges gather from more than 16 different cache lines on average.  The environment
        variable FLEXSPMV_RANDOM_GATHER=0/1 overrides None.

        ``gather_windows``: plan column segments per tile so that the kernel gathers from shared memory
        (include/flexspmv.h, FLEXSPMV_FLAG_GATHER_WINDOWS), for graphs that support it; None = off unless the
        environment variable FLEXSPMV_GATHER_WINDOWS is 1.  Costs 2 bytes of workspace per edge and a longer
        first call per matrix; results are bit-identical for equal tile size and CTA count.  Measured on B200:
        faster on small stencil matrices that are latency-bound (2-D Poisson 512^2: 14.4 us against 16.5 us per
        launch), slower on large ones
        (3-D Poisson: 62 % against 71 % of the HBM peak -- the kernel is bound by shared-memory / L1 data-pipe
        wavefronts there, and a gather from shared memory costs more of them than an L1-cached global gather)."""
        self.ir = ir
        if gather_windows is None:
            gather_windows = os.environ.get("FLEXSPMV_GATHER_WINDOWS", "0") == "1"
        self.gather_windows = bool(gather_windows)
        if random_gather is None and os.environ.get("FLEXSPMV_RANDOM_GATHER") in ("0", "1"):
            random_gather = os.environ["FLEXSPMV_RANDOM_GATHER"] == "1"
        self.random_gather = random_gather
        self.longest_row = longest_row
        self._locality: Dict[tuple, bool] = {}
        edge_sel = [s_ for s_ in ir.selector_register if s_.get("selector") == 1 and not s_.get("row_identity")]
        self._gather_dim = dim_of(edge_sel[0]["shape"]) if edge_sel else 1
        self.lib = load_library(lib_path)
        self._lib_path = lib_path
        self.prefix = symbol_prefix or ir.name
        self.tile_items, self.max_ctas = int(tile_items), int(max_ctas)
        self.non_gather, self.gathers, self.index_names = operator_signature(ir)
        self.value_names = self.non_gather + self.gathers
        self.arg_names = self.value_names + [n + "_idx" for n in self.index_names] + \
            ["row_end_offsets", "num_rows", "num_cols"]
        self._tensor_names = self.arg_names[:-2]
        self._out_kinds = [("row" if str(o["target"]) == "reducer" else "one" if "sum" in str(o["target"]) else "edge",
                            dim_of(o["shape"])) for o in ir.outputs]
        self._has_reducer = ir.has_reducer
        self._syms: Dict[str, _Symbols] = {}
        self._by_dtype: Dict[torch.dtype, _Symbols] = {}
        self._plans: "OrderedDict[tuple, tuple]" = OrderedDict()
        self.launches = 0    # kernels this object enqueued (plan kernels included)

    # -- helpers ----------------------------------------------------------------------------------
    def symbols(self, dtype: torch.dtype) -> _Symbols:
        if dtype not in _SFX:
            raise FlexSpmvError(f"Unsupported dtype for ValueT: {dtype}. Use float32, float64 or int64.")
        sfx = _SFX[dtype]
        if sfx not in self._syms:
            self._syms[sfx] = _Symbols(self.lib, f"{self.prefix}_{sfx}")
        return self._syms[sfx]

    def _bind(self, args, kwargs) -> list:
        if len(args) > len(self.arg_names):
            raise TypeError(f"merged_spmv_launch() takes {len(self.arg_names)} arguments ({len(args)} given)")
        vals = list(args)
        for n in self.arg_names[len(args):]:
            if n not in kwargs:
                raise TypeError(f"merged_spmv_launch() missing argument '{n}'")
            vals.append(kwargs[n])
        extra = set(kwargs) - set(self.arg_names[len(args):])
        if extra:
            raise TypeError(f"merged_spmv_launch() got unexpected keyword arguments {sorted(extra)}")
        return vals

    def _looks_random(self, idx: torch.Tensor, record_bytes: int) -> bool:
        """Whether 32 consecutive edges of a sample from the middle of the index array gather from more than 16
        different 128-byte cache lines on average.  Small matrices never qualify: they are latency-bound and the
        staged kernel serves them."""
        n = idx.numel()
        if n < (1 << 20):
            return False
        key = (idx.data_ptr(), idx._version, n)
        hit = self._locality.get(key)
        if hit is None:
            m = min(n, 1 << 18) // 32 * 32
            start = (n - m) // 2 // 32 * 32
            lines = (idx[start:start + m].view(-1, 32).long() * record_bytes) >> 7
            lines = lines.sort(dim=1).values
            distinct = 1 + (lines[:, 1:] != lines[:, :-1]).sum(dim=1)
            hit = bool(float(distinct.float().mean().item()) > 16.0)
            if len(self._locality) > 64:
                self._locality.clear()
            self._locality[key] = hit
        return hit

    def _by_type(self, dtype: torch.dtype) -> _Symbols:
        return self._by_dtype.get(dtype) or self._by_dtype.setdefault(dtype, self.symbols(dtype))

    def _flags(self, syms: _Symbols, values=(), indices=()) -> int:
        flags = 1 if (self.gather_windows and (syms.graph_info.reserved & 1)) else 0
        if (syms.graph_info.reserved & 2) and self.random_gather is not False and len(indices):
            if self.random_gather or self._looks_random(indices[0], self._gather_dim * values[0].element_size()):
                flags = 2
        return flags

    def _plan_for(self, syms: _Symbols, values, indices, ro: Optional[torch.Tensor], num_rows: int, num_edges: int,
                  num_cols: int, device) -> Tuple["_Plan", Desc]:
        """The planned workspace of a problem on the current stream (``device`` is current) and its descriptor."""
        flags = self._flags(syms, values, indices)
        if flags & 1:      # the windows are bounded by the gathered array's length: take it from the tensor itself
            num_cols = int(values[len(self.non_gather)].shape[0])
        if self._has_reducer:
            bits = 64 if ro.dtype == torch.int64 else 32
            of = (ro.data_ptr(), ro._version)
        else:
            num_rows, bits, of, ro = 0, 32, None, None
        # a workspace holds per-launch state (ticket, carries): launches that may overlap on the GPU must not
        # share one, so the plan is cached per stream as well as per matrix
        key = (id(syms), num_rows, num_edges, bits, self.tile_items, self.max_ctas, flags, of, device.index,
               _raw_stream(device.index), tuple((t.data_ptr(), t._version) for t in indices) if (flags & 1) else None)
        plan = self._plans.get(key)
        if plan is not None:
            self._plans.move_to_end(key)
            if plan.desc.num_vertices == num_cols:
                return plan, plan.desc
            return plan, Desc(num_rows, num_edges, num_cols, bits, self.tile_items, self.max_ctas, plan.desc.reserved)
        described = lambda longest: Desc(num_rows, num_edges, num_cols, bits, self.tile_items, self.max_ctas, flags | longest << 8)
        plan = self._make_plan(syms, described, ro, device, indices)
        self._plans[key] = plan
        while len(self._plans) > self.PLAN_CACHE_ENTRIES:
            self._plans.popitem(last=False)
        return plan, plan.desc

    def _make_plan(self, syms: _Symbols, described, ro: Optional[torch.Tensor], device, indices: Sequence[torch.Tensor] = ()) -> "_Plan":
        """A plan for ``described(longest)``, the descriptor that names the longest row.  Where its tiles go by that (bit 0 of
        ``uses_longest_row``), they are those of whole rows until the plan says that it has none."""
        if self.longest_row is not None:
            return self._plan_once(syms, described(self.longest_row if 0 < self.longest_row <= 32 else 0), ro, device, indices)
        unknown = described(0)
        by_row = syms.uses_longest_row(ctypes.byref(unknown))
        if not by_row or torch.cuda.is_current_stream_capturing():
            return self._plan_once(syms, unknown, ro, device, indices)
        plan = self._plan_once(syms, described(32), ro, device, indices)
        longest = self._longest_row(plan)
        if longest == 0 and by_row & 1:
            return self._plan_once(syms, unknown, ro, device, indices)
        plan.desc = described(longest)
        return plan

    def _longest_row(self, plan: "_Plan") -> int:
        """Part of the first call on a matrix: the plan's last kernel leaves the word in page-locked memory, and the host looks at it until it
        has changed (15 us of a first call; with a copy and a wait for the stream 25, with a device tensor and its ``item`` 40); behind much other work on the
        stream it waits for that instead."""
        view, until = plan._flag_view, time.perf_counter() + 100e-6
        while view[1] < 0 and time.perf_counter() < until:
            pass
        if view[1] < 0:
            torch.cuda.current_stream(plan.ws.device).synchronize()
        return max(int(view[1]), 0)

    def _plan_once(self, syms: _Symbols, desc: Desc, ro: Optional[torch.Tensor], device, indices: Sequence[torch.Tensor]) -> "_Plan":
        nbytes = ctypes.c_size_t()
        check(self.lib, syms.workspace_bytes(ctypes.byref(desc), ctypes.byref(nbytes)), "workspace_bytes")
        ws = torch.empty(nbytes.value, dtype=torch.uint8, device=device)
        ip = _pointers(indices)
        before = self.lib.flexspmv_plan_launches()
        check(self.lib, syms.plan(ctypes.byref(desc), ip, ctypes.c_void_p(ro.data_ptr() if ro is not None else 0),
                                  ctypes.c_void_p(ws.data_ptr()), ctypes.c_size_t(nbytes.value), _stream_ptr()),
              "plan")
        if desc.reserved & 1:      # gather windows: the second planning step reads the index array
            check(self.lib, syms.plan_windows(ctypes.byref(desc), ip, ctypes.c_void_p(ws.data_ptr()),
                                              ctypes.c_size_t(nbytes.value), _stream_ptr()), "plan_windows")
        # keep the row-offset tensor alive so its address cannot be recycled under a cached plan
        plan = _Plan(ws, nbytes.value, (ro, tuple(indices) if (desc.reserved & 1) else None), desc)
        plan._flag_view[1] = -1
        check(self.lib, self.lib.flexspmv_workspace_mirrors(ctypes.c_void_p(ws.data_ptr()), ctypes.c_void_p(plan.flag.data_ptr()),
                                                            ctypes.c_void_p(plan.flag.data_ptr() + 4), _stream_ptr()), "workspace_mirrors")
        self.launches += self.lib.flexspmv_plan_launches() - before
        return plan

    # -- the operator --------------------------------------------------------------------------------
    def merged_spmv_launch(self, *args, **kwargs):
        a = args if (not kwargs and len(args) == len(self.arg_names)) else self._bind(args, kwargs)
        nv = len(self.value_names)
        ni = nv + len(self.index_names)
        values, indices = a[:nv], a[nv:ni]
        row_end_offsets, num_rows, num_cols = a[ni], int(a[ni + 1]), int(a[ni + 2])
        for n, t in zip(self._tensor_names, a):
            if not isinstance(t, torch.Tensor):
                raise TypeError(f"{n} must be a torch.Tensor")
            if not t.is_cuda:
                raise FlexSpmvError(f"{n} must be a CUDA tensor")
            if not t.is_contiguous():
                raise FlexSpmvError(f"{n} must be contiguous")
        dispatch = values[0]
        dt = dispatch.dtype
        syms = self._by_type(dt)
        for n, t in zip(self.value_names, values):
            if t.dtype != dt:
                raise FlexSpmvError(f"{n} dtype mismatch")
        for n, t in zip(self.index_names, indices):
            if t.dtype != torch.int32:
                raise FlexSpmvError(f"{n}_idx dtype mismatch")
        ne = int(indices[0].numel()) if indices else num_cols
        if ne <= 0:
            raise FlexSpmvError("selector index must be non-empty")
        if self._has_reducer:
            if row_end_offsets.dtype not in (torch.int32, torch.int64):
                raise FlexSpmvError("row_end_offsets dtype mismatch")
            if row_end_offsets.numel() != num_rows + 1:
                raise FlexSpmvError("row_end_offsets must have length num_rows + 1")
        device = dispatch.device
        outputs: List[torch.Tensor] = []
        for kind, d in self._out_kinds:
            if kind == "one":
                shape = (d,)
            else:
                n = num_rows if kind == "row" else ne
                shape = (n,) if d == 1 else (n, d)
            outputs.append(torch.empty(shape, dtype=dt, device=device))
        self._launch(syms, values, indices, row_end_offsets, outputs, num_rows, ne, num_cols, device, "merged_spmv_launch")
        if not outputs:
            return None
        return tuple(outputs)

    def _launch(self, syms: _Symbols, values, indices, ro, outputs, num_rows: int, num_edges: int, num_cols: int, device,
                what: str) -> None:
        if _current_device() != device.index:
            with torch.cuda.device(device):
                return self._launch(syms, values, indices, ro, outputs, num_rows, num_edges, num_cols, device, what)
        plan, desc = self._plan_for(syms, values, indices, ro, num_rows, num_edges, num_cols, device)
        _raise_if_failed(self.lib, plan, what)
        st = syms.launch(ctypes.byref(desc), _pointers(values), _pointers(indices), ro.data_ptr() if self._has_reducer else 0,
                         _pointers(outputs), plan.ws_ptr, plan.nbytes, _raw_stream(device.index))
        if st != 0:
            check(self.lib, st, what)
        self.launches += 1
        if _CHECK_EVERY_CALL:
            self.check()

    __call__ = merged_spmv_launch

    def launch_into(self, values: Sequence[torch.Tensor], indices: Sequence[torch.Tensor],
                    row_end_offsets: Optional[torch.Tensor], outputs: Sequence[torch.Tensor],
                    num_rows: int, num_edges: int, num_cols: int = 0) -> None:
        """Same fused pass as ``merged_spmv_launch`` but into caller-provided output tensors (any
        tensor or slice whose storage is large enough; e.g. the owned part of the next iteration's
        vector).  No allocation, no checks beyond the C ABI's own; one kernel launch."""
        self._launch(self._by_type(values[0].dtype), values, indices, row_end_offsets, outputs, num_rows, num_edges, num_cols,
                     values[0].device, "launch_into")

    def prepare(self, values: Sequence[torch.Tensor], indices: Sequence[torch.Tensor],
                row_end_offsets: Optional[torch.Tensor], outputs: Sequence[torch.Tensor],
                num_rows: int, num_edges: int, num_cols: int = 0) -> "PreparedLaunch":
        """Binds one fixed set of tensors once (plan, workspace, C argument arrays) so that every later
        ``launch()`` is a single foreign call on the current stream: the form for time-stepping loops, where
        the reference wrapper re-marshals every argument on every call
        (python_wrapper/dynamic_replace_submodule.py:147-199).  The row offsets must not change while the
        object is in use; the value / index / output tensors may be rewritten in place."""
        syms = self._by_type(values[0].dtype)
        device = values[0].device
        with torch.cuda.device(device):
            plan, desc = self._plan_for(syms, values, indices, row_end_offsets, num_rows, num_edges, num_cols, device)
        return PreparedLaunch(self, syms, desc, list(values), list(indices), row_end_offsets if self._has_reducer else None,
                              list(outputs), plan)

    def prepare_step(self, values: Sequence[torch.Tensor], indices: Sequence[torch.Tensor], row_end_offsets: torch.Tensor,
                     outputs: Sequence[torch.Tensor], num_rows: int, num_edges: int, num_cols: int = 0) -> "Optional[PreparedLaunch]":
        """``prepare`` for a graph whose unit has a launch over all stages of a step (include/flexspmv.h,
        swe_delta_rk_T_step); None where the problem does not fit that launch.  ``rows_a_cta`` of the result: the consecutive rows
        that each of its CTAs takes."""
        syms = self._by_type(values[0].dtype)
        launch = self.prepare(values, indices, row_end_offsets, outputs, num_rows, num_edges, num_cols)
        with torch.cuda.device(values[0].device):
            launch.rows_a_cta = int(syms.also("step_fits")(ctypes.byref(launch._desc)))
        if not launch.rows_a_cta:
            return None
        launch._fn = _LAUNCH((syms.name("step"), self.lib))
        return launch

    def longest_row_of(self, launch: "PreparedLaunch") -> int:
        """The edges of the longest row of a prepared problem whose plan holds whole rows (include/flexspmv.h,
        flexspmv_workspace_longest_row), else 0.  Waits for the plan."""
        with torch.cuda.device(launch._device):
            return self._longest_row(launch._plan)

    def device_status(self, dtype: torch.dtype, row_end_offsets: Optional[torch.Tensor] = None) -> int:
        """Reads back the status word of the most recently used workspace (synchronises)."""
        if not self._plans:
            return 0
        ws = next(reversed(self._plans.values())).ws
        out = torch.zeros(1, dtype=torch.int32, device=ws.device)
        syms = self.symbols(dtype)
        with torch.cuda.device(ws.device):
            check(self.lib, syms.device_status(ctypes.c_void_p(ws.data_ptr()), ctypes.c_void_p(out.data_ptr()), _stream_ptr()),
                  "device_status")
        return int(out.item())

    def planned_whole_rows(self) -> bool:
        """Whether the plan made last found a matrix of short rows, every tile of which holds whole rows only
        (include/flexspmv.h, flexspmv_workspace_whole_rows).  Synchronises."""
        if not self._plans:
            return False
        ws = next(reversed(self._plans.values())).ws
        out = torch.zeros(1, dtype=torch.int32, device=ws.device)
        with torch.cuda.device(ws.device):
            self.lib.flexspmv_workspace_whole_rows.restype = ctypes.c_int
            check(self.lib, self.lib.flexspmv_workspace_whole_rows(ctypes.c_void_p(ws.data_ptr()), ctypes.c_void_p(out.data_ptr()),
                                                                   _stream_ptr()), "workspace_whole_rows")
        return int(out.item()) == 1

    def check(self) -> None:
        """Waits for the work enqueued so far on every device this object planned for, then raises
        FlexSpmvError if a kernel gave up on any of its cached workspaces (a bounded wait ran out, or a
        launch met a workspace that was not planned for its problem).  Call it after a timed region or a
        time-stepping loop; the launch path itself only looks at the host-side copy of the status."""
        plans = list(self._plans.values())
        for dev in {p.ws.device for p in plans}:
            torch.cuda.synchronize(dev)
        for p in plans:
            _raise_if_failed(self.lib, p, "check")


class PreparedLaunch:
    """One graph bound to one set of device tensors (see ``GraphExtension.prepare``)."""

    def __init__(self, ext: GraphExtension, syms: _Symbols, desc: Desc, values, indices, ro, outputs, plan: _Plan):
        self.ext, self._syms, self._desc = ext, syms, desc
        ws, ws_bytes = plan.ws, plan.nbytes
        self._plan = plan
        self._keep = (values, indices, ro, outputs, ws)       # the raw pointers below borrow these tensors
        self._device = ws.device.index
        self._planned = torch.cuda.Event()                    # the plan kernels were enqueued on this stream
        self._planned.record(torch.cuda.current_stream(ws.device))
        self._ordered = {torch.cuda.current_stream(ws.device).cuda_stream}
        self._args = (ctypes.byref(desc), _pointers(values), _pointers(indices), ro.data_ptr() if ro is not None else 0,
                      _pointers(outputs), ws.data_ptr(), ws_bytes)
        self._fn = syms.launch

    def launch(self) -> None:
        """Enqueues the fused pass on the current stream of the tensors' device.  The workspace carries
        per-launch state, so launches of one prepared object must be stream-ordered with one another:
        launching from a second stream needs a second prepared object."""
        if _current_device() != self._device:
            with torch.cuda.device(self._device):
                return self.launch()
        if self._plan._flag_view[0]:
            self.raise_if_failed()
        stream = _raw_stream(self._device)
        if stream not in self._ordered:                       # first use on another stream: after the plan
            if torch.cuda.is_current_stream_capturing():
                # an event recorded outside a capture cannot be waited on inside it
                raise FlexSpmvError("first launch of a prepared object on a stream that is being captured: launch it "
                                    "once on that stream before the capture begins")
            torch.cuda.current_stream().wait_event(self._planned)
            self._ordered.add(stream)
        st = self._fn(*self._args, stream)
        if st != 0:
            check(self.ext.lib, st, "launch")
        self.ext.launches += 1
        if _CHECK_EVERY_CALL:
            self.ext.check()

    __call__ = launch

    def failed(self) -> bool:
        """Whether a kernel has given up on this object's workspace, as far as the host has been told (one read of host
        memory, no synchronisation)."""
        return self._plan._flag_view[0] != 0

    def raise_if_failed(self, what: str = "launch") -> None:
        """Raises FlexSpmvError where ``failed()``."""
        _raise_if_failed(self.ext.lib, self._plan, what)


def load_builtin(name: str, **kw) -> GraphExtension:
    """Extension object for one of the graphs compiled into libflexspmv_b200.so."""
    from .graphs import ALL_GRAPHS
    return GraphExtension(ALL_GRAPHS[name](), **kw)
