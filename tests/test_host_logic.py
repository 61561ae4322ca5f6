"""Host-side logic that needs no GPU: IR -> operator signature, the CUDA emitter, tile configuration,
problem generators and the algorithmic-bytes figures of the benchmark configurations."""
import os

import numpy as np
import pytest

from flexspmv_b200 import graphs, problems
from flexspmv_b200.build import NVCC, NVCC_FLAGS
from flexspmv_b200.codegen import emit_cuda


def test_operator_signature_follows_reference_binding_order():
    # non-gather values, gather values, one index tensor per selector target (codegen/merged_gen_binding.py:65-78)
    assert graphs.operator_signature(graphs.spmv_graph()) == (["vals"], ["x"], ["selector"])
    assert graphs.operator_signature(graphs.spring_mass_graph()) == (["L", "k"], ["p"], ["sel_src", "sel_dst"])
    assert graphs.operator_signature(graphs.rusanov_graph()) == (["face"], ["U"], ["sel_self", "sel_nbr"])
    assert graphs.operator_signature(graphs.mixed_dims_graph()) == (["ea", "eb"], ["vx"], ["s0", "s1"])


def test_binding_argument_names_without_gpu():
    from flexspmv_b200.binding import GraphExtension
    ext = GraphExtension(graphs.spring_mass_graph())
    assert ext.arg_names == ["L", "k", "p", "sel_src_idx", "sel_dst_idx", "row_end_offsets", "num_rows", "num_cols"]
    with pytest.raises(TypeError):
        ext.merged_spmv_launch(1, 2, 3)                  # missing arguments
    import torch
    t = torch.zeros(4)
    with pytest.raises(RuntimeError):                    # CPU tensors are refused: there is no CPU path
        ext.merged_spmv_launch(t, t, t.reshape(2, 2), t.int(), t.int(), t.int(), 3, 3)


def test_emitter_is_deterministic_and_resolves_overloads():
    ir = graphs.ops_zoo_graph()
    a = emit_cuda.emit_graph(ir, "float32")
    assert a == emit_cuda.emit_graph(graphs.ops_zoo_graph(), "float32")
    assert "fx::zip(w, sel, fx::DivGuard{})" in a              # equal widths: guarded member operator/
    assert "fx::zip_sv(V(1.5), sel, fx::DivGuard{})" in a      # scalar / tensor: guarded
    assert "fx::zip_vs(a4, nn, fx::Div{})" in a                # tensor / scalar: plain IEEE divide
    assert "FLEXSPMV_DEFINE_GRAPH(ops_zoo_f32, gen_ops_zoo_f32::Graph, gen_ops_zoo_f32::Cfg, gen_ops_zoo_f32::CfgWin, gen_ops_zoo_f32::CfgLean)" in a
    r = emit_cuda.emit_graph(graphs.rusanov_graph(), "float64")
    assert "fx::PowHalf{}" in r and "kGatherNeedsRow = true" in r and "kNumReducers = 3, kAccDim = 3" in r
    s = emit_cuda.emit_graph(graphs.spring_mass_graph(), "float32")
    assert "kNumStreams = 1" in s        # only the sel_dst index array is staged: sel_src is the row id, L and k are read directly
    assert "r.L = fx::ldg_vec<V, 1>(p.L + e * 1);" in s
    assert "kNumStreams = 2" in emit_cuda.emit_graph(graphs.spmv_graph(), "float64")    # two-phase graphs stage values too
    body = s.split("struct GRow")[1]
    assert "sel_src_idx" not in body and "idx_sel_src" not in body      # the row-identity index array is never read
    assert "g.sel_src = fx::ldg_vec<V, 2>(p.p + row * 2);" in body      # it is the row the merge path already knows
    assert "int idx_sel_dst;" in body
    m = emit_cuda.emit_graph(graphs.mixed_dims_graph(), "int64")
    assert "fx::st_vec(p.out_t1 + (long long)e * 2, t1)" in m  # per-edge map output


def test_emitter_rejects_what_the_reference_cannot_express():
    ir = graphs.spmv_graph()
    ir.map_operations.insert(0, graphs.mop("bad", "gt", (1,), 0.5, "vals"))
    with pytest.raises(ValueError):
        emit_cuda.emit_graph(ir, "float32")
    ir2 = graphs.spmv_graph()
    ir2.map_operations.insert(0, graphs.mop("u", "cosh", (1,), "vals"))
    with pytest.raises(ValueError):
        emit_cuda.emit_graph(ir2, "float32")


def test_tile_configs_fit_shared_memory():
    for g, make in graphs.ALL_GRAPHS.items():
        ir = make()
        if not ir.has_reducer:
            continue
        for dt in graphs.GRAPH_DTYPES[g]:
            block, ipt, stages, ctas = emit_cuda.choose_config(ir, dt)
            assert block % 32 == 0 and ipt % 2 == 1 and block * ipt <= 65535
            assert emit_cuda.smem_bytes(ir, dt, block, ipt, stages) * ctas <= 227 * 1024 + 1024 * ctas

@pytest.mark.parametrize("dtype", ["float64", "int64"])
def test_wide_records_keep_the_tile_a_caller_may_ask_for(dtype):
    """Graphs of wide records: small CTAs that still take tiles of 256 items, as 256 threads of one edge did, and a byte of
    workspace more is not asked for."""
    import ctypes
    from flexspmv_b200.binding import Desc, load_library
    ir = graphs.mixed_dims_graph()
    block, ipt, stages, ctas = emit_cuda.wide_config(ir, dtype, emit_cuda.choose_config(ir, dtype))
    assert block * ipt == 256 and block == 64 and emit_cuda.smem_bytes(ir, dtype, block, ipt, stages) * ctas <= 227 * 1024 - 1024 * ctas
    assert emit_cuda.wide_config(ir, "float32", emit_cuda.choose_config(ir, "float32")) == emit_cuda.choose_config(ir, "float32")
    bytes_of = getattr(load_library(), f"flexspmv_mixed_dims_{emit_cuda.CTYPE[dtype][1]}_workspace_bytes")
    n, default = ctypes.c_size_t(), ctypes.c_size_t()
    for tile, code in ((193, 0), (256, 0), (257, -4)):
        assert bytes_of(ctypes.byref(Desc(1000, 9000, 1000, 32, tile, 0, 0)), ctypes.byref(n)) == code, tile
    assert bytes_of(ctypes.byref(Desc(1000, 9000, 1000, 32, 256, 0, 0)), ctypes.byref(n)) == 0
    assert bytes_of(ctypes.byref(Desc(1000, 9000, 1000, 32, 0, 0, 0)), ctypes.byref(default)) == 0 and n.value == default.value


def test_algorithmic_bytes_of_the_benchmark_configs():
    p0 = problems.poisson2d(512)
    assert (p0.num_rows, p0.nnz) == (262144, 1308672)
    assert problems.algorithmic_bytes(graphs.spmv_graph(), p0.num_rows, p0.nnz, p0.num_cols, 8, 4) == 20946948
    p1 = problems.spring_mass(64)
    assert p1.nnz == 8 * 64 * 64 - 6 * 64 * 2 + 4 - 0 or p1.nnz == int(p1.row_offsets[-1])
    n = 1024
    e1 = 8 * n * n - 12 * n + 4
    assert e1 == 8376324
    assert problems.algorithmic_bytes(graphs.spring_mass_graph(), n * n, e1, n * n, 4, 4) == 121487412
    assert problems.algorithmic_bytes(graphs.rusanov_graph(), 2 * n * n, 6 * n * n, 2 * n * n, 8, 4) == 285212676
    n3 = 512 ** 3
    nnz4 = 7 * n3 - 6 * 512 * 512
    assert nnz4 == 937951232
    assert problems.algorithmic_bytes(graphs.spmv_graph(), n3, nnz4, n3, 8, 8) == 14476640264


def test_generators_are_valid_csr():
    for prob in (problems.poisson2d(16), problems.poisson3d(6), problems.spring_mass(12), problems.shallow_water(8),
                 problems.powerlaw(2000, cap=300)):
        ro = prob.row_offsets
        assert ro[0] == 0 and (np.diff(ro) >= 0).all() and ro[-1] == prob.nnz and ro.shape[0] == prob.num_rows + 1
        for idx in prob.indices.values():
            assert idx.dtype == np.int32 and idx.min() >= 0 and idx.max() < prob.num_cols
    sm = problems.spring_mass(12)
    assert np.array_equal(sm.indices["sel_src"], np.repeat(np.arange(144), np.diff(sm.row_offsets)))
    sw = problems.shallow_water(8)
    nbr = sw.indices["sel_nbr"].reshape(-1, 3)
    own = np.arange(128)[:, None]
    back = nbr[nbr]                                   # neighbour relation is symmetric (or a boundary self-edge)
    assert ((back == own[:, None, :].repeat(3, axis=1).reshape(128, 3, 1)).any(axis=2) | (nbr == own)).all()
    face = sw.values["face"].reshape(-1, 3, 3)
    assert np.allclose((face[:, :, :2] * face[:, :, 2:3]).sum(axis=1), 0.0, atol=1e-15)   # closed cells: sum n*len = 0
    pl = problems.powerlaw(5000, cap=400)
    r = np.repeat(np.arange(5000), np.diff(pl.row_offsets))
    k = r.astype(np.int64) * (1 << 32) + pl.indices["selector"]
    assert (np.diff(k) >= 0).all()                    # columns sorted within each row


def test_warp_kernel_configuration_follows_the_value_width():
    """The emitter gives the random-column kernel 1024-thread CTAs for 4-byte values and 768-thread CTAs for 8-byte
    values (which need more than the 64 registers a 1024-thread CTA leaves a thread)."""
    from flexspmv_b200 import graphs
    from flexspmv_b200.codegen.emit_cuda import emit_graph
    ir = graphs.spmv_graph()
    assert "using CfgLean = flex::WarpCfg<1024, 5, 1>;" in emit_graph(ir, "float32", "spmv_f32")
    for dt, sym in (("float64", "spmv_f64"), ("int64", "spmv_i64")):
        assert "using CfgLean = flex::WarpCfg<768, 5, 1>;" in emit_graph(ir, dt, sym)


def test_shared_memory_holds_nothing_a_graphs_loops_do_not_use():
    """What a CTA claims is taken from the L1 cache in coarse steps: four CTAs of an SM stay below the 196 KB one, and a
    graph whose tiles are never moved to row starts (per-edge outputs) has no room for moved boundaries."""
    import ctypes
    from flexspmv_b200.binding import GraphInfo, load_library
    lib = load_library()

    def claimed(name, dtype):
        gi = GraphInfo()
        assert getattr(lib, f"flexspmv_{name}_{emit_cuda.CTYPE[dtype][1]}_info")(ctypes.byref(gi)) == 0
        return gi.smem_bytes

    for name, dtype in (("spmv", "float64"), ("spmv", "int64"), ("rusanov", "float32"), ("swe_delta", "float32"), ("swe_delta_rk", "float32"),
                        ("ops_zoo", "float32"), ("ops_zoo", "float64")):
        assert 4 * (claimed(name, dtype) + 1024) <= 196 * 1024, name      # the system takes 1 KB a CTA
    for dtype, tile in (("float32", 768), ("float64", 256), ("int64", 256)):
        ir = graphs.mixed_dims_graph()
        per_edge, streams = emit_cuda._stream_bytes_per_edge(ir, emit_cuda.VBYTES[dtype])
        acc = 8                                                           # two reducers, 2 and 6 wide
        per_tile = tile * (2 * per_edge + acc * emit_cuda.VBYTES[dtype] + 4)
        assert claimed("mixed_dims", dtype) <= per_tile + 2 * (32 * (streams + 1) + 16 + 128) + 2048


@pytest.mark.parametrize("make,dtype,batches", [(graphs.spring_mass_graph, "float64", (1, 1)), (graphs.rusanov_graph, "float32", (1, 1)),
                                                (graphs.swe_delta_graph, "float32", (1, 1)), (graphs.spring_mass_graph, "float32", (2, 1)),
                                                (graphs.swe_boundary_graph, "float32", (8, 8)), (graphs.swe_boundary_graph, "float64", (4, 1)),
                                                (graphs.spmv_graph, "float64", (1, 4)), (graphs.ops_zoo_graph, "float64", (1, 2))])
def test_edges_in_flight_per_row(make, dtype, batches):
    """(loop with carries, loop over whole rows): a row-mode graph with gathers takes one edge at a time unless it was
    tuned, and a map that divides at most two; more were spilled to local memory."""
    import re
    fields = re.search(r"using Cfg = flex::TileCfg<([^>]*)>", emit_cuda.emit_graph(make(), dtype)).group(1).split(", ")
    assert (int(fields[4]), int(fields[6])) == batches


def test_the_package_imports_without_torchs_cuda_internals():
    """A torch without CUDA has no torch._C._cuda_getDevice: the import must get as far as load_library's own message."""
    import os
    import subprocess
    import sys
    code = ("import torch\n"
            "for n in ('_cuda_getDevice', '_cuda_getCurrentRawStream'):\n"
            "    if hasattr(torch._C, n): delattr(torch._C, n)\n"
            "from flexspmv_b200 import binding\n"
            "assert binding._current_device is torch.cuda.current_device\n"
            "try: binding.load_library('/nowhere.so')\n"
            "except binding.FlexSpmvError as e: print(e)\n")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", code], cwd=root, capture_output=True, text=True)
    assert r.returncode == 0 and "not found" in r.stdout, r.stderr


def _wider(name):
    """A graph under a built-in one's name whose records are wider."""
    import copy
    ir = copy.deepcopy(graphs.ALL_GRAPHS[name]())
    if name == "rusanov":                # eight values a face, of which the map takes three
        for s_ in ir.inputs + ir.selector_register:
            if "face" in (s_["name"], s_.get("selector_name")):
                s_["shape"] = (8,)
        return ir
    width = (1,) if name == "spring_mass" else (2,)
    ir.inputs.insert(0, graphs.placeholder("c", width))
    ir.selector_register.insert(0, graphs.edge_register("c", width))
    last = next(op_ for op_ in ir.map_operations if op_["op"] == "mul")
    if name == "spring_mass":
        last["args"] = ["c" if a == "k" else a for a in last["args"]]
    return ir


@pytest.mark.parametrize("name,dtypes", [("spring_mass", ("float32", "float64")), ("swe_delta", ("float64",)), ("rusanov", ("float32", "float64"))])
def test_large_tiles_go_by_what_a_graph_moves(name, dtypes):
    """A graph takes the configuration for large launches by its records and operations: another one under the same name does not, the
    same one under another name does."""
    import copy
    for dt in dtypes:
        assert "CfgBig" in emit_cuda.emit_graph(graphs.ALL_GRAPHS[name](), dt, "it")
        other = copy.deepcopy(graphs.ALL_GRAPHS[name]())
        other.name = "traced"
        config = emit_cuda.big_config(other, dt)
        assert config == emit_cuda.big_config(graphs.ALL_GRAPHS[name](), dt) and emit_cuda.smem_bytes(other, dt, *config[:3]) <= emit_cuda.MAX_SMEM
        wider = _wider(name)
        assert emit_cuda.smem_bytes(wider, dt, *config[:3]) > emit_cuda.MAX_SMEM
        assert emit_cuda.big_config(wider, dt) is None
        longer = copy.deepcopy(other)       # more work an edge than was measured
        longer.map_operations.insert(-1, dict(longer.map_operations[0], name="more"))
        assert emit_cuda.big_config(longer, dt) is None
    assert emit_cuda.big_config(graphs.ALL_GRAPHS[name](), "int64") is None


@pytest.mark.skipif(not os.path.exists(NVCC), reason="needs nvcc")
@pytest.mark.parametrize("name,dt", [("spring_mass", "float32"), ("spring_mass", "float64"), ("swe_delta", "float64"), ("rusanov", "float64")])
def test_wider_records_under_a_built_in_name_compile(name, dt, tmp_path):
    import subprocess
    src = tmp_path / "unit.cu"
    src.write_text(emit_cuda.emit_graph(_wider(name), dt, "wider", windows=False))
    run = subprocess.run([NVCC] + NVCC_FLAGS + ["-cuda", str(src), "-o", str(tmp_path / "unit.ii")], capture_output=True, text=True)
    assert run.returncode == 0, run.stderr[-2000:]


@pytest.mark.parametrize("graph,edges,uses", [("spring_mass_f32", 8, 1), ("spring_mass_f64", 8, 1), ("rusanov_f64", 3, 1), ("swe_delta_f64", 3, 1),
                                              ("swe_delta_rk_f64", 3, 0), ("spmv_f64", 27, 1), ("spmv_f32", 27, 1), ("spmv_i64", 27, 0), ("spmv_f64", 33, 0),
                                              ("spmv_f64", 12, 0), ("rusanov_f64", 9, 0), ("edge_sum_f32", 3, 0), ("spmv_f64", 5, 2), ("spmv_i64", 5, 2), ("spmv_f64", 6, 0),
                                              ("spmv_f32", 7, 2), ("spmv_f32", 4, 0), ("spmv_f32", 8, 0), ("swe_boundary_f64", 5, 0)])
def test_which_launches_go_by_the_longest_row(graph, edges, uses):
    """On a million rows over 148 SMs: the workspace of a descriptor that names the longest row has fewer, larger tiles where the library
    says that it matters, and is the same one elsewhere.  What is no row length is nothing known."""
    import ctypes
    from flexspmv_b200.binding import Desc, load_library
    lib = load_library()

    def bytes_of(reserved, **kw):
        d, n = Desc(1 << 20, edges << 20, 1 << 20, 32, kw.get("tile_items", 0), kw.get("max_ctas", 0), reserved), ctypes.c_size_t()
        assert getattr(lib, f"flexspmv_{graph}_workspace_bytes")(ctypes.byref(d), ctypes.byref(n)) == 0
        return n.value, getattr(lib, f"flexspmv_{graph}_uses_longest_row")(ctypes.byref(d))

    (unknown, asked), (known, also) = bytes_of(0), bytes_of(edges << 8)
    assert asked == also == uses and (known < unknown) == bool(uses & 1)
    assert all(bytes_of(n << 8)[0] == unknown for n in (33, 63, 65, 96, 257, 1 << 20))
    for kw in ({"max_ctas": 7}, {"tile_items": 64}):
        assert bytes_of(edges << 8, **kw)[1] == uses & 2 and bytes_of(edges << 8, **kw) == bytes_of(0, **kw)


@pytest.mark.parametrize("given,uses,longest,planned,described", [(None, 0, 9, [0], 0), (None, 1, 9, [32], 9), (None, 1, 0, [32, 0], 0), (0, 1, 9, [0], 0),
                                                                  (7, 1, 9, [7], 7), (None, 2, 5, [32], 5), (None, 2, 0, [32], 0)])
def test_a_plan_is_asked_for_the_longest_row(given, uses, longest, planned, described, monkeypatch):
    from flexspmv_b200.binding import Desc, GraphExtension
    import torch
    made = []

    def plan_once(syms, desc, *rest):
        made.append(desc.reserved >> 8)
        return type("Plan", (), {"desc": desc})()

    ext = GraphExtension(graphs.spring_mass_graph(), longest_row=given)
    monkeypatch.setattr(ext, "_plan_once", plan_once)
    monkeypatch.setattr(ext, "_longest_row", lambda plan: longest)
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    syms = type("Syms", (), {"uses_longest_row": staticmethod(lambda desc: uses)})()
    plan = ext._make_plan(syms, lambda n: Desc(10, 20, 10, 32, 0, 0, n << 8), None, None)
    assert made == planned and plan.desc.reserved >> 8 == described
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: True)
    made.clear()
    plan = ext._make_plan(syms, lambda n: Desc(10, 20, 10, 32, 0, 0, n << 8), None, None)
    assert made == [given or 0] and plan.desc.reserved >> 8 == (given or 0)


def test_the_reference_arm_times_no_restatement():
    import json
    import subprocess
    import sys
    from oracle import ref_run
    if ref_run.available("spmv"):
        pytest.skip("the reference's operator is here")
    bench = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "bench.py")
    run = subprocess.run([sys.executable, bench, "--impl", "reference", "--grid", "16", "--steps", "1", "--warmup", "3"], capture_output=True, text=True)
    line = json.loads(run.stdout.strip().splitlines()[-1])
    assert run.returncode == 0 and line["impl"] == "reference" and line["unavailable"] and "value" not in line
