"""IR -> ``merged_binding.cu``: the torch-extension shim of one fused graph.

Counterpart of the reference's binding generator (codegen/merged_gen_binding.py:9-237), which fills
cuda_template/merged_binding_template.cu.  The emitted file defines the same Python-visible function,
``merged_spmv_launch``, with the same positional order and keyword names (codegen/merged_gen_binding.py:65-78:
non-gather value inputs, gather value inputs, one ``<target>_idx`` tensor per selector, ``row_end_offsets``,
``num_rows``, ``num_cols``), the same checks and the same return convention (a tuple of outputs: reducer
``(num_rows[, dim])``, ``sum`` aggregator ``(dim,)``, per-edge output ``(ne[, dim])``; nothing when the graph has no
allocated output, :100-134), so the reference's own build step

    ext = torch.utils.cpp_extension.load(name=..., sources=["<root>/merged_binding.cu"],
                                         extra_include_paths=[root, root + "/include"], ...)

(test_full/easier_full.py:359-373) works on it unchanged.  Like the reference flow, which writes its generated
headers into ``<root>/include``, ``generate_binding_code`` writes there the generated kernel units of the graph
(one per value type, from codegen/emit_cuda.py) and the hand-written kernel headers they include; the binding
includes them, so the extension is one self-contained translation unit.

What the shim does differently from the template it replaces:
  * outputs are ``torch::empty`` (every element is written by the kernels; the reference needs zeros for its
    atomicAdd accumulation, :100-110), scratch comes from torch's caching allocator and is planned once per
    (row offsets, version, stream) and cached, instead of cudaMalloc / cudaFree on every call
    (cuda_template/merged_binding_template.cu:42-49);
  * ``row_end_offsets`` may be int32 or int64;
  * an unsupported value dtype raises (the template prints to stderr and falls off the end of a non-void
    function, :65-68); the int64 value type is compiled when asked for, as the reference's optional
    ``torch::kLong`` case (:143-157);
  * a non-zero status of the C entry points becomes a TORCH_CHECK failure with the library's message, and
    ``device_status()`` reads back the status word of the most recent workspace (0, or the code of a kernel
    that gave up).
"""
from __future__ import annotations

import os
from typing import Iterable, Optional

from ..graphs import GraphIR, dim_of, operator_signature
from .emit_cuda import CTYPE, emit_graph

_PKG = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_ROOT = os.path.dirname(_PKG)
_TORCH_TYPE = {"float32": "torch::kFloat", "float64": "torch::kDouble", "int64": "torch::kLong"}

KERNEL_HEADERS = ("flex_common.cuh", "flex_tensor.cuh", "flex_tile_kernel.cuh", "flex_warp_kernel.cuh", "flex_warp_ahead.cuh",
                  "flex_edge_kernel.cuh", "flex_graph_api.cuh", "flex_core.cu")


def binding_source(ir: GraphIR, symbol: str, dtypes: Iterable[str]) -> str:
    """Text of merged_binding.cu for ``ir``; the graph units ``include/merged_graph_<symbol>_<type>.cuh`` and the
    kernel headers are expected on the include path."""
    dtypes = tuple(dtypes)
    non_gather, gathers, index_names = operator_signature(ir)
    values = non_gather + gathers
    idx_args = [n + "_idx" for n in index_names]
    has_red = ir.has_reducer
    dispatch = values[0]
    params = [f"torch::Tensor {n}" for n in values + idx_args] + ["torch::Tensor row_end_offsets", "int64_t num_rows",
                                                                  "int64_t num_cols"]
    call_args = ", ".join(values + idx_args + ["row_end_offsets", "num_rows", "num_cols"])
    L = []
    w = L.append
    w(f"// GENERATED by flexspmv_b200.codegen.merged_gen_binding -- graph '{ir.name}', digest {ir.digest()}")
    w("#include <torch/extension.h>")
    w("#include <ATen/cuda/CUDAContext.h>")
    w("#include <c10/cuda/CUDAGuard.h>")
    w("#include <list>")
    w("#include <mutex>")
    w("#include <tuple>")
    w("")
    w("// library-wide entry points (partition, plan helpers) and the fused kernels of this graph, one unit per value type")
    w('#include "flex_core.cu"')
    for dt in dtypes:
        w(f'#include "merged_graph_{symbol}_{CTYPE[dt][1]}.cuh"')
    w("")
    w("namespace {")
    w("")
    w("// One planned workspace per (row offsets, their version, sizes, stream): the merge-path partition of a matrix is")
    w("// computed once and reused by every later call.  A workspace holds per-launch state, hence the stream in the key.")
    w("struct PlanEntry {")
    w("  const void* ro_ptr; uint32_t ro_version; int64_t num_rows, ne; int offset_bits, device; cudaStream_t stream; int type_tag;")
    w("  torch::Tensor ws, ro_keep;")
    w("  int32_t reserved;                   // of the descriptor that the workspace was planned for")
    w("};")
    w("std::mutex g_mu;")
    w("std::list<PlanEntry> g_plans;          // most recently used first")
    w("constexpr size_t kMaxPlans = 8;")
    w("")
    w("struct Entry {   // the C entry points of one value type")
    w("  int (*workspace_bytes)(const flexspmv_desc*, size_t*);")
    w("  int (*plan)(const flexspmv_desc*, const void* const*, const void*, void*, size_t, void*);")
    w("  int (*launch)(const flexspmv_desc*, const void* const*, const void* const*, const void*, void* const*, void*, size_t, void*);")
    w("  int (*uses_longest_row)(const flexspmv_desc*);")
    w("  int (*device_status)(const void*, int32_t*, void*);")
    w("  int type_tag;")
    w("};")
    for i, dt in enumerate(dtypes):
        s = f"{symbol}_{CTYPE[dt][1]}"
        w(f"const Entry kEntry_{CTYPE[dt][1]} = {{flexspmv_{s}_workspace_bytes, flexspmv_{s}_plan_indexed, flexspmv_{s}_launch, "
          f"flexspmv_{s}_uses_longest_row, flexspmv_{s}_device_status, {i}}};")
    w("")
    w("// A planned workspace; `d.reserved` becomes that of the descriptor it was planned for.  Where the tiles go by the longest row they")
    w("// are those of whole rows, unless the plan says that it has none (one read back at plan time, not while the stream is captured).")
    w("torch::Tensor planned_workspace(const Entry& e, flexspmv_desc& d, const void* const* indices, const torch::Tensor& ro,")
    w("                                bool has_rows, const torch::Tensor& like, cudaStream_t stream) {")
    w("  const void* ro_ptr = has_rows ? ro.data_ptr() : nullptr;")
    w("  const uint32_t ver = has_rows ? ro._version() : 0u;")
    w("  const int device = like.get_device();")
    w("  std::lock_guard<std::mutex> lock(g_mu);")
    w("  for (auto it = g_plans.begin(); it != g_plans.end(); ++it) {")
    w("    if (it->ro_ptr == ro_ptr && it->ro_version == ver && it->num_rows == d.num_rows && it->ne == d.num_edges &&")
    w("        it->offset_bits == d.offset_bits && it->device == device && it->stream == stream && it->type_tag == e.type_tag) {")
    w("      g_plans.splice(g_plans.begin(), g_plans, it);")
    w("      d.reserved = g_plans.front().reserved;")
    w("      return g_plans.front().ws;")
    w("    }")
    w("  }")
    w("  torch::Tensor ws;")
    w("  auto plan = [&] {")
    w("    size_t bytes = 0;")
    w("    int st = e.workspace_bytes(&d, &bytes);")
    w('    TORCH_CHECK(st == 0, "merged_spmv_launch (workspace size) failed: ", flexspmv_error_string(st));')
    w("    ws = torch::empty({(int64_t)bytes}, torch::TensorOptions().dtype(torch::kUInt8).device(like.device()));")
    w("    st = e.plan(&d, indices, ro_ptr, ws.data_ptr(), bytes, stream);")
    w('    TORCH_CHECK(st == 0, "merged_spmv_launch (plan) failed: ", flexspmv_error_string(st));')
    w("  };")
    w("  const int32_t unknown = d.reserved;")
    w("  cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;")
    w("  const int by_row = has_rows ? e.uses_longest_row(&d) : 0;        // bit 0: the tiles do")
    w("  if (by_row && cudaStreamIsCapturing(stream, &capturing) == cudaSuccess && capturing == cudaStreamCaptureStatusNone) {")
    w("    d.reserved = unknown | FLEXSPMV_LONGEST_ROW(32);")
    w("    plan();")
    w("    torch::Tensor out = torch::empty({1}, torch::TensorOptions().dtype(torch::kInt).device(like.device()));")
    w("    const int st = flexspmv_workspace_longest_row(ws.data_ptr(), out.data_ptr<int32_t>(), stream);")
    w('    TORCH_CHECK(st == 0, "merged_spmv_launch (longest row) failed: ", flexspmv_error_string(st));')
    w("    const int longest = out.item<int32_t>();")
    w("    d.reserved = longest ? unknown | FLEXSPMV_LONGEST_ROW(longest) : unknown;")
    w("    if (!longest && (by_row & 1)) plan();")
    w("  } else {")
    w("    plan();")
    w("  }")
    w("  g_plans.push_front(PlanEntry{ro_ptr, ver, d.num_rows, d.num_edges, d.offset_bits, device, stream, e.type_tag, ws,")
    w("                               has_rows ? ro : torch::Tensor(), d.reserved});")
    w("  while (g_plans.size() > kMaxPlans) g_plans.pop_back();")
    w("  return ws;")
    w("}")
    w("")
    # return type
    n_out = len(ir.outputs)
    ret = "void" if n_out == 0 else "std::tuple<" + ", ".join(["torch::Tensor"] * n_out) + ">"
    w(f"{ret} merged_spmv_launch_typed(const Entry& e, c10::ScalarType value_type,")
    w("    " + ",\n    ".join(params) + ") {")
    for n in values + idx_args + ["row_end_offsets"]:
        w(f'  TORCH_CHECK({n}.is_cuda(), "{n} must be a CUDA tensor");')
        w(f'  TORCH_CHECK({n}.is_contiguous(), "{n} must be contiguous");')
    for n in values:
        w(f'  TORCH_CHECK({n}.scalar_type() == value_type, "{n} dtype mismatch");')
    for n in idx_args:
        w(f'  TORCH_CHECK({n}.scalar_type() == torch::kInt, "{n} dtype mismatch");')
    if has_red:
        w('  TORCH_CHECK(row_end_offsets.scalar_type() == torch::kInt || row_end_offsets.scalar_type() == torch::kLong,')
        w('              "row_end_offsets dtype mismatch");')
        w('  TORCH_CHECK(row_end_offsets.numel() == num_rows + 1, "row_end_offsets must have length num_rows + 1");')
    ne_expr = f"{idx_args[0]}.numel()" if idx_args else "num_cols"
    w(f"  const int64_t ne = {ne_expr};")
    w('  TORCH_CHECK(ne > 0, "selector index must be non-empty");')
    w(f"  const c10::cuda::CUDAGuard guard({dispatch}.device());")
    w(f"  auto options_val = torch::TensorOptions().dtype(value_type).device({dispatch}.device());")
    out_vars = []
    for i, o in enumerate(ir.outputs):
        d = dim_of(o["shape"])
        tgt = str(o["target"])
        base = "num_rows" if tgt == "reducer" else (None if "sum" in tgt else "ne")
        shape = f"{d}" if base is None else (base if d == 1 else f"{base}, {d}")
        var = f"out_{i}_{o['name']}"
        w(f"  torch::Tensor {var} = torch::empty({{{shape}}}, options_val);      // every element is written by the kernel")
        out_vars.append(var)
    w("  flexspmv_desc d;")
    w(f"  d.num_rows = {'num_rows' if has_red else '0'}; d.num_edges = ne; d.num_vertices = num_cols;")
    w(f"  d.offset_bits = {'row_end_offsets.scalar_type() == torch::kLong ? 64 : 32' if has_red else '32'};")
    w("  d.tile_items = 0; d.max_ctas = 0; d.reserved = 0;")
    w("  cudaStream_t stream = at::cuda::getCurrentCUDAStream().stream();")
    w("  const void* values[] = {" + ", ".join(f"{n}.data_ptr()" for n in values) + ("" if values else "nullptr") + "};")
    w("  const void* indices[] = {" + ", ".join(f"{n}.data_ptr()" for n in idx_args) + ("" if idx_args else "nullptr") + "};")
    w(f"  torch::Tensor ws = planned_workspace(e, d, indices, row_end_offsets, {'true' if has_red else 'false'}, {dispatch}, stream);")
    w("  void* outputs[] = {" + ", ".join(f"{v}.data_ptr()" for v in out_vars) + ("" if out_vars else "nullptr") + "};")
    w(f"  const int st = e.launch(&d, values, indices, {'row_end_offsets.data_ptr()' if has_red else 'nullptr'}, outputs, ws.data_ptr(),")
    w("                          (size_t)ws.numel(), stream);")
    w('  TORCH_CHECK(st == 0, "merged_spmv_launch failed: ", flexspmv_error_string(st));')
    if out_vars:
        w("  return std::make_tuple(" + ", ".join(out_vars) + ");")
    w("}")
    w("")
    w(f"{ret} merged_spmv_launch_bind(")
    w("    " + ",\n    ".join(params) + ") {")
    w(f'  TORCH_CHECK({dispatch}.device().is_cuda(), "CUDA device required");')
    w(f"  switch ({dispatch}.scalar_type()) {{")
    for dt in dtypes:
        w(f"    case {_TORCH_TYPE[dt]}:")
        w(f"      return merged_spmv_launch_typed(kEntry_{CTYPE[dt][1]}, {_TORCH_TYPE[dt]}, {call_args});")
    w("    default:")
    w(f'      TORCH_CHECK(false, "Unsupported dtype for ValueT: ", {dispatch}.scalar_type(), " (compiled: {", ".join(dtypes)})");')
    w("  }")
    w("}")
    w("")
    w("// Status word of the most recently used workspace (synchronises the current stream): 0, or the FLEXSPMV_ERR_* a")
    w("// kernel raised (a bounded device-side wait ran out; the workspace was not planned for the problem).")
    w("int64_t device_status() {")
    w("  PlanEntry p;")
    w("  {")
    w("    std::lock_guard<std::mutex> lock(g_mu);")
    w("    if (g_plans.empty()) return 0;")
    w("    p = g_plans.front();")
    w("  }")
    w("  const c10::cuda::CUDAGuard guard(p.ws.device());")
    w("  torch::Tensor out = torch::zeros({1}, torch::TensorOptions().dtype(torch::kInt).device(p.ws.device()));")
    w(f"  const Entry& e = kEntry_{CTYPE[dtypes[0]][1]};      // the status word sits at the same place for every value type")
    w("  const int st = e.device_status(p.ws.data_ptr(), out.data_ptr<int32_t>(), at::cuda::getCurrentCUDAStream().stream());")
    w('  TORCH_CHECK(st == 0, "device_status failed: ", flexspmv_error_string(st));')
    w("  return out.item<int32_t>();")
    w("}")
    w("")
    w("}  // namespace")
    w("")
    w("PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {")
    w('  m.def("merged_spmv_launch", &merged_spmv_launch_bind, "Run the fused gather-map-reduce kernel"')
    for n in values + idx_args + ["row_end_offsets", "num_rows", "num_cols"]:
        w(f'        , py::arg("{n}")')
    w("  );")
    w('  m.def("device_status", &device_status, "Status word of the most recent workspace (synchronises)");')
    w("}")
    return "\n".join(L) + "\n"


def generate_binding_code(project_root: str, inputs, outputs, selector_register, map_operations=None,
                          reducer_operations=None, aggregator_operations=None, name: str = "fused",
                          dtypes: Iterable[str] = ("float32", "float64"), ir: Optional[GraphIR] = None) -> str:
    """Writes ``<project_root>/merged_binding.cu`` and, under ``<project_root>/include``, the generated kernel units
    and the kernel headers it includes.  Takes the tracer's lists as the reference's function does
    (codegen/merged_gen_binding.py:9-21) plus the three operation lists (the kernels are generated here, not in
    a separate step), or a ready ``GraphIR``.  Returns the path of the binding."""
    if ir is None:
        ir = GraphIR(name, list(inputs), list(outputs), list(selector_register), list(map_operations or []),
                     list(reducer_operations or []), list(aggregator_operations or []))
    dtypes = tuple(dtypes)
    symbol = f"merged_{ir.name}"
    inc = os.path.join(project_root, "include")
    os.makedirs(inc, exist_ok=True)

    def write_if_changed(path: str, text: str):
        if not os.path.exists(path) or open(path).read() != text:
            with open(path, "w") as f:
                f.write(text)

    for h in KERNEL_HEADERS:
        with open(os.path.join(_PKG, "csrc", h)) as f:
            write_if_changed(os.path.join(inc, h), f.read())
    with open(os.path.join(_ROOT, "include", "flexspmv.h")) as f:
        write_if_changed(os.path.join(inc, "flexspmv.h"), f.read())
    for dt in dtypes:
        sym = f"{symbol}_{CTYPE[dt][1]}"
        write_if_changed(os.path.join(inc, f"merged_graph_{sym}.cuh"), emit_graph(ir, dt, sym, windows=False))
    path = os.path.join(project_root, "merged_binding.cu")
    write_if_changed(path, binding_source(ir, symbol, dtypes))
    return path


# flags a driver should add to its load(...) call: the sm_100a target (the kernels use bulk async copies and
# mbarriers); everything else in the reference's call may stay as it is
EXTRA_CUDA_CFLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "--expt-relaxed-constexpr", "-diag-suppress", "177"]


def load_binding(ir: GraphIR, project_root: str, dtypes: Iterable[str] = ("float32", "float64"), verbose: bool = False):
    """generate_binding_code + the reference's build step (test_full/easier_full.py:359-373): returns the loaded
    extension module, whose ``merged_spmv_launch`` the runtime wrapper calls."""
    import hashlib
    from torch.utils.cpp_extension import load
    src = generate_binding_code(project_root, None, None, None, ir=ir, dtypes=dtypes)
    h = hashlib.sha1()
    for root, _, files in sorted(os.walk(project_root)):
        for fn in sorted(files):
            if fn.endswith((".cu", ".cuh", ".h")):
                with open(os.path.join(root, fn), "rb") as f:
                    h.update(f.read())
    build_dir = os.path.join(project_root, "build")
    os.makedirs(build_dir, exist_ok=True)
    os.environ.setdefault("TORCH_CUDA_ARCH_LIST", "10.0a")
    return load(name=f"new_{ir.name}_{h.hexdigest()[:12]}", sources=[src],
                extra_include_paths=[project_root, os.path.join(project_root, "include")],
                extra_cflags=["-O3", "-DNDEBUG"], extra_cuda_cflags=["-O3", "-DNDEBUG"] + EXTRA_CUDA_CFLAGS,
                build_directory=build_dir, verbose=verbose)
