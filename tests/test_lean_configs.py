"""Configurations that FLEXSPMV_CFG_OVERRIDE may name for the warp kernel: each compiles, for both offset widths, with the second
configuration that the launch derives from it."""
import os
import subprocess

import pytest

from flexspmv_b200 import build, graphs
from flexspmv_b200.codegen.emit_cuda import emit_graph


def compile_unit(dtype, symbol, override, tmp_path, monkeypatch):
    monkeypatch.setenv("FLEXSPMV_CFG_OVERRIDE", override)
    src, obj = tmp_path / "unit.cu", tmp_path / "unit.o"
    src.write_text(emit_graph(graphs.spmv_graph(), dtype, symbol, windows=False))
    assert override.split("=")[1].replace(",", ", ") in src.read_text()
    # the host side alone sees every static assertion of the kernels' bodies
    r = subprocess.run([build.NVCC] + build.NVCC_FLAGS + ["--cuda", "-c", str(src), "-o", str(obj)], capture_output=True, text=True)
    return r.returncode, r.stdout + r.stderr


@pytest.mark.skipif(not os.path.exists(build.NVCC), reason="needs nvcc")
@pytest.mark.parametrize("dtype,override", [("float32", "spmv_f32_lean=512,5,2"), ("float32", "spmv_f32_lean=256,5,4"), ("float32", "spmv_f32_lean=32,5,16"),
                                            ("float64", "spmv_f64_lean=512,5,1"), ("float64", "spmv_f64_lean=384,5,2"),
                                            ("float64", "spmv_f64_lean=1024,5,1")])
def test_warp_kernel_overrides_compile(dtype, override, tmp_path, monkeypatch):
    code, log = compile_unit(dtype, override.split("_lean")[0], override, tmp_path, monkeypatch)
    assert code == 0, log[-2000:]


def test_every_compiled_warp_kernel_is_launched():
    """The library holds one warp kernel per graph, offset width and configuration: the plain form of the configuration that the
    emitter gives, the form for few chunks a warp of the one that the launch derives from it."""
    import re
    from flexspmv_b200.binding import DEFAULT_LIB
    symbols = subprocess.run(["nm", "-C", DEFAULT_LIB], check=True, capture_output=True, text=True).stdout
    found = {m.groups() for m in re.finditer(r"flex::(flex_warp\w*kernel)<\(anonymous namespace\)::gen_(spmv_f(?:32|64))::Graph, ([a-z ]+), "
                                             r"flex::WarpCfg<(\d+), 5, 1> ?>", symbols)}
    want = {(kernel, graph, offsets, threads) for graph, large, small in (("spmv_f32", "1024", "768"), ("spmv_f64", "768", "640"))
            for kernel, threads in (("flex_warp_kernel", large), ("flex_warp_ahead_kernel", small)) for offsets in ("int", "long long")}
    assert found == want
