"""The workloads this framework's speed is measured on, each through the entry point a user's program calls.

A case names a kind of work, its sizes and its value type.  ``prepare`` builds on the GPU, from a seed alone, what a
program holds before the call: the matrix or mesh, the state vectors and -- for the time-stepping forms -- the bound
launch or the model object.  ``run`` makes one call.  Every kind is drawn over the sizes it meets in use, odd ones
among them.

  poisson2d, poisson3d   y = A x with 5- / 7-point Laplacians: bound once with ``prepare``, launched every iteration
                         (solvers, explicit time steps)
  banded27               y = A x with 27 columns a row near the diagonal (finite elements, 3-D meshes), ``launch_into``
  powerlaw               y = A x with power-law row lengths and random columns (graphs), the operator call that the
                         runtime wrapper makes, which allocates its outputs
  spring_mass            forces on a lattice of particles with 8 neighbours each, bound once
  rusanov                finite-volume fluxes over the faces of a triangulated square, bound once
  swe_step               one Runge-Kutta step of the shallow-water model, replayed from its CUDA graph
  mixed_dims             a traced graph of mixed widths (2 and 6 values a record, two reducers, a per-edge output),
                         the operator call
  edge_sum               a graph without a reducer: per-edge products and their global sum, the operator call
  sort_edges             set-up of an unsorted reducer: stable sort of the edges by row, CSR offsets, one per-edge
                         tensor brought into the sorted order
"""
from __future__ import annotations

import math

import torch

from flexspmv_b200 import graphs, problems
from flexspmv_b200.binding import load_builtin
from flexspmv_b200.multi_gpu import poisson3d_planes_device
from flexspmv_b200.python_wrapper.dynamic_replace_submodule import permute_edges, sort_edges_by_row
from flexspmv_b200.shallow_water import ShallowWaterStep

DTYPES = {"f32": torch.float32, "f64": torch.float64}
VBYTES = {"f32": 4, "f64": 8}
_EXT = {}


def _ext(name):
    """One operator object per graph for the whole program, as a program loads it."""
    if name not in _EXT:
        _EXT[name] = load_builtin(name)
    return _EXT[name]


def listed():
    return [
        # the smallest everyday matrix: 262 144 rows, a launch of a few microseconds inside a solver's loop
        {"name": "poisson2d_512_f64", "kind": "poisson2d", "n": 512, "dtype": "f64"},
        # an ordinary grid of odd size in single precision, int32 offsets
        {"name": "poisson3d_145_f32", "kind": "poisson3d", "n": 145, "dtype": "f32", "offset_bits": 32},
        # the benchmark's headline matrix: 134 M rows, 938 M non-zeros, int64 offsets
        {"name": "poisson3d_512_f64", "kind": "poisson3d", "n": 512, "dtype": "f64", "offset_bits": 64},
        # finite-element-like rows, longer than a stencil's and shorter than a graph's hubs
        {"name": "banded27_300k_f64", "kind": "banded27", "rows": 300007, "dtype": "f64"},
        # a graph of ordinary size, double precision
        {"name": "powerlaw_200k_f64", "kind": "powerlaw", "rows": 200003, "dtype": "f64"},
        # the benchmark's power-law matrix: 2^24 rows, about 260 M non-zeros
        {"name": "powerlaw_2e24_f32", "kind": "powerlaw", "rows": 1 << 24, "dtype": "f32"},
        # the benchmark's particle lattice
        {"name": "spring_mass_1024_f32", "kind": "spring_mass", "n": 1024, "dtype": "f32"},
        # the benchmark's triangulated square: 2.1 M cells
        {"name": "rusanov_1024_f64", "kind": "rusanov", "n": 1024, "dtype": "f64"},
        # the model on the same mesh, and on a small one where every launch counts
        {"name": "swe_step_1024_f64", "kind": "swe_step", "n": 1024},
        {"name": "swe_step_101_f64", "kind": "swe_step", "n": 101},
        # a traced graph that no configuration was tuned for
        {"name": "mixed_dims_250k_f32", "kind": "mixed_dims", "rows": 250001, "dtype": "f32"},
        # edges that arrive unsorted: 8.4 M of them for 1 M rows
        {"name": "sort_edges_8m", "kind": "sort_edges", "rows": 1048579, "edges": 8388593},
    ]


def _log_size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["poisson2d", "poisson3d", "banded27", "powerlaw", "spring_mass", "rusanov", "swe_step", "mixed_dims",
                       "edge_sum", "sort_edges"])
    case = {"kind": kind}
    if kind == "poisson2d":
        case.update(n=_log_size(rng, 100, 3000), dtype=rng.choice(["f32", "f64"]))
    elif kind == "poisson3d":
        case.update(n=_log_size(rng, 30, 400), dtype=rng.choice(["f32", "f64"]), offset_bits=rng.choice([32, 64]))
    elif kind == "banded27":
        case.update(rows=_log_size(rng, 10_000, 3_000_000), dtype=rng.choice(["f32", "f64"]))
    elif kind == "powerlaw":
        case.update(rows=_log_size(rng, 10_000, 8_000_000), dtype=rng.choice(["f32", "f64"]))
    elif kind == "spring_mass":
        case.update(n=_log_size(rng, 100, 2000), dtype=rng.choice(["f32", "f64"]))
    elif kind == "rusanov":
        case.update(n=_log_size(rng, 100, 1500), dtype=rng.choice(["f32", "f64"]))
    elif kind == "swe_step":
        case.update(n=_log_size(rng, 50, 1500))
    elif kind == "mixed_dims":
        case.update(rows=_log_size(rng, 10_000, 1_000_000), dtype=rng.choice(["f32", "f64"]))
    elif kind == "edge_sum":
        case.update(edges=_log_size(rng, 100_000, 60_000_000), dtype=rng.choice(["f32", "f64"]))
    else:
        rows = _log_size(rng, 1000, 8_000_000)
        case.update(rows=rows, edges=_log_size(rng, max(20_000, rows), 30_000_000))
    return case


# ---- inputs ------------------------------------------------------------------------------------------------------

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _uniform(g, shape, dtype, lo=-1.0, hi=1.0):
    return torch.rand(shape, generator=g, device="cuda", dtype=dtype) * (hi - lo) + lo


def _csr_from_candidates(cols, valid):
    """cols, valid: (rows, k).  Offsets (int32), columns of the valid entries in row order, their row ids."""
    ro = torch.zeros(cols.shape[0] + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(valid.sum(dim=1), dim=0, out=ro[1:])
    return ro.to(torch.int32), cols[valid].to(torch.int32)


def _poisson2d(n, dtype):
    idx = torch.arange(n * n, device="cuda")
    i, j = idx // n, idx % n
    steps = torch.tensor([-n, -1, 0, 1, n], device="cuda")
    valid = torch.stack([i > 0, j > 0, i >= 0, j < n - 1, i < n - 1], dim=1)
    ro, cols = _csr_from_candidates(idx[:, None] + steps, valid)
    stencil = torch.tensor([-1.0, -1.0, 4.0, -1.0, -1.0], device="cuda", dtype=dtype)
    return ro, cols, stencil.expand(n * n, 5)[valid].contiguous()


def _banded27(rows, g, dtype):
    """27 columns a row: nine runs of three around offsets of a 3-D mesh numbering, fewer at the ends."""
    m = max(2, int(round(rows ** (1.0 / 3.0))))
    steps = sorted(a * m * m + b * m + c for a in (-1, 0, 1) for b in (-1, 0, 1) for c in (-1, 0, 1))
    cols = torch.arange(rows, device="cuda")[:, None] + torch.tensor(steps, device="cuda")
    ro, cols = _csr_from_candidates(cols, (cols >= 0) & (cols < rows))
    return ro, cols, _uniform(g, (cols.numel(),), dtype)


def _lattice(n):
    idx = torch.arange(n * n, device="cuda")
    i, j = idx // n, idx % n
    steps = [(a, b) for a in (-1, 0, 1) for b in (-1, 0, 1) if (a, b) != (0, 0)]
    valid = torch.stack([(i + a >= 0) & (i + a < n) & (j + b >= 0) & (j + b < n) for a, b in steps], dim=1)
    ro, dst = _csr_from_candidates(idx[:, None] + torch.tensor([a * n + b for a, b in steps], device="cuda"), valid)
    return ro, _rows_of(ro).to(torch.int32), dst


def _triangles(n):
    """The n x n square split into 2 n^2 triangles (the cell numbering of ``problems.shallow_water``): per cell its three
    neighbours (the cell itself at a wall) and the outward normals and lengths of its faces."""
    hs = 1.0 / n
    sq = torch.arange(n * n, device="cuda")
    iy, ix = sq // n, sq % n
    cl, cu = 2 * sq, 2 * sq + 1
    nbr = torch.empty((2 * n * n, 3), dtype=torch.int64, device="cuda")
    nbr[0::2] = torch.stack([torch.where(iy > 0, 2 * (sq - n) + 1, cl), torch.where(ix < n - 1, 2 * (sq + 1) + 1, cl), cu], dim=1)
    nbr[1::2] = torch.stack([cl, torch.where(iy < n - 1, 2 * (sq + n), cu), torch.where(ix > 0, 2 * (sq - 1), cu)], dim=1)
    r = math.sqrt(0.5)
    face = torch.empty((2 * n * n, 3, 3), dtype=torch.float64, device="cuda")
    face[0::2] = torch.tensor([[0.0, -1.0, hs], [1.0, 0.0, hs], [-r, r, hs * math.sqrt(2.0)]], dtype=torch.float64, device="cuda")
    face[1::2] = torch.tensor([[r, -r, hs * math.sqrt(2.0)], [0.0, 1.0, hs], [-1.0, 0.0, hs]], dtype=torch.float64, device="cuda")
    return nbr, face


def _rusanov(n, g, dtype):
    nbr, face = _triangles(n)
    cells = 2 * n * n
    U = torch.stack([_uniform(g, (cells,), torch.float64, 0.9, 1.1), _uniform(g, (cells,), torch.float64, -0.2, 0.2),
                     _uniform(g, (cells,), torch.float64, -0.2, 0.2)], dim=1)
    own = torch.arange(cells, device="cuda").repeat_interleave(3)
    ro = (3 * torch.arange(cells + 1, device="cuda")).to(torch.int32)
    return ro, face.reshape(-1, 3).to(dtype).contiguous(), U.to(dtype).contiguous(), own.to(torch.int32), nbr.reshape(-1).to(torch.int32)


def _swe_mesh(n, g):
    nbr, face = _triangles(n)
    cells = 2 * n * n
    own = torch.arange(cells, device="cuda").repeat_interleave(3)
    nb, fc = nbr.reshape(-1), face.reshape(-1, 3)
    wall = nb == own
    fx, fy = fc[:, 0] * fc[:, 2], fc[:, 1] * fc[:, 2]
    zero = torch.zeros(cells, dtype=torch.float64, device="cuda")
    bx, by = zero.index_add(0, own[wall], -fx[wall]), zero.index_add(0, own[wall], -fy[wall])
    bcells = torch.unique(own[wall])
    inner = ~wall
    h = _uniform(g, (cells,), torch.float64, 0.95, 1.05)
    return {"src": nb[inner].to(torch.int32), "dst": own[inner].to(torch.int32), "bcells": bcells.to(torch.int32),
            "alpha": _uniform(g, (int(inner.sum()),), torch.float64, 0.4, 0.6), "sx": (-fx[inner]).contiguous(), "sy": (-fy[inner]).contiguous(),
            "bsx": bx[bcells].contiguous(), "bsy": by[bcells].contiguous(),
            "area": torch.full((cells,), 0.5 / (n * n), dtype=torch.float64, device="cuda"),
            "h": h, "uh": _uniform(g, (cells,), torch.float64, -0.05, 0.05), "vh": _uniform(g, (cells,), torch.float64, -0.05, 0.05)}


def _swe_dt(n):
    return 1e-4 / n       # far below the stability limit: thousands of steps stay in the same regime


def _mixed(rows, g, dtype):
    """Rows of 0 to 16 edges, in random order, whose two end points lie near the row."""
    ln = (torch.arange(rows, device="cuda") % 17)[torch.randperm(rows, generator=g, device="cuda")]
    ro = torch.zeros(rows + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(ln, dim=0, out=ro[1:])
    own = torch.repeat_interleave(torch.arange(rows, device="cuda"), ln)
    e = own.numel()
    near = lambda: (own + torch.randint(-200, 201, (e,), generator=g, device="cuda")).clamp_(0, rows - 1).to(torch.int32)
    return (ro.to(torch.int32), near(), near(), _uniform(g, (e, 2), dtype), _uniform(g, (e, 6), dtype), _uniform(g, (rows, 2), dtype))


def _inputs(case, seed):
    """The arrays of one case, named."""
    kind, g = case["kind"], _gen(seed)
    dt = DTYPES[case.get("dtype", "f64")]
    if kind in ("poisson2d", "poisson3d"):
        n = case["n"]
        if kind == "poisson2d":
            ro, cols, vals = _poisson2d(n, dt)
        else:
            ro, cols, vals = poisson3d_planes_device(n, 0, n, "cuda", dt, torch.int64 if case["offset_bits"] == 64 else torch.int32)
        return {"ro": ro, "cols": cols, "vals": vals, "x": _uniform(g, (ro.numel() - 1,), dt)}
    if kind == "banded27":
        ro, cols, vals = _banded27(case["rows"], g, dt)
        return {"ro": ro, "cols": cols, "vals": vals, "x": _uniform(g, (case["rows"],), dt)}
    if kind == "powerlaw":
        ro, cols, vals, x = problems.powerlaw_device(case["rows"], seed)
        return {"ro": ro, "cols": cols, "vals": vals.to(dt), "x": x.to(dt)}
    if kind == "spring_mass":
        n = case["n"]
        ro, src, dst = _lattice(n)
        h = 1.0 / n
        at = torch.arange(n * n, device="cuda")
        p = torch.stack([(at % n) * h, (at // n) * h], dim=1).to(torch.float64) + _uniform(g, (n * n, 2), torch.float64, -0.2 * h, 0.2 * h)
        p = p.to(dt).contiguous()
        L = ((p[dst.long()] - p[src.long()]).double().norm(dim=1) * _uniform(g, (dst.numel(),), torch.float64, 0.9, 1.1)).to(dt)
        return {"ro": ro, "src": src, "dst": dst, "L": L, "k": _uniform(g, (dst.numel(),), dt, 0.5, 2.0), "p": p}
    if kind == "rusanov":
        ro, face, U, own, nbr = _rusanov(case["n"], g, dt)
        return {"ro": ro, "face": face, "U": U, "own": own, "nbr": nbr}
    if kind == "swe_step":
        return _swe_mesh(case["n"], g)
    if kind == "mixed_dims":
        ro, s0, s1, ea, eb, vx = _mixed(case["rows"], g, dt)
        return {"ro": ro, "s0": s0, "s1": s1, "ea": ea, "eb": eb, "vx": vx}
    if kind == "edge_sum":
        e = case["edges"]
        nv = max(1, e // 8)
        sel = (torch.arange(e, device="cuda") // 8).clamp_(max=nv - 1).to(torch.int32)      # eight edges a vertex, in order
        return {"sel": sel, "ew": _uniform(g, (e, 2), dt, 0.0, 1.0), "vx": _uniform(g, (nv, 2), dt, 0.0, 1.0)}
    rows, e = case["rows"], case["edges"]
    return {"ids": torch.randint(0, rows, (e,), generator=g, device="cuda"), "w": _uniform(g, (e, 2), torch.float32)}


def prepare(case, seed):
    a = _inputs(case, seed)
    kind = case["kind"]
    st = {"kind": kind, "a": a}
    if kind in ("poisson2d", "poisson3d"):
        rows = a["ro"].numel() - 1
        st["y"] = torch.empty(rows, dtype=a["x"].dtype, device="cuda")
        st["step"] = _ext("spmv").prepare([a["vals"], a["x"]], [a["cols"]], a["ro"], [st["y"]], rows, a["cols"].numel(), rows)
    elif kind == "banded27":
        st["y"] = torch.empty_like(a["x"])
        st["ext"] = _ext("spmv")
    elif kind == "powerlaw":
        st["ext"] = _ext("spmv")
    elif kind == "spring_mass":
        rows = a["p"].shape[0]
        st["y"] = torch.empty_like(a["p"])
        st["step"] = _ext("spring_mass").prepare([a["L"], a["k"], a["p"]], [a["src"], a["dst"]], a["ro"], [st["y"]], rows,
                                                 a["dst"].numel(), rows)
    elif kind == "rusanov":
        rows = a["U"].shape[0]
        st["y"] = [torch.empty(rows, dtype=a["U"].dtype, device="cuda") for _ in range(3)]
        st["step"] = _ext("rusanov").prepare([a["face"], a["U"]], [a["own"], a["nbr"]], a["ro"], st["y"], rows, a["nbr"].numel(), rows)
    elif kind == "swe_step":
        st["model"] = ShallowWaterStep(a, dt=_swe_dt(case["n"]))
        st["model"].capture()
    elif kind == "mixed_dims":
        st["ext"] = _ext("mixed_dims")
    elif kind == "edge_sum":
        st["ext"] = _ext("edge_sum")
        st["no_rows"] = torch.zeros(1, dtype=torch.int32, device="cuda")
    else:
        st["rows"] = case["rows"]
    return st


def run(st):
    kind, a = st["kind"], st["a"]
    if kind in ("poisson2d", "poisson3d", "spring_mass", "rusanov"):
        st["step"].launch()
        return st["y"]
    if kind == "banded27":
        rows = a["x"].numel()
        st["ext"].launch_into([a["vals"], a["x"]], [a["cols"]], a["ro"], [st["y"]], rows, a["cols"].numel(), rows)
        return st["y"]
    if kind == "powerlaw":
        rows = a["x"].numel()
        return st["ext"].merged_spmv_launch(a["vals"], a["x"], a["cols"], a["ro"], rows, rows)
    if kind == "swe_step":
        st["model"].replay()
        return [a["h"], a["uh"], a["vh"]]
    if kind == "mixed_dims":
        rows = a["vx"].shape[0]
        return st["ext"].merged_spmv_launch(a["ea"], a["eb"], a["vx"], a["s0"], a["s1"], a["ro"], rows, rows)
    if kind == "edge_sum":
        return st["ext"].merged_spmv_launch(a["ew"], a["vx"], a["sel"], st["no_rows"], 0, a["vx"].shape[0])
    perm, ro = sort_edges_by_row(a["ids"], st["rows"])
    return {"perm": perm, "ro": ro, "w": permute_edges(a["w"], perm)}


# ---- what one pass cannot do without -----------------------------------------------------------------------------

def _powerlaw_edges(rows):
    return int(15.5 * rows)       # the generator's mean row length after rounding and clipping


def work(case):
    kind = case["kind"]
    vb = VBYTES[case.get("dtype", "f64")]

    def graph(name, rows, edges, vertices, offset_bytes=4):
        return problems.algorithmic_bytes(graphs.ALL_GRAPHS[name](), rows, edges, vertices, vb, offset_bytes)

    if kind == "poisson2d":
        n = case["n"]
        e = 5 * n * n - 4 * n
        return {"bytes": graph("spmv", n * n, e, n * n), "flops": 2 * e}
    if kind == "poisson3d":
        n = case["n"]
        e = 7 * n ** 3 - 6 * n * n
        return {"bytes": graph("spmv", n ** 3, e, n ** 3, case["offset_bits"] // 8), "flops": 2 * e}
    if kind == "banded27":
        r = case["rows"]
        return {"bytes": graph("spmv", r, 27 * r, r), "flops": 2 * 27 * r}
    if kind == "powerlaw":
        r = case["rows"]
        return {"bytes": graph("spmv", r, _powerlaw_edges(r), r), "flops": 2 * _powerlaw_edges(r)}
    if kind == "spring_mass":
        n = case["n"]
        e = 8 * n * n - 12 * n + 4
        return {"bytes": graph("spring_mass", n * n, e, n * n), "flops": 14 * e}
    if kind == "rusanov":
        c = 2 * case["n"] ** 2
        return {"bytes": graph("rusanov", c, 3 * c, c), "flops": 60 * 3 * c}
    if kind == "swe_step":
        # a step needs four flux evaluations one after the other: each reads the mesh and a state and writes the next
        # state and the running sum of the increments
        c = 2 * case["n"] ** 2
        e = 3 * c - 4 * case["n"]
        stage = e * (4 + 3 * 8) + (c + 1) * 4 + c * 8 * (1 + 3 + 3 + 3 + 3 + 3)
        return {"bytes": 4 * stage, "flops": 4 * (45 * e + 15 * c)}
    if kind == "mixed_dims":
        r = case["rows"]
        return {"bytes": graph("mixed_dims", r, 8 * r, r), "flops": 8 * r * 24}
    if kind == "edge_sum":
        e = case["edges"]
        return {"bytes": graph("edge_sum", 0, e, max(1, e // 8)), "flops": 4 * e}
    e, r = case["edges"], case["rows"]
    return {"bytes": e * (8 + 4) + (r + 1) * 8 + e * (4 + 8 + 8), "flops": 0}


def tolerance(case):
    """Four times what sums in another order showed against 64-bit (for fp64: exactly rounded) results."""
    kind = case["kind"]
    if kind == "sort_edges":
        return "exact"
    if kind == "swe_step":
        return {"rel": 1e-14, "max": 1e-13}
    if kind == "powerlaw":        # rows of up to 100 000 terms of either sign
        return {"rel": 2e-14, "max": 2e-12} if case["dtype"] == "f64" else {"rel": 6e-6, "max": 3e-4}
    if kind == "spring_mass":     # length minus rest length cancels to a tenth of either
        return {"rel": 8e-15, "max": 4e-13} if case["dtype"] == "f64" else {"rel": 4e-6, "max": 2e-4}
    return {"rel": 4e-15, "max": 2e-13} if case["dtype"] == "f64" else {"rel": 2e-6, "max": 1e-4}


# ---- the same results in 64 bits ---------------------------------------------------------------------------------

def _rows_of(ro):
    r = ro.long()
    return torch.repeat_interleave(torch.arange(r.numel() - 1, device=r.device), r[1:] - r[:-1])


def _sum_rows(terms, rows_of, rows):
    out = torch.zeros((rows,) + tuple(terms.shape[1:]), dtype=torch.float64, device=terms.device)
    return out.index_add_(0, rows_of, terms)


def _swe_delta(m, h, uh, vh):
    src, dst, b, nc = m["src"].long(), m["dst"].long(), m["bcells"].long(), m["area"].numel()
    rec = lambda phi: (1.0 - m["alpha"]) * phi[src] + m["alpha"] * phi[dst]
    hf, uf, vf = rec(h), rec(uh), rec(vh)
    u, v, p = uf / hf, vf / hf, 0.5 * hf * hf
    ux, vy, bp = uf * m["sx"], vf * m["sy"], 0.5 * h[b] ** 2
    return (-_sum_rows(ux + vy, dst, nc) / m["area"],
            -(_sum_rows((u * uf + p) * m["sx"] + u * vy, dst, nc) + _sum_rows(bp * m["bsx"], b, nc)) / m["area"],
            -(_sum_rows(v * ux + (v * vf + p) * m["sy"], dst, nc) + _sum_rows(bp * m["bsy"], b, nc)) / m["area"])


def exact(case, seed):
    kind, a = case["kind"], _inputs(case, seed)
    a = {k: (v.double() if v.is_floating_point() else v) for k, v in a.items()}
    if kind in ("poisson2d", "poisson3d", "banded27", "powerlaw"):
        rows = a["ro"].numel() - 1
        out = torch.zeros(rows, dtype=torch.float64, device="cuda")
        step = 1 << 24
        for r0 in range(0, rows, step):            # blocks of rows bound the memory of the products
            r1 = min(rows, r0 + step)
            e0, e1 = int(a["ro"][r0]), int(a["ro"][r1])
            terms = a["vals"][e0:e1] * a["x"][a["cols"][e0:e1].long()]
            out[r0:r1] = _sum_rows(terms, _rows_of(a["ro"][r0:r1 + 1]), r1 - r0)
        return (out,) if kind == "powerlaw" else out
    if kind == "spring_mass":
        d = a["p"][a["dst"].long()] - a["p"][a["src"].long()]
        n = (d * d).sum(dim=1).sqrt()
        f = (a["k"] * (n - a["L"]))[:, None] * d / n[:, None]
        return _sum_rows(f, a["src"].long(), a["p"].shape[0])
    if kind == "rusanov":
        face, own = a["face"], a["own"].long()
        nx, ny, ln = face[:, 0], face[:, 1], face[:, 2]

        def side(U):
            h, hu, hv = U[:, 0], U[:, 1], U[:, 2]
            un = (hu * nx + hv * ny) / h
            p = h * h * 4.905
            return U, (h * un, hu * un + p * nx, hv * un + p * ny), un.abs() + (9.81 * h).sqrt()

        (Ui, Fi, si), (Uj, Fj, sj) = side(a["U"][own]), side(a["U"][a["nbr"].long()])
        lam = torch.maximum(si, sj)
        return [_sum_rows((0.5 * (Fi[k] + Fj[k]) - 0.5 * lam * (Uj[:, k] - Ui[:, k])) * ln, own, a["U"].shape[0]) for k in range(3)]
    if kind == "swe_step":
        dt, x = _swe_dt(case["n"]), (a["h"], a["uh"], a["vh"])
        ds = [_swe_delta(a, *x)]
        for c in (0.5 * dt, 0.5 * dt, dt):
            ds.append(_swe_delta(a, *[x[k] + c * ds[-1][k] for k in range(3)]))
        return [x[k] + dt / 6 * (ds[0][k] + ds[1][k] + ds[2][k] + ds[3][k]) for k in range(3)]
    if kind == "mixed_dims":
        t1 = (a["vx"][a["s0"].long()] + a["vx"][a["s1"].long()]) * a["ea"]
        rows, of = a["vx"].shape[0], _rows_of(a["ro"])
        return (_sum_rows(-t1, of, rows), _sum_rows(a["eb"] * t1.repeat(1, 3) - 0.25, of, rows), t1)
    if kind == "edge_sum":
        prod = a["ew"] * a["vx"][a["sel"].long()]
        return (prod, prod.sum(dim=0))
    return None
