"""The heat-geodesic work a program has this package do, case by case, through its public calls.

``listed()`` names the cases and ``draw(rng)`` makes more of the same ranges; ``prepare`` makes what
a program holds before the call, ``run`` is one pass, ``work`` what a pass cannot do without,
``tolerance`` how far another correct implementation may be off, and ``exact`` the same outputs in
64-bit torch without this package's code (Jacobi sweeps for the heat system, whose every entry
keeps its own precision down to 1e-170, and conjugate gradients for the Poisson system).

A mesh is one of

- ``torus``: the revolved grid with jittered vertices (0.1 of the mean edge), ``cols x rows``;
- ``sphere``: an icosphere with 1 % radial noise, ``level`` subdivisions;
- ``sheet``: an open, bumpy, jittered height field, ``cols x rows`` vertices (it has a rim).
"""

import functools
import math

import numpy as np
import torch

from ordito_b200 import _lib, creation
from ordito_b200.device import DeviceArray
from ordito_b200.heat import BatchStep, extend_scalar, heat_geodesic, heat_geodesic_batch, heat_operators
from ordito_b200.mesh import Trimesh
from ordito_b200.packed import PackedMeshes

# ---------------------------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------------------------


def listed():
    return [
        # One query on a small mesh, everything built for the call: latency and launches.
        {"name": "query_sphere_642", "kind": "query", "mesh": "sphere", "level": 3, "method": "meshlab", "sources": 1},
        # One query on the mid-size sphere of the single-query configuration.
        {"name": "query_sphere_10k", "kind": "query", "mesh": "sphere", "level": 5, "method": "meshlab", "sources": 1},
        # One query on an open scan-like patch of odd size by the discretization that pins its rim.
        {"name": "query_sheet_igl_20k", "kind": "query", "mesh": "sheet", "cols": 151, "rows": 133, "method": "igl",
         "sources": 3},
        # One query on the benchmark's torus, nothing held: assembly, analysis, factors, solves.
        {"name": "query_torus_131k", "kind": "query", "mesh": "torus", "cols": 512, "rows": 256, "method": "meshlab",
         "sources": 1},
        # One query on a scan of millions of vertices, the largest mesh of the configurations.
        {"name": "query_torus_2600k", "kind": "query", "mesh": "torus", "cols": 2048, "rows": 1280,
         "method": "meshlab", "sources": 1},
        # An interactive program: one more query on a mesh it keeps (both factors held).
        {"name": "resident_torus_131k", "kind": "resident", "mesh": "torus", "cols": 512, "rows": 256, "sources": 1},
        # The serving loop's step: 64 single-source queries on a resident mesh, recorded once.
        {"name": "served_torus_131k_64", "kind": "served", "mesh": "torus", "cols": 512, "rows": 256, "columns": 64},
        # A batch by the plain call with its defaults (one refinement step), ragged source sets.
        {"name": "batch_sphere_41k_16", "kind": "batch", "mesh": "sphere", "level": 6, "columns": 16,
         "poisson": "factor", "refine": 1},
        # A batch whose Poisson systems go through the mixed-precision multigrid solve.
        {"name": "batch_multigrid_262k_8", "kind": "batch", "mesh": "torus", "cols": 640, "rows": 410, "columns": 8,
         "poisson": "multigrid", "refine": 0},
        # A data set of many small and middling meshes solved as one system.
        {"name": "packed_48_meshes_16", "kind": "packed", "meshes": 48, "columns": 16, "largest": 20000},
        # The operators alone, for a program with its own solver: pattern, table, rows.
        {"name": "operators_torus_655k", "kind": "operators", "mesh": "torus", "cols": 1024, "rows": 640,
         "method": "meshlab"},
        # A field extended from a few vertices of a resident mesh (colours, weights, landmarks).
        {"name": "extend_torus_131k", "kind": "extend", "mesh": "torus", "cols": 512, "rows": 256, "sources": 12},
    ]


def draw(rng):
    kind = rng.choice(["query", "query", "query", "resident", "served", "served", "batch", "batch", "packed",
                       "operators", "extend"])
    if kind == "packed":
        return {"kind": kind, "meshes": rng.randint(2, 64), "columns": rng.randint(1, 16),
                "largest": _log_int(rng, 500, 20000)}
    largest = {"query": 400_000, "resident": 300_000, "served": 160_000, "batch": 160_000, "operators": 1_500_000,
               "extend": 200_000}[kind]
    case = {"kind": kind}
    case.update(_draw_mesh(rng, largest))
    if kind in ("query", "operators"):
        case["method"] = rng.choice(["meshlab", "meshlab", "igl", "potpourri3d"])
    if kind in ("query", "resident", "extend"):
        case["sources"] = _log_int(rng, 1, 40)
    if kind in ("served", "batch"):
        case["columns"] = _log_int(rng, 1, 64)
    if kind == "batch":
        case["poisson"] = rng.choice(["factor", "factor", "multigrid"])
        case["refine"] = rng.choice([0, 1])
        if case["poisson"] == "multigrid":
            case["columns"] = min(case["columns"], 16)
    return case


def _log_int(rng, low, high):
    return min(high, max(low, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def _draw_mesh(rng, largest):
    mesh = rng.choice(["torus", "torus", "sheet", "sphere"])
    if mesh == "sphere":
        return {"mesh": mesh, "level": rng.choice([k for k in range(2, 7) if 10 * 4**k + 2 <= largest])}
    n = _log_int(rng, 200, largest)
    cols = max(12, int(round(math.sqrt(n * rng.uniform(1.0, 2.5)))))
    return {"mesh": mesh, "cols": cols, "rows": max(8, n // cols)}


# ---------------------------------------------------------------------------------------------
# Meshes, made on the GPU from the seed
# ---------------------------------------------------------------------------------------------


def _sizes(case):
    """(vertices, faces) of a case's mesh."""
    if case["kind"] == "packed":
        shapes = [_sizes(dict(m, kind="one")) for m in _packed_specs(case)]
        return sum(v for v, _ in shapes), sum(f for _, f in shapes)
    if case["mesh"] == "sphere":
        return 10 * 4 ** case["level"] + 2, 20 * 4 ** case["level"]
    c, r = case["cols"], case["rows"]
    return (c * r, 2 * c * r) if case["mesh"] == "torus" else (c * r, 2 * (c - 1) * (r - 1))


def _entries(case):
    """Stored entries of the operators: the vertices and every edge both ways."""
    n, f = _sizes(case)
    if case["mesh"] == "sheet":
        c, r = case["cols"], case["rows"]
        edges = (c - 1) * r + c * (r - 1) + (c - 1) * (r - 1)
    else:
        edges = 3 * f // 2
    return n + 2 * edges


@functools.lru_cache(maxsize=8)
def _icosphere(level):
    v, f = creation.icosphere(level)
    return torch.from_numpy(v).cuda().double(), torch.from_numpy(f).cuda()


def _grid(cols, rows, wrap):
    i, j = torch.meshgrid(torch.arange(cols, device="cuda"), torch.arange(rows, device="cuda"), indexing="ij")
    if not wrap:
        ci, cj = i[:-1, :-1].reshape(-1), j[:-1, :-1].reshape(-1)
    else:
        ci, cj = i.reshape(-1), j.reshape(-1)
    ni, nj = (ci + 1) % cols, (cj + 1) % rows
    a, b, c, d = ci * rows + cj, ni * rows + cj, ni * rows + nj, ci * rows + nj
    faces = torch.stack((torch.stack((a, b, c), 1), torch.stack((a, c, d), 1)), 1).reshape(-1, 3)
    return i.double(), j.double(), faces.int()


def _mesh(case, seed):
    """``(vertices float32 (V, 3), faces int32 (F, 3))`` on the GPU."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))

    def noise(*shape):
        return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float64)

    if case["mesh"] == "sphere":
        base, faces = _icosphere(case["level"])
        return (base * (1.0 + 0.01 * noise(base.shape[0], 1))).float().contiguous(), faces.clone()
    cols, rows = case["cols"], case["rows"]
    if case["mesh"] == "torus":
        i, j, faces = _grid(cols, rows, True)
        u, v = 2.0 * math.pi * i / cols, 2.0 * math.pi * j / rows
        ring = 1.0 + 0.3 * torch.cos(v)
        xyz = torch.stack((ring * torch.cos(u), ring * torch.sin(u), 0.3 * torch.sin(v)), -1).reshape(-1, 3)
    else:
        i, j, faces = _grid(cols, rows, False)
        x, y = i / (cols - 1) * cols / rows, j / (rows - 1)
        xyz = torch.stack((x, y, 0.15 * torch.sin(5.0 * x) * torch.cos(4.0 * y)), -1).reshape(-1, 3)
    p = xyz[faces.long()]
    edge = ((p[:, [1, 2, 0]] - p).square().sum(-1).sqrt()).mean()
    return (xyz + 0.1 * edge * noise(cols * rows, 3)).float().contiguous(), faces.contiguous()


@functools.lru_cache(maxsize=64)
def _packed_shapes(meshes, columns, largest):
    rng = np.random.default_rng(meshes * 1000003 + columns * 1009 + largest)
    specs = []
    for _ in range(meshes):
        n = int(round(math.exp(rng.uniform(math.log(150), math.log(largest)))))
        queries = int(rng.integers(1, columns + 1))
        if rng.random() < 0.3:
            level = max(2, min(6, int(math.log(max(n, 163) / 10.0, 4))))
            specs.append(("sphere", level, 0, queries))
        else:
            cols = max(12, int(round(math.sqrt(n * rng.uniform(1.0, 2.5)))))
            specs.append(("torus", cols, max(8, n // cols), queries))
    specs[0] = specs[0][:3] + (columns,)
    return tuple(specs)


def _packed_specs(case):
    out = []
    for name, a, b, queries in _packed_shapes(case["meshes"], case["columns"], case["largest"]):
        spec = {"mesh": name, "queries": queries}
        spec.update({"level": a} if name == "sphere" else {"cols": a, "rows": b})
        out.append(spec)
    return out


def _packed_inputs(case, seed):
    rng = np.random.default_rng(seed)
    meshes, queries = [], []
    for m, spec in enumerate(_packed_specs(case)):
        meshes.append(_mesh(spec, seed * 4099 + m))
        queries.append([int(s) for s in rng.choice(meshes[-1][0].shape[0], size=spec["queries"], replace=False)])
    return meshes, queries


def _sources(case, seed):
    """The source vertices of a case: a list of sets for the batched kinds, one set otherwise."""
    rng = np.random.default_rng(seed + 77)
    n = _sizes(case)[0]
    if case["kind"] == "served":
        return [[int(s)] for s in rng.choice(n, size=case["columns"], replace=False)]
    if case["kind"] == "batch":
        return [[int(s) for s in rng.choice(n, size=int(rng.integers(1, 4)), replace=False)]
                for _ in range(case["columns"])]
    return rng.choice(n, size=case["sources"], replace=False).astype(np.int32)


def _values(case, seed):
    return np.random.default_rng(seed + 78).uniform(-1.0, 1.0, size=case["sources"])


# ---------------------------------------------------------------------------------------------
# What a program holds, and one pass
# ---------------------------------------------------------------------------------------------


def _as_torch(array):
    return torch.as_tensor(array, device="cuda")


def prepare(case, seed):
    kind = case["kind"]
    state = {"kind": kind, "case": case}
    if kind == "packed":
        meshes, queries = _packed_inputs(case, seed)
        host = [(v.cpu().numpy(), f.cpu().numpy()) for v, f in meshes]
        state.update(packed=PackedMeshes(host, max_columns=case["columns"]), queries=queries)
        return state
    vertices, faces = _mesh(case, seed)
    state.update(vertices=vertices, faces=faces.reshape(-1))
    if kind == "operators":
        state["entries"] = _entries(case)
        return state
    sources = _sources(case, seed)
    state["sources"] = sources
    if kind == "query":
        return state
    mesh = state["mesh"] = Trimesh(vertices, state["faces"])
    if kind == "extend":
        state["values"] = _values(case, seed)
        mesh.heat_solver().factor(("heat",))
        return state
    solver = mesh.heat_solver(None, method="meshlab")
    solver.factor(("heat",) if case.get("poisson") == "multigrid" else ("heat", "poisson"))
    if case.get("poisson") == "multigrid":
        solver.poisson_multigrid  # noqa: B018 -- the hierarchy is built on first use
    if kind == "served":
        import ctypes  # noqa: PLC0415

        k = case["columns"]
        solver.tune(k)
        stream = ctypes.c_void_p(0)
        _lib.call("ob_stream_create", ctypes.byref(stream))
        state["step"] = BatchStep(
            mesh, solver, DeviceArray.from_host(np.array([s[0] for s in sources], dtype=np.int32)),
            DeviceArray.from_host(np.arange(k + 1, dtype=np.int32)), k,
            DeviceArray.empty((k, mesh.n_vertices), np.float64), stream)
        _lib.call("ob_stream_synchronize", stream)
    return state


def run(state):
    kind, case = state["kind"], state["case"]
    if kind == "query":
        return _as_torch(heat_geodesic(state["vertices"], state["faces"], state["sources"], method=case["method"]))
    if kind == "resident":
        return _as_torch(heat_geodesic(state["mesh"], state["sources"]))
    if kind == "served":
        return _as_torch(state["step"].launch(None))
    if kind == "batch":
        return _as_torch(heat_geodesic_batch(state["mesh"], state["sources"], refine=case["refine"],
                                             poisson=case["poisson"]))
    if kind == "packed":
        packed = state["packed"]
        k = packed.load(state["queries"])
        return _as_torch(packed.run(k))
    if kind == "operators":
        ops = heat_operators(state["vertices"], state["faces"], method=case["method"])
        n = state["entries"]
        return {"offsets": _as_torch(ops.laplacian.offsets), "columns": _as_torch(ops.laplacian.columns)[:n],
                "laplacian": _as_torch(ops.laplacian.values)[:n], "heat": _as_torch(ops.heat_system.values)[:n],
                "poisson": _as_torch(ops.poisson_system.values)[:n], "cot": _as_torch(ops.cot_entries),
                "normals": _as_torch(ops.face_normals), "areas": _as_torch(ops.face_areas)}
    return _as_torch(extend_scalar(state["mesh"], state["sources"], state["values"]))


# ---------------------------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------------------------


def _factor_values(n):
    """Values of a nested-dissection factor of a surface mesh: 31/4 n log2 n (George 1973)."""
    return 7.75 * n * math.log2(max(n, 2))


def work(case):
    n, f = _sizes(case)
    kind = case["kind"]
    mesh_in = 12 * n + 12 * f
    if kind == "query":
        # Mesh in, distances out; two solves by a method of optimal order, ~500 flops a vertex.
        return {"bytes": mesh_in + 8 * n, "flops": 1000 * n + 200 * f}
    if kind == "operators":
        nnz = _entries(case)
        return {"bytes": mesh_in + 4 * (n + 1) + (4 + 3 * 8) * nnz + 28 * f, "flops": 80 * f + 4 * nnz}
    k = 2 if kind == "extend" else case.get("columns", 1)
    systems = 1 if kind == "extend" or case.get("poisson") == "multigrid" else 2
    if kind == "packed":
        values = sum(_factor_values(_sizes(dict(m, kind="one"))[0]) for m in _packed_specs(case))
    else:
        values = _factor_values(n)
    # The held factors once, the corners' tables of the divergence once, the fields out; each factor
    # value is one multiply-add a column and direction.
    out = {"bytes": systems * 8 * values + 8 * n * (1 if kind == "extend" else k), "flops": systems * 4 * values * k}
    if kind != "extend":
        out["bytes"] += 144 * f
        out["flops"] += 60 * f * k
    if case.get("poisson") == "multigrid":
        out["bytes"] += 8 * 7 * n
        out["flops"] += 500 * n * k
    return out


def tolerance(case):
    """About four times what the package's outputs measured off ``exact`` over these ranges."""
    if case["kind"] == "operators":
        # float32 geometry, one rounding an operation (6e-8 measured); whole numbers are exact.
        return {"rel": 2.5e-7, "max": 2e-6}
    # Distances and extensions: float64 solves of operators from float32 geometry (1e-9 to 1e-8
    # measured, 2.3e-7 on grids of cells six times as long as wide); the plain call's conjugate
    # gradients stop at relative residuals of 1e-8 and 1e-6 of an entry.
    return {"rel": 1e-6, "max": 1e-5}


# ---------------------------------------------------------------------------------------------
# The same outputs in 64 bits, by plain torch
# ---------------------------------------------------------------------------------------------


def _assemble(x, faces, method, t_floor=True):
    """L, the lumped mass, the time step and the faces' terms of a mesh, from float64 positions."""
    n = x.shape[0]
    p = x[faces]  # (F, 3, 3)
    side = torch.stack((p[:, 2] - p[:, 1], p[:, 0] - p[:, 2], p[:, 1] - p[:, 0]), 1)  # opposite each corner
    normal = torch.linalg.cross(p[:, 1] - p[:, 0], p[:, 2] - p[:, 0])
    double = normal.norm(dim=1)
    unit, area = normal / double[:, None], 0.5 * double
    cot = torch.stack([-(side[:, (e + 1) % 3] * side[:, (e + 2) % 3]).sum(1) for e in range(3)], 1)
    cot = cot / (2.0 * double)[:, None]  # half cotangents
    i = faces[:, [1, 2, 0]].reshape(-1)
    j = faces[:, [2, 0, 1]].reshape(-1)
    c = cot.reshape(-1)
    diagonal = torch.zeros(n, dtype=torch.float64, device="cuda").index_add_(0, i, -c).index_add_(0, j, -c)
    own = torch.arange(n, device="cuda")
    lap = torch.sparse_coo_tensor(torch.stack((torch.cat((i, j, own)), torch.cat((j, i, own)))),
                                  torch.cat((c, c, diagonal)), (n, n)).coalesce()
    length = side.norm(dim=2)
    if method == "igl":
        sq = length.square()
        obtuse = cot < 0.0
        share = torch.stack([0.25 * (sq[:, (e + 1) % 3] * cot[:, (e + 1) % 3] + sq[:, (e + 2) % 3] * cot[:, (e + 2) % 3])
                             for e in range(3)], 1)
        blunt = torch.where(obtuse, 0.5, 0.25) * area[:, None]
        share = torch.where(obtuse.any(1)[:, None], blunt, share)
    else:
        share = (area / 3.0)[:, None].expand(-1, 3)
    mass = torch.zeros(n, dtype=torch.float64, device="cuda").index_add_(0, faces.reshape(-1), share.reshape(-1))
    if method == "meshlab":
        h = length.mean()
    else:
        at, to = lap.indices()
        upper = to > at
        h = (x[at[upper]] - x[to[upper]]).norm(dim=1).mean()
    t = float(h) ** 2
    if t_floor:
        box = x.max(0).values - x.min(0).values
        t = max(t, (float(box.norm()) / 400.0) ** 2)
    return {"lap": lap, "mass": mass, "t": t, "cot": cot, "unit": unit, "area": area, "x": x, "faces": faces}


def _csr(at, to, values, n):
    return torch.sparse_coo_tensor(torch.stack((at, to)), values, (n, n)).coalesce().to_sparse_csr()


def _diffuse(a, t, rhs, keep=None):
    """``(M - t L) u = rhs`` by damped Jacobi sweeps: sums of almost only positive terms, so every
    entry converges in its own precision. ``keep``: the free vertices."""
    n = rhs.shape[0]
    at, to = a["lap"].indices()
    values = -t * a["lap"].values()
    off = at != to
    if keep is not None:
        off = off & keep[at] & keep[to]
        rhs = rhs * keep[:, None]
    diagonal = torch.empty(n, dtype=torch.float64, device="cuda")
    diagonal[at[at == to]] = values[at == to]
    diagonal = diagonal + a["mass"]
    # Rows with weights of both signs (obtuse faces) are damped to where the sweeps contract.
    spread = torch.zeros(n, dtype=torch.float64, device="cuda").index_add_(0, at[off], values[off].abs())
    damped = torch.maximum(diagonal, 0.52 * (diagonal + spread))
    own = torch.arange(n, device="cuda")
    sweep = _csr(torch.cat((at[off], own)), torch.cat((to[off], own)),
                 torch.cat((-values[off] / damped[at[off]], (damped - diagonal) / damped)), n)
    first = rhs / damped[:, None]
    u = first.clone()
    for _ in range(400):
        for _ in range(63):
            u = torch.addmm(first, sweep, u)
        new = torch.addmm(first, sweep, u)
        change = (new - u).abs()
        u = new
        if bool((change <= 2e-14 * u.abs()).all()) and bool((u != 0).any(1).sum() >= (n if keep is None else keep.sum()) * 0.999):
            break
    return u


def _integrate(a, rhs, shift=0.0):
    """``(-L + shift) phi = rhs``, up to a constant (the shift to the sources takes it out), by
    Jacobi-preconditioned conjugate gradients, the columns in step."""
    n = rhs.shape[0]
    rhs = rhs - rhs.mean(0)
    at, to = a["lap"].indices()
    values = -a["lap"].values() + torch.where(at == to, shift, 0.0)
    matrix = _csr(at, to, values, n)
    diagonal = torch.empty(n, dtype=torch.float64, device="cuda")
    diagonal[at[at == to]] = values[at == to]
    inverse = (1.0 / diagonal)[:, None]
    x, r = torch.zeros_like(rhs), rhs.clone()
    z = inverse * r
    p, rz = z.clone(), (r * z).sum(0)
    goal = 1e-13 * rhs.norm(dim=0)
    for i in range(60000):
        q = matrix @ p
        alpha = torch.where(rz > 0, rz / (p * q).sum(0), 0.0)
        x += alpha * p
        r -= alpha * q
        r -= r.mean(0)
        if i % 50 == 49 and bool((r.norm(dim=0) <= goal).all()):
            break
        z = inverse * r
        new = (r * z).sum(0)
        p = z + torch.where(rz > 0, new / rz, 0.0) * p
        rz = new
    return x


def _divergence(a, u):
    """Minus the divergence of the faces' unit gradients of the columns of ``u``."""
    out = torch.zeros_like(u)
    x, faces, cot = a["x"], a["faces"], a["cot"]
    p = x[faces]
    side = torch.stack((p[:, 2] - p[:, 1], p[:, 0] - p[:, 2], p[:, 1] - p[:, 0]), 1)
    turned = torch.linalg.cross(a["unit"][:, None, :].expand(-1, 3, -1), side) / (2.0 * a["area"])[:, None, None]
    for c in range(u.shape[1]):
        w = u[:, c][faces]
        w = w / w.abs().max(1, keepdim=True).values.clamp_min(1e-300)
        g = (w[:, :, None] * turned).sum(1)
        g = g / g.abs().max(1, keepdim=True).values.clamp_min(1e-300)
        g = g / g.norm(dim=1, keepdim=True).clamp_min(1e-300)
        along = (side * g[:, None, :]).sum(2)  # each side with the gradient
        for e in range(3):
            b, d = (e + 1) % 3, (e + 2) % 3  # corner e's edges: side d towards corner b, side b from corner d
            out[:, c].index_add_(0, faces[:, e], cot[:, d] * along[:, d] - cot[:, b] * along[:, b])
    return out


def _shift(phi, sources):
    at = torch.tensor(sources, dtype=torch.long, device="cuda")
    offset = phi[at].mean()
    return phi - offset if phi.mean() - offset >= 0 else offset - phi


def _seed(n, sets):
    u = torch.zeros(n, len(sets), dtype=torch.float64, device="cuda")
    for c, s in enumerate(sets):
        u[torch.tensor(np.asarray(s), dtype=torch.long, device="cuda"), c] = 1.0
    return u


def _distances(a, sets, method):
    n = a["x"].shape[0]
    seeds = _seed(n, sets)
    heat = _diffuse(a, a["t"], seeds)
    if method == "igl":
        faces = a["faces"]
        i, j = faces[:, [1, 2, 0]].reshape(-1), faces[:, [2, 0, 1]].reshape(-1)
        key, count = torch.unique(torch.minimum(i, j) * n + torch.maximum(i, j), return_counts=True)
        rim = key[count == 1]
        if rim.numel():
            keep = torch.ones(n, dtype=torch.bool, device="cuda")
            keep[rim // n] = False
            keep[rim % n] = False
            heat = 0.5 * (heat + _diffuse(a, a["t"], seeds, keep))
    phi = _integrate(a, _divergence(a, heat), 1e-6 if method == "potpourri3d" else 0.0)
    return torch.stack([_shift(phi[:, c], np.asarray(s)) for c, s in enumerate(sets)])


def exact(case, seed):
    kind = case["kind"]
    if kind == "packed":
        return _exact_packed(case, seed)
    vertices, faces = _mesh(case, seed)
    x, tri = vertices.double(), faces.long()
    if kind == "operators":
        a = _assemble(x, tri, case["method"], t_floor=False)
        lap = a["lap"]
        at, to = lap.indices()
        heat = -a["t"] * lap.values() + torch.where(at == to, a["mass"][at], 0.0)
        offsets = torch.zeros(x.shape[0] + 1, dtype=torch.long, device="cuda")
        offsets[1:] = torch.bincount(at, minlength=x.shape[0]).cumsum(0)
        return {"offsets": offsets.int(), "columns": to.int(), "laplacian": lap.values(), "heat": heat,
                "poisson": -lap.values(), "cot": a["cot"], "normals": a["unit"], "areas": a["area"]}
    sources = _sources(case, seed)
    if kind == "extend":
        a = _assemble(x, tri, "potpourri3d")
        at = torch.from_numpy(sources).long().cuda()
        rhs = torch.zeros(x.shape[0], 2, dtype=torch.float64, device="cuda")
        rhs[at, 0] = 1.0
        rhs[at, 1] = torch.from_numpy(_values(case, seed)).cuda()
        u = _diffuse(a, a["t"], rhs)
        return u[:, 1] / u[:, 0]
    method = case.get("method", "meshlab")
    a = _assemble(x, tri, method)
    sets = sources if kind in ("served", "batch") else [sources]
    out = _distances(a, sets, method)
    return out if kind in ("served", "batch") else out[0]


def _exact_packed(case, seed):
    """Mesh by mesh; 0 where a mesh has no query in a column."""
    meshes, queries = _packed_inputs(case, seed)
    blocks = []
    for (vertices, faces), q in zip(meshes, queries):
        a = _assemble(vertices.double(), faces.long(), "meshlab")
        block = torch.zeros(case["columns"], vertices.shape[0], dtype=torch.float64, device="cuda")
        block[: len(q)] = _distances(a, [[s] for s in q], "meshlab")
        blocks.append(block)
    return torch.cat(blocks, 1)
