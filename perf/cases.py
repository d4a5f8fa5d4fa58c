"""What this framework is timed on: the DEC operators, the multigrid solves and cycles, the batched
solves and wedges, and the learned smoother, each through the package's public entry points.

A case is a dict of plain values whose "kind" names the path:

  operators   one evaluation of the primal operators on a mesh: ∧01, ∧11, d1, ∧02, d0, the divergence
              dual_d1 (⋆1 d0 f) and the Laplacian -- what a time step of a physics code calls
  wedges      many ∧11 products in one batched call
  dual        the dual-dual operators: the Lie derivative, the dual Laplacian, the primal-dual wedge
  solve       (L + c I) u = b to a relative residual from u = 0, one or many right-hand sides
  cycles      multigrid_vcycles / multigrid_wcycles with the reference's smoother (Krylov CG)
  inverse     dec_Δ⁻¹: full multigrid with W-cycles and the CG smoother on the Laplacian
  batch       uneven solves over several hierarchies, a shift per right-hand side
  learned     solves smoothed by the per-vertex network
  train       Adam steps of that network, its loss and its gradient

Meshes are the ones the package's own workloads use (binary-subdivided unit icospheres; triangulated
grids with odd rows shifted by half a cell), made here with numpy so that the expected values (`exact`)
come from this file and torch alone.  Inputs are uniform[-1, 1), as those workloads draw them.
"""
import functools
import importlib.util
import math
import pathlib
import sys
from types import SimpleNamespace

import numpy as np
import torch

ROOT = pathlib.Path(__file__).resolve().parent.parent


def _dec():
    if "dec_b200" not in sys.modules:
        pkg = ROOT / "combinatorialspaces.jl_b200"
        spec = importlib.util.spec_from_file_location("dec_b200", pkg / "__init__.py",
                                                      submodule_search_locations=[str(pkg)])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["dec_b200"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["dec_b200"]


# ---- cases --------------------------------------------------------------------------------------

def listed():
    return [
        # the plain-operator workload at its own size: latency and launches count
        dict(name="operators_grid128_f64", kind="operators", mesh="grid", nx=128, ny=128, dtype="float64"),
        # a resolved sphere in double precision, the reference's own float type
        dict(name="operators_sphere8_f64", kind="operators", mesh="sphere", level=8, dtype="float64"),
        # the largest mesh of the workloads, single precision
        dict(name="operators_sphere9_f32", kind="operators", mesh="sphere", level=9, dtype="float32"),
        # the batched workload's wedge evaluations
        dict(name="wedges_1024_sphere7_f32", kind="wedges", mesh="sphere", level=7, count=1024, dtype="float32"),
        # dual-dual operators of a fluid step on a ragged mid-size grid
        dict(name="dual_grid_97x81", kind="dual", nx=97, ny=81),
        # one right-hand side in double precision (a time step's implicit solve): V(3,3) to 1e-10
        dict(name="solve_sphere6_f64_1", kind="solve", mesh="sphere", level=6, nrhs=1, precision=0, pre=3, post=3,
             ratio=4.0, inner=1, coarse_max=0, rtol=1e-10),
        # the headline: 32 right-hand sides on the L8 icosphere, FP32 cycles in FP64 refinement to 1e-8
        dict(name="solve_sphere8_f32_32", kind="solve", mesh="sphere", level=8, nrhs=32, precision=1, pre=0, post=2,
             ratio=3.0, inner=3, coarse_max=170, rtol=1e-8),
        # the uneven batch: 512 solves over icospheres L4-L7 and grids 65^2-513^2
        dict(name="batch_512_uneven", kind="batch", solves=512, small=0, large=3, draw=3, rtol=1e-8),
        # the reference's own cycle (3 CG steps before and after) on the double-precision workload's mesh
        dict(name="cycles_cg_sphere6", kind="cycles", mesh="sphere", level=6, nrhs=1, steps=3, mu=1, cycles=5),
        # the reference's inverse Laplacian with its defaults (3 CG steps, 5 W-cycles a level)
        dict(name="inverse_laplacian_grid", kind="inverse", nx=9, ny=9, levels=4, steps=3, cycles=5),
        # the learned smoother inside the mixed-precision solve
        dict(name="learned_sphere7_32", kind="learned", level=7, nrhs=32, sweeps=1, inner=2, rtol=1e-8),
        # one block of the training schedule: 10 Adam steps on two L6 fields, then loss and gradient
        dict(name="train_sphere6", kind="train", level=6, fields=2, batch=65536, steps=10),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["operators", "operators", "wedges", "dual", "solve", "solve", "cycles", "inverse", "batch",
                       "learned", "train"])
    dtype = rng.choice(["float64", "float32"])
    if kind == "operators":
        if rng.random() < 0.7:
            return dict(kind=kind, mesh="grid", nx=_log_int(rng, 24, 1200), ny=_log_int(rng, 24, 1200), dtype=dtype)
        return dict(kind=kind, mesh="sphere", level=rng.randint(4, 8), dtype=dtype)
    if kind == "wedges":
        if rng.random() < 0.5:
            level = rng.randint(4, 7)
            most = min(1024, 1024 * 4 ** (7 - level) // (2 if dtype == "float64" else 1))
            return dict(kind=kind, mesh="sphere", level=level, count=_log_int(rng, 2, most), dtype=dtype)
        return dict(kind=kind, mesh="grid", nx=rng.randint(33, 257), ny=rng.randint(33, 257),
                    count=_log_int(rng, 2, 400), dtype=dtype)
    if kind == "dual":
        return dict(kind=kind, nx=_log_int(rng, 17, 230), ny=_log_int(rng, 17, 230))
    if kind == "solve":
        mesh = rng.choice(["sphere", "grid"])
        precision = rng.choice([0, 1])
        plain = rng.random() < 0.5
        d = dict(kind=kind, mesh=mesh, nrhs=_log_int(rng, 1, 40), precision=precision, pre=3 if plain else 0,
                 post=3 if plain else 2, ratio=4.0 if plain else 3.0, inner=1 if plain else 3,
                 coarse_max=rng.choice([0, 170]), rtol=rng.choice([1e-8, 1e-10]))
        if mesh == "sphere":
            d.update(level=rng.randint(4, 7))
        else:
            d.update(nx=rng.randint(4, 9), ny=rng.randint(4, 9), level=rng.randint(3, 6))
        return d
    if kind == "cycles":
        return dict(kind=kind, mesh="sphere", level=rng.randint(4, 7), nrhs=_log_int(rng, 1, 8), steps=rng.randint(1, 4),
                    mu=rng.choice([1, 1, 2]), cycles=rng.randint(1, 8))
    if kind == "inverse":
        return dict(kind=kind, nx=rng.randint(3, 11), ny=rng.randint(3, 11), levels=rng.randint(2, 5),
                    steps=rng.randint(2, 4), cycles=rng.randint(2, 5))
    if kind == "batch":
        small = rng.randint(0, 2)
        return dict(kind=kind, solves=_log_int(rng, 24, 500), small=small, large=rng.randint(max(1, small), 3),
                    draw=rng.randint(0, 999), rtol=1e-8)
    if kind == "learned":
        return dict(kind=kind, level=rng.randint(5, 7), nrhs=_log_int(rng, 4, 32), sweeps=rng.choice([1, 2]),
                    inner=rng.choice([1, 2]), rtol=1e-8)
    return dict(kind=kind, level=rng.choice([5, 6, 7]), fields=rng.randint(1, 4), batch=rng.choice([16384, 40000, 65536]),
                steps=rng.randint(4, 12))


# ---- meshes -------------------------------------------------------------------------------------

def _glue(points, tris, radial):
    """A delta set from triangles of increasing vertices: edges numbered as triangles first use them,
    (v0, v1), (v1, v2), (v0, v2); triangles oriented by their normal (outward, or up)."""
    t = np.asarray(tris, np.int64)
    pairs = np.stack([t[:, [0, 1]], t[:, [1, 2]], t[:, [0, 2]]], 1).reshape(-1, 2)
    key = pairs[:, 0] * len(points) + pairs[:, 1]
    _, first, inv = np.unique(key, return_index=True, return_inverse=True)
    order = np.argsort(first, kind="stable")
    rank = np.empty_like(order)
    rank[order] = np.arange(len(order))
    e = rank[inv.reshape(-1)].reshape(-1, 3)
    src = pairs[first[order]]
    m = SimpleNamespace(points=np.asarray(points, np.float64), ev0=src[:, 1].astype(np.int32),
                        ev1=src[:, 0].astype(np.int32), te0=e[:, 1].astype(np.int32), te1=e[:, 2].astype(np.int32),
                        te2=e[:, 0].astype(np.int32))
    return _orient(m, radial)


def _orient(m, radial):
    v = _corners(m)
    p = m.points
    nrm = np.cross(p[v[1]] - p[v[0]], p[v[2]] - p[v[0]])
    up = np.einsum("ij,ij->i", nrm, p[v[0]]) if radial else nrm[:, 2]
    m.tri_orientation = (up > 0).astype(np.int8)
    m.edge_orientation = np.zeros(len(m.ev0), np.int8)
    return m


def _corners(m):
    return m.ev1[m.te1], m.ev0[m.te2], m.ev0[m.te1]


@functools.lru_cache(maxsize=8)
def _grid(nx, ny):
    y, x = np.divmod(np.arange(nx * ny), nx)
    pts = np.stack([x + 0.5 * (y % 2), y.astype(float), np.zeros(nx * ny)], 1)
    r, c = np.divmod(np.arange((nx - 1) * (ny - 1)), nx - 1)
    i = c + nx * r
    even = np.stack([np.stack([i, i + 1, i + nx], 1), np.stack([i + 1, i + nx, i + nx + 1], 1)], 1)
    odd = np.stack([np.stack([i, i + nx, i + nx + 1], 1), np.stack([i, i + 1, i + nx + 1], 1)], 1)
    return _glue(pts, np.where((r % 2 == 0)[:, None, None], even, odd).reshape(-1, 3), False)


def _icosahedron():
    g = (1 + 5 ** 0.5) / 2
    p = np.array([[s * a, t * b * g, 0] for a in (1,) for b in (1,) for s in (-1, 1) for t in (-1, 1)], float)
    p = np.concatenate([p, p[:, [2, 0, 1]], p[:, [1, 2, 0]]])
    d = np.linalg.norm(p[:, None] - p[None], axis=2)
    near = (d > 0) & (d < 2.1)
    f = [(a, b, c) for a in range(12) for b in range(a + 1, 12) for c in range(b + 1, 12)
         if near[a, b] and near[b, c] and near[a, c]]
    return _glue(p / np.linalg.norm(p[0]), f, True)


def _refine(m, radial):
    """Binary subdivision: vertex nv + e is edge e's midpoint (on the unit sphere when radial)."""
    nv, ne, nt = len(m.points), len(m.ev0), len(m.te0)
    ev0, ev1 = np.empty(2 * ne + 3 * nt, np.int32), np.empty(2 * ne + 3 * nt, np.int32)
    ev0[:2 * ne:2] = ev0[1:2 * ne:2] = nv + np.arange(ne)
    ev1[:2 * ne:2], ev1[1:2 * ne:2] = m.ev0, m.ev1
    a, b, c = (x.astype(np.int64) for x in (m.te0, m.te1, m.te2))
    inner = 2 * ne + 3 * np.arange(nt)
    for k, (s, t) in enumerate(((a, b), (b, c), (a, c))):
        ev1[inner + k], ev0[inner + k] = nv + s, nv + t
    te = np.empty((nt, 4, 3), np.int64)
    te[:, 0] = np.stack([inner + 1, inner + 2, inner], 1)
    te[:, 1] = np.stack([inner + 1, 2 * c + 1, 2 * b + 1], 1)
    te[:, 2] = np.stack([inner + 2, 2 * c, 2 * a + 1], 1)
    te[:, 3] = np.stack([inner, 2 * b, 2 * a], 1)
    te = te.reshape(-1, 3).astype(np.int32)
    mid = (m.points[m.ev0] + m.points[m.ev1]) / 2
    if radial:
        mid /= np.linalg.norm(mid, axis=1, keepdims=True)
    f = SimpleNamespace(points=np.concatenate([m.points, mid]), ev0=ev0, ev1=ev1, te0=te[:, 0].copy(),
                        te1=te[:, 1].copy(), te2=te[:, 2].copy())
    return _orient(f, radial)


@functools.lru_cache(maxsize=6)
def _sphere(level):
    return _icosahedron() if level == 0 else _refine(_sphere(level - 1), True)


def _coarse(case):
    """The coarsest mesh of a hierarchy and its radius."""
    if case.get("mesh") == "sphere":
        return _icosahedron(), 1.0
    return _grid(case["nx"], case["ny"]), 0.0


def _mesh(case):
    return _grid(case["nx"], case["ny"]) if case.get("mesh", "grid") == "grid" else _sphere(case["level"])


def _center(case):
    return "barycenter" if case.get("mesh", "grid") == "grid" else "circumcenter"


def _dev_mesh(case):
    m = _mesh(case)
    return _dec().Mesh(m.points, m.ev0, m.ev1, m.te0, m.te1, m.te2, m.edge_orientation, m.tri_orientation,
                       center=_center(case))


def _uniform(seed, dtype, *shapes):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    return [torch.rand(s, dtype=dtype, device="cuda", generator=gen).mul_(2).sub_(1) for s in shapes]


# ---- inputs and plans ---------------------------------------------------------------------------

# the batch's meshes, by the size step of both families: icosphere L4-L7, grid 65^2-513^2
def _batch_groups(case):
    types = [("sphere", k + 4) for k in range(case["small"], case["large"] + 1)]
    types += [("grid", k + 3) for k in range(case["small"], case["large"] + 1)]
    counts = np.bincount(np.random.default_rng(case["draw"]).integers(0, len(types), case["solves"]),
                         minlength=len(types))
    return [(mesh, level, int(c)) for (mesh, level), c in zip(types, counts) if c > 0]


def _batch_coarse(mesh):
    return (_icosahedron(), 1.0) if mesh == "sphere" else (_grid(9, 9), 0.0)


def _vertices(coarse, levels):
    """Vertices after `levels` binary subdivisions."""
    nv, ne, nt = len(coarse.points), len(coarse.ev0), len(coarse.te0)
    for _ in range(levels):
        nv, ne, nt = nv + ne, 2 * ne + 3 * nt, 4 * nt
    return nv


def _batch_inputs(case, seed):
    rng = np.random.default_rng(seed)
    out = []
    for q, (mesh, level, count) in enumerate(_batch_groups(case)):
        n = _vertices(_batch_coarse(mesh)[0], level)
        shift = np.exp(rng.uniform(math.log(0.1), math.log(10.0), count))
        out.append((shift, _uniform(seed * 64 + q, torch.float64, (count, n))[0]))
    return out


def _network():
    """Weights of a damped-Jacobi step (y = 0.7 f0) with small random units beside it."""
    g = np.random.default_rng(4)
    w1 = g.uniform(-0.27, 0.27, (64, 16))
    w2 = g.uniform(-0.21, 0.21, (64, 64))
    w3 = g.uniform(-2e-3, 2e-3, 64)
    w1[:2] = 0
    w1[0, 0], w1[1, 0] = 1, -1
    w2[:2] = 0
    w2[0, 0] = w2[1, 1] = 1
    w3[:2] = 0.7, -0.7
    return np.concatenate([w1.ravel(), np.zeros(64), w2.ravel(), np.zeros(64), w3, np.zeros(1)]).astype(np.float32)


def _hierarchy(case, coarse, radius, **opts):
    return _dec().MultigridData(coarse, case["level"], center="circumcenter", project_radius=radius, **opts)


def prepare(case, seed):
    dec, kind = _dec(), case["kind"]
    s = SimpleNamespace(kind=kind, case=case)
    if kind == "operators":
        g, dt = _dev_mesh(case), case["dtype"]
        s.w01, s.w11, s.w02 = (dec.dec_wedge_product(i, j, g, dt) for i, j in ((0, 1), (1, 1), (0, 2)))
        s.d0, s.d1, s.dd1 = dec.dec_differential(0, g, dt), dec.dec_differential(1, g, dt), dec.dec_dual_derivative(1, g, dt)
        s.star1, s.lap = dec.hodge_operator(1, g, dtype=dt), dec.laplace_beltrami(g, dt)
        s.f, s.a, s.b = _uniform(seed, getattr(torch, dt), g.nv, g.ne, g.ne)
    elif kind == "wedges":
        g, dt = _dev_mesh(case), case["dtype"]
        s.w11 = dec.dec_wedge_product(1, 1, g, dt)
        s.a, s.b = _uniform(seed, getattr(torch, dt), (case["count"], g.ne), (case["count"], g.ne))
        s.out = torch.empty((case["count"], g.nt), dtype=getattr(torch, dt), device="cuda")
    elif kind == "dual":
        g = _dev_mesh(case)
        s.lie, s.lap, s.w11 = dec.lie_derivative_dd(1, 1, g), dec.dual_laplacian(1, g), dec.dec_wedge_product_pd(1, 1, g)
        s.f, s.g = _uniform(seed, torch.float64, g.ne, g.ne)
    elif kind in ("solve", "learned"):
        if kind == "solve":
            coarse, radius = _coarse(case)
            s.mg = _hierarchy(case, coarse, radius, shift=1.0, smoother=1, precision=case["precision"], pre=case["pre"],
                              post=case["post"], cheb_ratio=case["ratio"], inner_cycles=case["inner"],
                              coarse_max=case["coarse_max"])
        else:
            s.mg = _hierarchy(case, _icosahedron(), 1.0, shift=1.0, smoother=3, precision=1, pre=case["sweeps"],
                              post=case["sweeps"], cheb_ratio=3.0, inner_cycles=case["inner"], coarse_max=170)
            s.mlp = dec.SmootherMLP(4)
            s.mlp.params = _network()
            s.mg.set_smoother_mlp(s.mlp)
        s.b, = _uniform(seed, torch.float64, (case["nrhs"], s.mg.n))
        s.u = torch.zeros_like(s.b)
    elif kind == "cycles":
        s.mg = _hierarchy(case, _icosahedron(), 1.0, shift=1.0, smoother=2, pre=case["steps"], post=case["steps"],
                          mu=case["mu"])
        s.b, = _uniform(seed, torch.float64, (case["nrhs"], s.mg.n))
        s.u = torch.zeros_like(s.b)
    elif kind == "inverse":
        s.inv = dec.dec_inverse_laplacian(0, _grid(case["nx"], case["ny"]), case["levels"], steps=case["steps"],
                                          cycles=case["cycles"])
        # a solvable right-hand side, L x
        s.b = s.inv.md.level_op(0) @ _uniform(seed, torch.float64, s.inv.md.n)[0]
    elif kind == "batch":
        s.mgs, s.shifts, s.bs = [], [], []
        for (mesh, level, _), (shift, b) in zip(_batch_groups(case), _batch_inputs(case, seed)):
            coarse, radius = _batch_coarse(mesh)
            s.mgs.append(_hierarchy(dict(level=level), coarse, radius, shift=0.0, smoother=1, precision=1, pre=0,
                                    post=2, cheb_ratio=3.0, coarse_solver=2, coarse_max=170, inner_cycles=3))
            s.shifts.append(shift)
            s.bs.append(b)
        s.us = [torch.zeros_like(b) for b in s.bs]
        s.batch = dec.Batch(s.mgs)
    else:
        s.mg = _hierarchy(case, _icosahedron(), 1.0, shift=1.0, smoother=1, precision=0)
        s.op = s.mg.level_op(0)
        u, = _uniform(seed, torch.float64, (case["fields"], s.mg.n))
        s.r = torch.stack([-(s.op @ x) for x in u])   # residuals of A u = 0 from rough iterates
        s.mlp = dec.SmootherMLP(4)
    return s


def run(s):
    if s.kind == "operators":
        d1a, d0f = s.d1 @ s.a, s.d0 @ s.f
        return dict(w01=s.w01(s.f, s.a), w11=s.w11(s.a, s.b), d1a=d1a, w02=s.w02(s.f, d1a), d0f=d0f,
                    div=s.dd1 @ (s.star1 @ d0f), lap=s.lap @ s.f)
    if s.kind == "wedges":
        return s.w11.batched(s.a, s.b, s.out)
    if s.kind == "dual":
        return dict(lie=s.lie(s.f, s.g), lap=s.lap(s.f), w11=s.w11(s.f, s.g))
    if s.kind in ("solve", "learned"):
        return s.mg.solve(s.u, s.b, rtol=s.case["rtol"], max_iters=60, use_initial_guess=False)[0]
    if s.kind == "cycles":
        dec = _dec()
        return (dec.multigrid_vcycles if s.case["mu"] == 1 else dec.multigrid_wcycles)(s.u, s.b, s.mg, s.case["cycles"])
    if s.kind == "inverse":
        u = s.inv(s.b)
        return u - u.mean()   # the solution is defined up to a constant
    if s.kind == "batch":
        for u in s.us:
            u.zero_()
        s.batch.solve(s.us, s.bs, shifts=s.shifts, rtol=s.case["rtol"], max_iters=60)
        return s.us
    s.mlp.train(s.op, s.r, s.case["steps"], batch=s.case["batch"])
    loss, grad = s.mlp.loss_grad(s.op, s.r)
    return dict(params=s.mlp.params, loss=loss, grad=grad)


# ---- work ---------------------------------------------------------------------------------------

def _sizes(case):
    if case.get("mesh", "grid") == "grid" and "level" not in case:
        nx, ny = case["nx"], case["ny"]
        return nx * ny, nx * (ny - 1) + (nx - 1) * ny + (nx - 1) * (ny - 1), 2 * (nx - 1) * (ny - 1)
    nt = 20 * 4 ** case["level"]
    return nt // 2 + 2, nt * 3 // 2, nt


def work(case):
    kind = case["kind"]
    if kind in ("operators", "wedges", "dual"):
        nv, ne, nt = _sizes(case)
        z = 4 if case.get("dtype") == "float32" else 8
        if kind == "operators":
            by = ne * (8 + 2 * z) + nv * z                      # ∧01
            by += nt * (12 + 4 * z) + 2 * ne * z                # ∧11
            by += nt * (13 + z) + ne * z                        # d1
            by += nt * (12 + 5 * z) + nv * z                    # ∧02
            by += ne * (9 + z) + nv * z                         # d0
            by += 3 * ne * z + ne * z + 2 * ne * 4 + nv * z     # ⋆1, then the signed vertex rows
            by += nv * 7 * (4 + z) + 2 * nv * z                 # Laplacian
            return dict(bytes=by, flops=4 * ne + 15 * nt + 13 * nv)
        if kind == "wedges":
            return dict(bytes=case["count"] * (2 * ne + nt) * z + nt * (12 + 3 * z), flops=case["count"] * nt * 14)
        # two solves with ⋆1 (about 30 steps of two products each) and the operators around them
        return dict(bytes=ne * (2 * 30 * 2 * (6 * 12 + 5 * 8) + 300), flops=2 * 30 * 2 * ne * 30)
    if kind in ("solve", "learned", "cycles"):
        n = _vertices(_coarse(case)[0] if kind == "solve" else _icosahedron(), case["level"])
        if kind == "cycles":
            k = case["cycles"] * 2 * case["steps"] * (4 / 3 if case["mu"] == 1 else 2)
            return dict(bytes=k * n * (6 * 12 + 8 + 6 * 8 * case["nrhs"]), flops=k * n * case["nrhs"] * 24)
        if kind == "solve":
            z = 4 if case["precision"] else 8
            cycles = -math.log10(case["rtol"]) * 1.1
            sweeps = case["pre"] + case["post"]
        else:
            z, sweeps = 4, 2 * case["sweeps"]
            cycles = 9
        k = cycles * 4 / 3
        by = k * n * ((sweeps + 1) * (6 * (4 + z) + z) + (3 * sweeps + 3) * z * case["nrhs"]) + 16 * n * case["nrhs"]
        fl = k * n * case["nrhs"] * (10368 * sweeps if kind == "learned" else 16 * (sweeps + 1))
        return dict(bytes=by, flops=fl)
    if kind == "inverse":
        n = _vertices(_grid(case["nx"], case["ny"]), case["levels"])
        k = case["cycles"] * 2 * case["steps"] * 2 * 4 / 3
        return dict(bytes=k * n * (6 * 12 + 8 + 6 * 8), flops=k * n * 24)
    if kind == "batch":
        by = sum(10 * 4 / 3 * _vertices(_batch_coarse(m)[0], lv) * (3 * 52 + 9 * 4 * c) for m, lv, c in _batch_groups(case))
        return dict(bytes=by, flops=by / 2)
    n = case["fields"] * _sizes(dict(mesh="sphere", level=case["level"]))[0]
    b = min(n, case["batch"])
    return dict(bytes=case["steps"] * (n * 200 + b * 100), flops=(case["steps"] + 1) * (n * 10240 + b * 30720))


# ---- expected values, in 64 bits ----------------------------------------------------------------

class _Geo:
    """The dual complex of a mesh in float64 on the GPU: diagonal stars, wedge weights, signs."""

    def __init__(self, m, center):
        def ix(a):
            return torch.as_tensor(np.asarray(a, np.int64), device="cuda")
        self.v0, self.v1 = ix(m.ev0), ix(m.ev1)                 # target, source
        self.e = [ix(m.te0), ix(m.te1), ix(m.te2)]
        self.v = [ix(x) for x in _corners(m)]
        self.nv, self.ne, self.nt = len(m.points), len(m.ev0), len(m.te0)
        p = torch.as_tensor(m.points, device="cuda")
        self.es = torch.as_tensor(m.edge_orientation, device="cuda").double() * 2 - 1
        self.ts = torch.as_tensor(m.tri_orientation, device="cuda").double() * 2 - 1
        q = [p[x] for x in self.v]
        cr = torch.linalg.cross(q[1] - q[0], q[2] - q[0])
        self.area = cr.norm(dim=1) / 2
        if center == "barycenter":
            c = (q[0] + q[1] + q[2]) / 3
        else:
            l = [((q[1] - q[2]) ** 2).sum(1), ((q[0] - q[2]) ** 2).sum(1), ((q[0] - q[1]) ** 2).sum(1)]
            w = [l[k] * (l[(k + 1) % 3] + l[(k + 2) % 3] - l[k]) for k in range(3)]
            c = sum(w[k][:, None] * q[k] for k in range(3)) / (w[0] + w[1] + w[2])[:, None]
        mid = (p[self.v0] + p[self.v1]) / 2
        dl = [(c - mid[e]).norm(dim=1) for e in self.e]
        length = (p[self.v0] - p[self.v1]).norm(dim=1)
        self.star1 = self._add(self.ne, self.e, dl) / length
        # dual area of each corner: the two elementary triangles (corner, edge midpoint, center)
        self.da = []
        for k in range(3):
            a = 0
            for j in range(3):
                if j != k:
                    a = a + torch.linalg.cross(mid[self.e[j]] - q[k], c - q[k]).norm(dim=1) / 2
            self.da.append(a)
        self.star0 = self._add(self.nv, self.v, self.da)
        self.p, self.c, self.mid = p, c, mid

    @staticmethod
    def _add(n, idx, val):
        out = torch.zeros(n, dtype=torch.float64, device="cuda")
        for i, v in zip(idx, val):
            out.index_add_(0, i, v)
        return out

    def d0(self, f):
        return self.es * (f[self.v0] - f[self.v1])

    def d1(self, a):
        x = [self.es[e] * a[e] for e in self.e]
        return self.ts * (x[0] - x[1] + x[2])

    def dd1(self, a):     # -d0ᵀ
        x = self.es * a
        return -(self._add(self.nv, [self.v0], [x]) - self._add(self.nv, [self.v1], [x]))

    def dd0(self, t):     # d1ᵀ
        x = self.ts * t
        return self._add(self.ne, self.e, [self.es[self.e[0]] * x, -self.es[self.e[1]] * x, self.es[self.e[2]] * x])

    def w11(self, a, b):
        ae, be, s = ([x[..., e] for e in self.e] for x in (a, b, self.es))
        h = self.ts * 2 * self.area
        return (s[1] * s[2] * self.da[0] / h * (ae[2] * be[1] - ae[1] * be[2]) +
                s[0] * s[2] * self.da[1] / h * (ae[2] * be[0] - ae[0] * be[2]) +
                s[0] * s[1] * self.da[2] / h * (ae[1] * be[0] - ae[0] * be[1]))

    def geometric_star1(self):
        """The sparse ⋆1 of FastDEC, dense."""
        ed = [self.e[2], self.e[1], self.e[0]]
        ev = [self.p[self.v0[e]] - self.p[self.v1[e]] for e in ed]
        dv = [self.c - self.mid[e] for e in ed]
        dv[1] = -dv[1]

        def sgn(z):
            return torch.where(z == 0, torch.ones_like(z), z.sign())

        def crossdot(a, b):
            x = torch.linalg.cross(a, b)
            return x.norm(dim=1) * sgn(x[:, 2])
        rel = sgn(torch.linalg.cross(ev[0], dv[0])[:, 2])
        g = torch.zeros(self.ne * self.ne, dtype=torch.float64, device="cuda")
        for i in range(3):
            g.index_add_(0, ed[i] * self.ne + ed[i], rel * crossdot(ev[i], dv[i]) / (ev[i] ** 2).sum(1))
            for j in range(3):
                if j != i:
                    k = 3 - i - j
                    val = (ev[i] * dv[i]).sum(1) / (ev[i] ** 2).sum(1) * (ev[i] * ev[k]).sum(1)
                    g.index_add_(0, ed[i] * self.ne + ed[j], rel * val / crossdot(ev[j], ev[k]))
        return g.view(self.ne, self.ne)


def _exact_solve(coarse, radial, levels, shift, b):
    """(⋆0⁻¹ d0ᵀ ⋆1 d0 + c_j) u_j = b_j in float64: conjugate gradients on the ⋆0-weighted operator,
    preconditioned by V-cycles over the subdivisions (damped Jacobi; R = Pᵀ)."""
    ms = [coarse]
    for _ in range(levels):
        ms.append(_refine(ms[-1], radial))
    c = torch.as_tensor(shift, dtype=torch.float64, device="cuda").expand(b.shape[0])
    lv = []
    for m in ms:
        g = _Geo(m, "circumcenter")
        deg = g._add(g.nv, [g.v0, g.v1], [g.star1, g.star1])
        lv.append((g.v0, g.v1, g.star1[:, None], g.star0[:, None], 1 / (deg[:, None] + g.star0[:, None] * c), len(m.points)))

    def apply(k, x):
        v0, v1, w, m0, _, _ = lv[k]
        y = m0 * c * x
        d = w * (x[v0] - x[v1])
        return y.index_add_(0, v0, d).index_add_(0, v1, d, alpha=-1)

    def cycle(k, r):
        dinv = lv[k][4]
        x = 0.7 * dinv * r
        if k == 0:
            for _ in range(60):
                x = x + 0.7 * dinv * (r - apply(k, x))
            return x
        x = x + 0.7 * dinv * (r - apply(k, x))
        q = r - apply(k, x)
        v0, v1, nc = lv[k - 1][0], lv[k - 1][1], lv[k - 1][5]
        rc = q[:nc] + 0
        rc.index_add_(0, v0, q[nc:], alpha=0.5).index_add_(0, v1, q[nc:], alpha=0.5)
        z = cycle(k - 1, rc)
        x[:nc] += z
        x[nc:] += (z[v0] + z[v1]) / 2
        for _ in range(2):
            x = x + 0.7 * dinv * (r - apply(k, x))
        return x
    top = len(lv) - 1
    rhs = (lv[top][3] * b.t()).contiguous()
    x = torch.zeros_like(rhs)
    r, p, rz = rhs.clone(), None, None
    for _ in range(60):
        z = cycle(top, r)
        new = (r * z).sum(0)
        p = z if p is None else z + new / rz * p
        rz = new
        q = apply(top, p)
        a = rz / (p * q).sum(0)
        x += a * p
        r -= a * q
        if float((r.norm(dim=0) / rhs.norm(dim=0)).max()) < 3e-15:
            break
    return x.t().contiguous()


def exact(case, seed):
    kind = case["kind"]
    if kind == "operators":
        g = _Geo(_mesh(case), _center(case))
        f, a, b = (x.double() for x in _uniform(seed, getattr(torch, case["dtype"]), g.nv, g.ne, g.ne))
        d1a, d0f = g.d1(a), g.d0(f)
        w02 = d1a * sum(g.da[k] / g.area * f[g.v[k]] for k in range(3))
        return dict(w01=0.5 * a * (f[g.v0] + f[g.v1]), w11=g.w11(a, b), d1a=d1a, w02=w02, d0f=d0f,
                    div=g.dd1(g.star1 * d0f), lap=-g.dd1(g.star1 * d0f) / g.star0)
    if kind == "wedges":
        g = _Geo(_mesh(case), _center(case))
        a, b = _uniform(seed, getattr(torch, case["dtype"]), (case["count"], g.ne), (case["count"], g.ne))
        out = torch.empty((case["count"], g.nt), dtype=torch.float64, device="cuda")
        for j in range(0, case["count"], 64):
            out[j:j + 64] = g.w11(a[j:j + 64].double(), b[j:j + 64].double())
        return out
    if kind == "dual":
        g = _Geo(_mesh(case), _center(case))
        if g.ne > 30000:
            return None
        f, _ = _uniform(seed, torch.float64, g.ne, g.ne)
        st = g.geometric_star1()
        inv = torch.linalg.solve(-st, f)
        return dict(lie=None, lap=st @ g.d0(g.dd1(f) / g.star0) + g.dd0(g.d1(inv) / g.area), w11=None)
    if kind in ("solve", "learned"):
        coarse, radius = _coarse(case) if kind == "solve" else (_icosahedron(), 1.0)
        b, = _uniform(seed, torch.float64, (case["nrhs"], _vertices(coarse, case["level"])))
        return _exact_solve(coarse, radius > 0, case["level"], 1.0, b)
    if kind == "batch":
        out = []
        for (mesh, level, _), (shift, b) in zip(_batch_groups(case), _batch_inputs(case, seed)):
            coarse, radius = _batch_coarse(mesh)
            out.append(_exact_solve(coarse, radius > 0, level, shift, b))
        return out
    return None   # a fixed number of cycles or of training steps: no value of its own
