"""Workloads that a user of lpmcxx_b200 runs through its public entry points, for timing.

A case is a dict of plain values; `prepare` makes what the user's program holds before the call (device particles,
host meshes, solvers), `run` makes one call, `work` counts the bytes and operations it cannot do without and
`exact` gives the 64-bit answer from plain torch where that takes seconds.

Particles of a "mesh" case are the centroids (sources) and vertices (targets only) of a refined icosahedron or
cube on the unit sphere, as the package's own configurations; those of a case with "n_src" are a seeded
selection of a rotated Fibonacci lattice, for sizes that no mesh has.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import lpmcxx_b200 as L
from lpmcxx_b200.learned import load as load_selector

DT = 0.005                # time step of the package's RK4 workloads
LEARNED_EPS = 5e-7        # per-pair budget, order bias and acceptance parameter of the learned workloads
LEARNED_BIAS = 2
LEARNED_THETA = 0.55
PAIRS_EXACT = 4e11        # most pairwise terms that exact() sums (about 20 s)


# ------------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # one velocity evaluation of the smallest mesh in use (icosahedron refined 3 times), double precision:
        # a latency-bound call
        {"name": "direct_f64_mesh3", "kind": "direct", "precision": "f64", "mesh": "icos", "level": 3, "delta": 0.0},
        # the same on an ordinary mesh (82k faces): the parity path of DirectSum
        {"name": "direct_f64_mesh6", "kind": "direct", "precision": "f64", "mesh": "icos", "level": 6, "delta": 0.0},
        # single-precision pair arithmetic on an ordinary cubed sphere, and on a large icosahedral mesh
        {"name": "direct_f32_cube6", "kind": "direct", "precision": "f32", "mesh": "cube", "level": 6, "delta": 0.0},
        {"name": "direct_f32_mesh7", "kind": "direct", "precision": "f32", "mesh": "icos", "level": 7, "delta": 0.0},
        # meshfree 1/(4 pi r) potential of an odd number of charges
        {"name": "poisson_direct_f64", "kind": "poisson_direct", "precision": "f64", "n": 20011},
        # DirectSum::meshSolve from host arrays with a scalar kernel (stream function from vorticity)
        {"name": "greens_host_mesh5", "kind": "greens_host", "mesh": "icos", "level": 5},
        # a time step of the reference's own size of run: RK4 on 7,682 particles, double-precision direct sums
        {"name": "rk4_direct_f64_mesh4", "kind": "rk4_direct", "precision": "f64", "mesh": "icos", "level": 4},
        # TreeSum with the package's default solver (order 8, theta 0.7, 512 per leaf) on an ordinary mesh
        {"name": "tree_fixed_mesh6", "kind": "tree", "precision": "f32", "order": 8, "theta": 0.7, "leaf": 512,
         "mesh": "icos", "level": 6},
        # the headline: an RK4 step of 1,966,082 particles with the learned treecode
        {"name": "rk4_learned_mesh8", "kind": "rk4_learned", "leaf": 512, "mesh": "icos", "level": 8},
        # the 3D Poisson treecode workload, and a small call of the same solver
        {"name": "poisson_tree_1m", "kind": "poisson_tree", "precision": "f32", "order": 6, "theta": 0.6, "leaf": 256,
         "n": 1048576},
        {"name": "poisson_tree_50k", "kind": "poisson_tree", "precision": "f32", "order": 6, "theta": 0.6, "leaf": 256,
         "n": 50021},
        # an ensemble step: four vortices on each of three mesh sizes, advanced together
        {"name": "ensemble_mesh567", "kind": "ensemble", "leaf": 512, "levels": "5,6,7", "per_level": 4},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["direct", "direct", "poisson_direct", "greens_host", "rk4_direct", "tree", "tree",
                       "rk4_learned", "poisson_tree", "ensemble"])
    if kind == "direct":
        precision = rng.choice(["f64", "f32"])
        n = _log_int(rng, 640, 330_000 if precision == "f32" else 90_000)
        return {"kind": kind, "precision": precision, "n_src": n, "n_vert": rng.randrange(n // 2, n + 1),
                "delta": rng.choice([0.0, 0.0, 0.05])}
    if kind == "poisson_direct":
        return {"kind": kind, "precision": rng.choice(["f64", "f32"]), "n": _log_int(rng, 1000, 120_000)}
    if kind == "greens_host":
        return {"kind": kind, "mesh": rng.choice(["icos", "cube"]), "level": rng.choice([3, 4, 5]),
                "shift": rng.randrange(1, 1000)}
    if kind == "rk4_direct":
        n = _log_int(rng, 640, 40_000)
        return {"kind": kind, "precision": rng.choice(["f64", "f32"]), "n_src": n, "n_vert": n // 2 + 2}
    if kind == "tree":
        n = _log_int(rng, 10_000, 700_000)
        return {"kind": kind, "precision": rng.choice(["f32", "f32", "f64"]), "order": rng.randrange(4, 11),
                "theta": rng.choice([0.5, 0.6, 0.7]), "leaf": rng.choice([256, 512]), "n_src": n, "n_vert": n // 2 + 2}
    if kind == "rk4_learned":
        n = _log_int(rng, 10_000, 1_000_000)
        return {"kind": kind, "leaf": rng.choice([256, 512]), "n_src": n, "n_vert": n // 2 + 2}
    if kind == "poisson_tree":
        return {"kind": kind, "precision": "f32", "order": rng.randrange(3, 9), "theta": rng.choice([0.5, 0.6, 0.7]),
                "leaf": rng.choice([128, 256]), "n": _log_int(rng, 10_000, 1_000_000)}
    sizes = [_log_int(rng, 10_000, 300_000) for _ in range(rng.randrange(2, 7))]
    return {"kind": kind, "leaf": 512, "sizes": ",".join(str(n) for n in sizes)}


# ------------------------------------------------------------------------------------------------ inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 17)


def _unit(v):
    return v / v.norm(dim=-1, keepdim=True)


def _rotation(seed):
    q, _ = np.linalg.qr(np.random.default_rng(int(seed) + 5).normal(size=(3, 3)))
    return torch.tensor(q, device="cuda")


def _icos_faces():
    g = (1.0 + 5.0 ** 0.5) / 2.0
    v = np.array([(s * a, t * b, 0.0) for s in (-1, 1) for t in (-1, 1) for a, b in ((1.0, g),)])
    v = np.concatenate([v, np.roll(v, 1, axis=1), np.roll(v, 2, axis=1)])
    tri = [(i, j, k) for i in range(12) for j in range(i) for k in range(j)
           if all(abs(np.linalg.norm(v[p] - v[q]) - 2.0) < 1e-9 for p, q in ((i, j), (j, k), (i, k)))]
    return _unit(torch.tensor(v[np.array(tri)], device="cuda"))          # (20, 3, 3)


def _cube_faces():
    out = []
    for a in range(3):
        for s in (-1.0, 1.0):
            quad = np.zeros((4, 3))
            quad[:, a] = s
            quad[:, (a + 1) % 3] = (-1.0, 1.0, 1.0, -1.0)
            quad[:, (a + 2) % 3] = (-1.0, -1.0, 1.0, 1.0)
            out.append(quad)
    return _unit(torch.tensor(np.array(out), device="cuda"))            # (6, 4, 3)


def _refine(f):
    m = [_unit(f[:, i] + f[:, (i + 1) % f.shape[1]]) for i in range(f.shape[1])]
    if f.shape[1] == 3:
        kids = [(f[:, 0], m[0], m[2]), (m[0], f[:, 1], m[1]), (m[2], m[1], f[:, 2]), (m[0], m[1], m[2])]
    else:
        c = _unit(f.sum(dim=1))
        kids = [(f[:, 0], m[0], c, m[3]), (m[0], f[:, 1], m[1], c), (c, m[1], f[:, 2], m[2]), (m[3], c, m[2], f[:, 3])]
    return torch.stack([torch.stack(k, dim=1) for k in kids], dim=1).reshape(-1, f.shape[1], 3)


def _mesh(kind, level, seed):
    """Centroids and areas of the faces of every level (coarse first) with the divided mask, and the vertices."""
    f = _icos_faces() if kind == "icos" else _cube_faces()
    cen, area, div = [], [], []
    for lev in range(level + 1):
        cen.append(_unit(f.sum(dim=1)))
        half = f[:, 2:] - f[:, :1]
        a = torch.linalg.cross(f[:, 1] - f[:, 0], half[:, 0]).norm(dim=1)
        if f.shape[1] == 4:
            a = a + torch.linalg.cross(half[:, 0], half[:, 1]).norm(dim=1)
        area.append(a * (4.0 * math.pi / a.sum()) if lev == level else torch.zeros_like(a))
        div.append(torch.full((f.shape[0],), lev < level, device="cuda"))
        if lev < level:
            f = _refine(f)
    corners = f.reshape(-1, 3)
    key = (corners * 2.0 ** 30).round().to(torch.int64)                 # equal corners, from either side of an edge
    key = (key[:, 0] * 0x9E3779B1 + key[:, 1]) * 0x85EBCA77 + key[:, 2]
    _, first = torch.sort(key, stable=True)
    k = key[first]
    keep = torch.ones_like(k, dtype=torch.bool)
    keep[1:] = k[1:] != k[:-1]
    vert = corners[first[keep].sort().values]
    rot = _rotation(seed)
    return torch.cat(cen) @ rot, torch.cat(area), torch.cat(div), vert @ rot


def _vorticity(x, seed):
    """A Rossby-Haurwitz wave (wave number 4) and a Gaussian vortex of seeded centre and strength."""
    r = np.random.default_rng(int(seed) + 11)
    c = r.normal(size=3)
    c = torch.tensor(c / np.linalg.norm(c), device="cuda")
    z = x[:, 2]
    rh = 2.0 * z - 30.0 * torch.cos(4.0 * torch.atan2(x[:, 1], x[:, 0])) * z * (z * z - 1.0) ** 2
    return rh + float(r.uniform(0.5, 2.0)) * 4.0 * math.pi * torch.exp(-16.0 * ((x - c) ** 2).sum(dim=1))


def _particles(case, seed):
    """(n, 4) particles (sources first; the others have strength 0) and the number of sources."""
    if "mesh" in case:
        cen, area, div, vert = _mesh(case["mesh"], case["level"], seed)
        x, area = cen[~div], area[~div]
        pts = torch.cat([x, vert])
    else:
        n = case["n_src"] + case["n_vert"]
        i = torch.arange(n, dtype=torch.float64, device="cuda") + 0.5
        z = 1.0 - 2.0 * i / n
        phi = math.pi * (1.0 + 5.0 ** 0.5) * i
        r = torch.sqrt(1.0 - z * z)
        pts = _unit(torch.stack([r * torch.cos(phi), r * torch.sin(phi), z], dim=1)) @ _rotation(seed)
        pts = pts[torch.randperm(n, generator=_gen(seed), device="cuda")]
        x = pts[: case["n_src"]]
        area = torch.full((x.shape[0],), 4.0 * math.pi / x.shape[0], dtype=torch.float64, device="cuda")
    zeta = _vorticity(x, seed)
    w = (zeta - (zeta * area).sum() / area.sum()) * area
    p = torch.zeros((pts.shape[0], 4), dtype=torch.float64, device="cuda")
    p[:, :3] = pts
    p[: x.shape[0], 3] = w
    return p, x.shape[0]


def _charges(case, seed):
    """(n, 4) points uniform in [-1, 1]^3 with charges uniform in [-1, 1]."""
    return 2.0 * torch.rand((case["n"], 4), dtype=torch.float64, device="cuda", generator=_gen(seed)) - 1.0


def _members(case):
    if "levels" in case:
        return [{"mesh": "icos", "level": int(v)} for v in case["levels"].split(",") for _ in range(case["per_level"])]
    return [{"n_src": int(n), "n_vert": int(n) // 2 + 2} for n in case["sizes"].split(",")]


def _host_mesh(case, seed):
    cen, area, div, vert = _mesh(case["mesh"], case["level"], seed + case.get("shift", 0))
    zeta = _vorticity(cen, seed)
    leaf = ~div
    zeta = zeta - (zeta[leaf] * area[leaf]).sum() / area.sum()
    return cen, area, div, vert, zeta


# ------------------------------------------------------------------------------------------------ the user's program
def _prec(case):
    return L.LPM_PREC_F64 if case.get("precision") == "f64" else L.LPM_PREC_F32


def prepare(case, seed):
    kind, s = case["kind"], {"kind": case["kind"]}
    ctx = L.Context(0)
    if kind == "greens_host":
        cen, area, div, vert, zeta = (t.cpu().numpy() for t in _host_mesh(case, seed))
        s["mesh"] = L.SphereMesh(case["mesh"], case["level"], vert, cen, area, div.astype(np.uint8))
        s["src"], s["ctx"] = zeta, ctx
        return s
    ctx.use_torch_stream()
    if kind in ("direct", "poisson_direct"):
        scalar = kind == "poisson_direct"
        p, n_src = (_charges(case, seed), case["n"]) if scalar else _particles(case, seed)
        s["kernel"] = L.poisson_kernel() if scalar else L.biot_savart_kernel(1.0, case["delta"])
        s["prec"], s["tgt"], s["src"], s["n_coincident"] = _prec(case), p, p[:n_src].clone(), n_src
        s["out"] = torch.empty((1 if scalar else 3, p.shape[0]), dtype=torch.float64, device="cuda")
    elif kind in ("tree", "poisson_tree"):
        scalar = kind == "poisson_tree"
        p, n_src = (_charges(case, seed), case["n"]) if scalar else _particles(case, seed)
        kernel = L.poisson_kernel() if scalar else L.biot_savart_kernel()
        solver = L.tree_solver(_prec(case), case["order"], case["leaf"], case["theta"])
        s["tree"] = L.TreeSum(ctx, kernel, solver, n_src, p.shape[0])
        s["tgt"], s["src"] = p, p[:n_src].clone()
        s["out"] = torch.empty((1 if scalar else 3, p.shape[0]), dtype=torch.float64, device="cuda")
    elif kind in ("rk4_direct", "rk4_learned"):
        p, n_src = _particles(case, seed)
        if kind == "rk4_direct":
            solver = L.direct_solver(_prec(case))
        else:
            solver = L.tree_solver(L.LPM_PREC_F32, 8, case["leaf"], LEARNED_THETA, learned=True, tolerance=LEARNED_EPS)
        s["rk"] = L.RK4(ctx, L.biot_savart_kernel(), solver, n_src, p.shape[0])
        if kind == "rk4_learned":
            s["rk"].set_mlp(load_selector()[0])
            s["rk"].set_param("order_bias", LEARNED_BIAS)
        s["state"], s["out"] = p, torch.empty_like(p)
    else:
        members = [_particles(m, 101 * seed + i) for i, m in enumerate(_members(case))]
        solver = L.tree_solver(L.LPM_PREC_F32, 8, case["leaf"], LEARNED_THETA, learned=True, tolerance=LEARNED_EPS)
        s["ens"] = L.Ensemble(ctx, L.biot_savart_kernel(), solver, [n for _, n in members],
                              [p.shape[0] for p, _ in members], 8)
        s["ens"].set_mlp(load_selector()[0])
        s["ens"].set_param("order_bias", LEARNED_BIAS)
        s["inst"] = [s["ens"].instance(i) for i in range(len(members))]
        s["states"] = [p for p, _ in members]
        s["out"] = [torch.empty_like(p) for p, _ in members]
        torch.cuda.synchronize()  # the instances' own streams read the states
    s["ctx"] = ctx
    return s


def run(state):
    kind = state["kind"]
    if kind == "greens_host":
        return state["ctx"].direct_sum_mesh(L.sphere_greens_kernel(), L.LPM_PREC_F64, state["mesh"], state["src"])
    if kind in ("direct", "poisson_direct"):
        state["ctx"].direct_sum_dev(state["kernel"], state["prec"], state["src"], state["tgt"], state["out"],
                                    state["n_coincident"])
        return state["out"]
    if kind in ("tree", "poisson_tree"):
        state["tree"].eval(state["src"], state["tgt"], state["out"])
        return state["out"]
    if kind in ("rk4_direct", "rk4_learned"):
        state["rk"].set_state(state["state"])
        state["rk"].step(DT, 1, use_graph=True)
        return state["rk"].get_state(state["out"])
    for rk, p in zip(state["inst"], state["states"]):
        rk.set_state(p)
    state["ens"].step(DT, 1, use_graph=True)
    return [rk.get_state(o) for rk, o in zip(state["inst"], state["out"])]


# ------------------------------------------------------------------------------------------------ work
def _sizes(case):
    if "n" in case:
        return case["n"], case["n"]
    if "mesh" in case:
        icos, q = case["mesh"] == "icos", 4 ** case["level"]
        n_src, n_vert = (20 * q, 10 * q + 2) if icos else (6 * q, 6 * q + 2)
        return n_src, n_src + n_vert
    return case["n_src"], case["n_src"] + case["n_vert"]


def _tree_flops(n_src, n_tgt, leaf, scalar):
    """A treecode's operations, estimated: per target a level of the tree costs a few hundred far coefficients
    (8 or 2 operations each), and the leaves around it a few leaves' pairs (17 or 11 operations each)."""
    levels = max(1.0, math.log(max(n_src / leaf, 1.0)) / math.log(8.0 if scalar else 4.0))
    return n_tgt * ((2.0 * 6000 if scalar else 8.0 * 3000) * levels + (11.0 if scalar else 17.0) * 8.0 * leaf)


def work(case):
    kind = case["kind"]
    if kind == "ensemble":
        parts = [work({**m, "kind": "rk4_learned", "leaf": case["leaf"]}) for m in _members(case)]
        return {"bytes": sum(p["bytes"] for p in parts), "flops": sum(p["flops"] for p in parts)}
    n_src, n_tgt = _sizes(case)
    pairs = float(n_src) * n_tgt
    if kind == "direct":
        return {"bytes": 32.0 * n_src + 24.0 * n_tgt + 24.0 * n_tgt, "flops": 17.0 * pairs}
    if kind == "poisson_direct":
        return {"bytes": 32.0 * n_src + 24.0 * n_tgt + 8.0 * n_tgt, "flops": 11.0 * pairs}
    if kind == "greens_host":
        return {"bytes": 41.0 * n_src + 24.0 * n_tgt + 8.0 * n_tgt, "flops": 30.0 * pairs}
    if kind == "rk4_direct":
        return {"bytes": 64.0 * n_tgt, "flops": 4.0 * 17.0 * pairs}
    if kind == "rk4_learned":
        return {"bytes": 64.0 * n_tgt, "flops": 4.0 * _tree_flops(n_src, n_tgt, case["leaf"], False)}
    scalar = kind == "poisson_tree"
    return {"bytes": 32.0 * n_src + 24.0 * n_tgt + (8.0 if scalar else 24.0) * n_tgt,
            "flops": _tree_flops(n_src, n_tgt, case["leaf"], scalar)}


# ------------------------------------------------------------------------------------------------ 64-bit answers
def _chunks(n_tgt, n_src):
    step = max(1, int(2.5e8 / max(n_src, 1)))
    return range(0, n_tgt, step), step


def _velocity(src, tgt, delta=0.0):
    """-1/(4 pi) sum_j w_j (x cross y_j) / (1 - x . y_j + delta^2); terms with a vanishing denominator dropped."""
    out = torch.empty((3, tgt.shape[0]), dtype=torch.float64, device="cuda")
    y, w = src[:, :3].contiguous(), src[:, 3]
    starts, step = _chunks(tgt.shape[0], src.shape[0])
    for a in starts:
        x = tgt[a:a + step, :3]
        den = torch.addmm(torch.full((1, 1), 1.0 + delta * delta, dtype=torch.float64, device="cuda"), x, y.T, alpha=-1.0)
        f = torch.where(den.abs() > 1e-13, w / den, 0.0)
        g = f @ y - f.sum(dim=1, keepdim=True) * x
        out[:, a:a + step] = torch.linalg.cross(x, g).T / (-4.0 * math.pi)
    return out


def _potential(p):
    out = torch.empty((1, p.shape[0]), dtype=torch.float64, device="cuda")
    starts, step = _chunks(p.shape[0], p.shape[0])
    for a in starts:
        r2 = sum((p[a:a + step, c, None] - p[None, :, c]) ** 2 for c in range(3))
        out[0, a:a + step] = torch.where(r2 > 0.0, r2.rsqrt(), 0.0) @ p[:, 3] / (4.0 * math.pi)
    return out


def _rk4_step(p, n_src):
    def moved(base, a, u):
        q = base.clone()
        q[:, :3] = _unit(base[:, :3] + a * u.T)
        return q

    k1 = _velocity(p[:n_src], p)
    p1 = moved(p, 0.5 * DT, k1)
    k2 = _velocity(p1[:n_src], p1)
    p2 = moved(p, 0.5 * DT, k2)
    k3 = _velocity(p2[:n_src], p2)
    p3 = moved(p, DT, k3)
    k4 = _velocity(p3[:n_src], p3)
    return moved(p, DT / 6.0, k1 + 2.0 * k2 + 2.0 * k3 + k4)


def exact(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        members = _members(case)
        if sum(4.0 * a * b for a, b in map(_sizes, members)) > PAIRS_EXACT:
            return None
        return [_rk4_step(*_particles(m, 101 * seed + i)) for i, m in enumerate(members)]
    n_src, n_tgt = _sizes(case)
    pairs = float(n_src) * n_tgt * (4.0 if kind.startswith("rk4") else 1.0)
    if pairs > (PAIRS_EXACT if kind != "poisson_tree" else PAIRS_EXACT / 4.0):
        return None
    if kind in ("poisson_direct", "poisson_tree"):
        return _potential(_charges(case, seed))
    if kind == "greens_host":
        cen, area, div, vert, zeta = _host_mesh(case, seed)
        leaf = torch.nonzero(~div).reshape(-1)
        y, w = cen[leaf], zeta[leaf] * area[leaf]

        def psi(x, own):
            out = torch.empty(x.shape[0], dtype=torch.float64, device="cuda")
            starts, step = _chunks(x.shape[0], y.shape[0])
            for a in starts:
                k = 1.0 - sum(x[a:a + step, c, None] * y[None, :, c] for c in range(3))
                if own:
                    k[torch.arange(k.shape[0], device="cuda"), a + torch.arange(k.shape[0], device="cuda")] = 1.0
                out[a:a + step] = torch.log(k) @ w / (-4.0 * math.pi)
            return out

        face = torch.zeros((1, cen.shape[0]), dtype=torch.float64, device="cuda")
        face[0, leaf] = psi(y, True)
        return psi(vert, False)[None], face
    p, n_src = _particles(case, seed)
    if kind.startswith("rk4"):
        return _rk4_step(p, n_src)
    return _velocity(p[:n_src], p, case.get("delta", 0.0))
