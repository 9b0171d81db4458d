"""The work that users of this framework have it do, as cases with sizes.

Each case names a ``kind`` (one way into the framework) and its sizes;
``listed()`` are the standing ones and ``draw(rng)`` gives more of the same
ranges.  Scenes come from ``fastmbcui_b200.scenes``: the point spacings, source
depths, densities and tolerances are those of the repository's scenes and
tests; only poses, shapes and sampled points change with the seed.

Kinds
  op        the mfs_torch operator with autograd: M.pinv @ F forward and the
            gradients of M and F backward, on a triangle-mesh scene
  assemble  the solid-angle collocation matrix and rigid-mode right-hand side
            of a mesh scene, as a simulation builds them every step
  solve     a new pose solved by the plain FP64 method (factor + batched PCG)
  many      isolated bodies of uneven size factored and solved concurrently
            (FP32 factor and recursion, FP64 residuals)
  boxes     boxes above a static floor: the mixed-precision solve, all rigid
            modes of the boxes, dense supernodes
  step      one step of a moving scene: a new FP32 factor and the block PCG of
            all rigid-mode columns on the INT8 FP64-accurate matvec, warm
            started from the poses before
  apply     the operator alone, K and K^T on a block of columns
  mass      added-mass tensor of solved strengths
"""
from __future__ import annotations

import math

import numpy as np
import torch

import fastmbcui_b200 as fb
from fastmbcui_b200 import mesh, scenes
from fastmbcui_b200.mfs_torch import ops
from fastmbcui_b200.trajectory import TrajectorySolver


def listed():
    return [
        # the smallest differentiable call: one coarse mesh body, where launches, copies and the host plan count
        {"name": "op_one_body", "kind": "op", "bodies": 1, "subdiv": 2},
        # a differentiable step of three fine mesh bodies (15360 faces, 7686 sources, 18 columns)
        {"name": "op_three_bodies", "kind": "op", "bodies": 3, "subdiv": 4},
        # the per-step collocation matrix of six fine mesh bodies, FP32 as the operator takes it
        {"name": "assemble_six_bodies", "kind": "assemble", "bodies": 6, "subdiv": 4},
        # the plain FP64 method on two bodies to the tight tolerance
        {"name": "solve_fp64", "kind": "solve", "bodies": 2, "pts": 1500},
        # the isolated solutions of uneven bodies, one solver and stream each
        {"name": "many_bodies", "kind": "many", "bodies": 10, "pts_min": 211, "pts_max": 803},
        # boxes above a floor at the dense pattern (rho 4, supernodes up to 512 wide)
        {"name": "boxes_floor", "kind": "boxes", "bodies": 6, "grid": 10, "floor_x": 120, "floor_y": 50},
        # one time step of 32 bodies, all 192 rigid-mode columns
        {"name": "step_32_bodies", "kind": "step", "bodies": 32, "pts": 750},
        # K and K^T in FP64 on the CUDA cores: residuals and the plain method, ten bodies, 60 columns
        {"name": "apply_fp64", "kind": "apply", "op": "fp64", "scene": "ellipsoids", "bodies": 10, "pts": 2000,
         "cols": 60},
        # the FP64-accurate INT8 operator at the width of a full block of columns
        {"name": "apply_int8_wide", "kind": "apply", "op": "int8", "scene": "ellipsoids", "bodies": 24, "pts": 2000,
         "cols": 144},
        # ... and at the width to which a block narrows once most columns have converged, ragged sizes
        {"name": "apply_int8_tail", "kind": "apply", "op": "int8", "scene": "ellipsoids", "bodies": 15, "pts": 2013,
         "cols": 41},
        # FP32 products of the coin scene, all 96 rigid modes of 16 coins
        {"name": "apply_fp32_coins", "kind": "apply", "op": "fp32", "scene": "coins", "bodies": 16, "pts": 4000,
         "cols": 96},
        # added mass and forces of 16 bodies, all rigid modes
        {"name": "added_mass", "kind": "mass", "bodies": 16, "pts": 2000},
    ]


def _spread(rng, lo, hi):
    """An integer in [lo, hi], spread over the logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["op", "assemble", "solve", "many", "boxes", "step", "apply", "apply", "apply", "mass"])
    if kind == "op":
        subdiv = rng.choice([2, 3, 4])
        return {"kind": kind, "bodies": rng.randint(1, 2 if subdiv == 4 else 6), "subdiv": subdiv}
    if kind == "assemble":
        return {"kind": kind, "bodies": rng.randint(1, 6), "subdiv": rng.choice([2, 3, 4])}
    if kind == "solve":
        return {"kind": kind, "bodies": rng.randint(1, 3), "pts": _spread(rng, 150, 1000)}
    if kind == "many":
        lo = _spread(rng, 100, 400)
        return {"kind": kind, "bodies": rng.randint(3, 10), "pts_min": lo, "pts_max": lo + _spread(rng, 20, 400)}
    if kind == "boxes":
        return {"kind": kind, "bodies": (b := rng.randint(2, 6)), "grid": rng.randint(4, 10),
                "floor_x": 20 * b - rng.randint(0, 4), "floor_y": rng.randint(35, 50)}
    if kind == "step":
        return {"kind": kind, "bodies": _spread(rng, 2, 31), "pts": _spread(rng, 150, 750)}
    if kind == "apply":
        op = rng.choice(["fp64", "int8", "fp32"])
        scene = rng.choice(["ellipsoids", "coins"])
        most = 12 if op == "fp64" else 16
        bodies = _spread(rng, 1, most)
        return {"kind": kind, "op": op, "scene": scene, "bodies": bodies, "pts": _spread(rng, 150, 1990),
                "cols": _spread(rng, 1, 6 * bodies)}
    return {"kind": kind, "bodies": _spread(rng, 1, 15), "pts": _spread(rng, 150, 2000)}


# --------------------------------------------------------------------------
# scenes
# --------------------------------------------------------------------------

def _dev(a, dtype=torch.float32):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=dtype, device="cuda")


def _f32(parts):
    """Stacked, with the coordinates rounded to FP32 values."""
    return np.concatenate(parts).astype(np.float32).astype(np.float64)


def _mesh(case, seed):
    """Turned icospheres in a row, sources 0.05 inside along the vertex normals."""
    rng = np.random.default_rng(seed)
    bodies = []
    for b in range(case["bodies"]):
        bodies.append((case["subdiv"], tuple(rng.uniform(0.6, 1.0, 3)), tuple(rng.uniform(-1.0, 1.0, 3)),
                       (2.6 * b, *rng.uniform(-0.3, 0.3, 2)), 0.05))
    return scenes.mesh_scene(bodies)


def _scene(case, seed):
    kind = case["kind"]
    if kind == "boxes":
        return _boxes(case["bodies"], case["grid"], case["floor_x"], case["floor_y"], seed)
    if kind == "apply" and case["scene"] == "coins":
        return scenes.coins_scene(case["bodies"], case["pts"], sample_seed=seed, pose_seed=seed + 1, box=12.0)
    return _ellipsoids(case["bodies"], case["pts"], seed)


_DEPTH = 1.15  # source depth in point spacings


def _ellipsoids(bodies, pts, seed, motion=0.0):
    """Random ellipsoids (semi-axes U[0.5, 1.5]) on the mapped Fibonacci
    lattice of scenes.ellipsoid_fibonacci_scene, sources somewhat more than a
    point spacing inside, placed with room for a motion."""
    rng = np.random.default_rng(seed)
    axes = rng.uniform(0.5, 1.5, size=(bodies, 3))
    box = 12.0 + 8.0 * motion
    while True:
        try:
            centers = scenes.random_centers(rng, axes.max(axis=1) + motion, box)
            break
        except RuntimeError:
            box += 0.5
    t = axes ** 1.6075  # areas by Thomsen's formula (1 %)
    areas = 4 * np.pi * ((t[:, 0] * t[:, 1] + t[:, 0] * t[:, 2] + t[:, 1] * t[:, 2]) / 3) ** (1 / 1.6075)
    u = scenes.fibonacci_sphere(pts)
    x, nx, y, w = [], [], [], []
    for b in range(bodies):
        p, n = u * axes[b], u / axes[b]
        n /= np.linalg.norm(n, axis=1, keepdims=True)
        R = scenes.random_rotation(rng)
        w.append((4.0 * np.pi / pts) * np.prod(axes[b]) * np.linalg.norm(u / axes[b], axis=1))
        p, n = p @ R.T + centers[b], n @ R.T
        x.append(p)
        nx.append(n)
        y.append(p - _DEPTH * math.sqrt(areas[b] / pts) * n)
    body = np.repeat(np.arange(bodies, dtype=np.int32), pts)
    return scenes.Scene(name=f"ellipsoids{bodies}", x=_f32(x), nx=_f32(nx), y=_f32(y), row_body=body, src_body=body,
                        centers=_f32([centers]), meta={"weights": np.concatenate(w)})


def _boxes(bodies, grid, floor_x, floor_y, seed):
    """Boxes (edge U[0.3, 1], turned, ``grid`` x ``grid`` points a face) above a
    static floor grid, sources 0.6 spacings inside, rho 4 and supernodes up to
    512 wide as in scenes.large_scene."""
    rng = np.random.default_rng(seed)
    x, nx, y, body, centers = [], [], [], [], []
    c = (np.arange(grid) + 0.5) / grid - 0.5
    a, b = (t.ravel() for t in np.meshgrid(c, c, indexing="ij"))
    spacing = 0.1
    span = (floor_x - 1) * spacing / bodies
    for k in range(bodies):
        side = rng.uniform(0.3, 1.0)
        p, n = [], []
        for ax in range(3):
            for sign in (-1.0, 1.0):
                q, m = np.zeros((grid * grid, 3)), np.zeros((grid * grid, 3))
                q[:, ax], q[:, (ax + 1) % 3], q[:, (ax + 2) % 3] = 0.5 * sign, a, b
                m[:, ax] = sign
                p.append(q * side)
                n.append(m)
        R = scenes.random_rotation(rng)
        cen = np.array([(k + 0.5) * span, rng.uniform(1.0, (floor_y - 1) * spacing - 1.0), rng.uniform(1.0, 2.5)])
        p, n = np.concatenate(p) @ R.T + cen, np.concatenate(n) @ R.T
        x.append(p)
        nx.append(n)
        y.append(p - 0.6 * side / grid * n)
        body += [k] * p.shape[0]
        centers.append(cen)
    gx, gy = np.meshgrid(np.arange(floor_x) * spacing, np.arange(floor_y) * spacing, indexing="ij")
    p = np.stack([gx.ravel(), gy.ravel(), np.zeros(gx.size)], 1)
    n = np.tile([0.0, 0.0, 1.0], (p.shape[0], 1))
    body = np.array(body + [bodies] * p.shape[0], np.int32)
    return scenes.Scene(name=f"boxes{bodies}", x=_f32(x + [p]), nx=_f32(nx + [n]), y=_f32(y + [p - 0.6 * spacing * n]),
                        row_body=body, src_body=body, centers=_f32([centers, [p.mean(0)]]), rho=4.0, max_super=512,
                        meta={"static": [bodies]})


def _uneven(case):
    """Points of each isolated body: evenly spread over the case's range."""
    return [int(round(p)) for p in np.linspace(case["pts_min"], case["pts_max"], case["bodies"])]


def _isolated(case, seed):
    return [_ellipsoids(1, p, 1000 * seed + b) for b, p in enumerate(_uneven(case))]


def _moving(case, seed, steps=4):
    base = _ellipsoids(case["bodies"], case["pts"], seed, motion=0.21)
    q, _ = scenes.trajectory_poses(case["bodies"], steps, seed + 1, amp_range=(0.005, 0.03))
    return [scenes.moved(base, q[k]) for k in range(steps)]


def _points(sc):
    return {"x": _dev(sc.x), "nx": _dev(sc.nx), "y": _dev(sc.y), "coef": sc.coef}


def _plan(sc):
    return fb.Plan(sc.y, sc.rho, sc.lam, sc.max_super)


def _block(seed, rows, cols, dtype):
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    return torch.randn(rows, cols, generator=g, device="cuda", dtype=torch.float64).to(dtype)


# --------------------------------------------------------------------------
# what a program has in hand, and one pass
# --------------------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    if kind == "op":
        m = _mesh(case, seed)
        M, rhs = mesh.assemble(m["V"], m["F"], m["S"], m["face_body"], m["body_pos"])
        # a deforming surface: the rigid modes and a tenth of them in uncorrelated velocity
        rhs = rhs + 0.1 * rhs.abs().max() * _block(seed + 1, rhs.shape[0], rhs.shape[1], torch.float32)
        return {"kind": kind, "M": M.requires_grad_(True), "F": rhs.requires_grad_(True),
                "S": torch.as_tensor(m["S"]), "G": _block(seed, M.shape[1], rhs.shape[1], torch.float32)}
    if kind == "assemble":
        m = _mesh(case, seed)
        return {"kind": kind, "V": _dev(m["V"]), "F": _dev(m["F"], torch.int32), "S": _dev(m["S"]),
                "face_body": _dev(m["face_body"], torch.int32), "body_pos": _dev(m["body_pos"])}
    if kind == "many":
        scs = _isolated(case, seed)
        return {"kind": kind, "plans": [_plan(sc) for sc in scs], "points": [_points(sc) for sc in scs],
                "F": [_dev(sc.rhs()) for sc in scs]}
    if kind == "step":
        scs = _moving(case, seed)
        sc = scs[-1]
        h = [_strengths(s) for s in scs[:-1]]  # the poses before, solved
        return {"kind": kind, "plan": _plan(sc), "points": _points(sc), "F": _dev(sc.rhs()),
                "X0": (3.0 * h[2] - 3.0 * h[1] + h[0]).float()}
    sc = _scene(case, seed)
    if kind in ("solve", "boxes"):
        return {"kind": kind, "plan": _plan(sc), "points": _points(sc),
                "F": _dev(sc.rhs(), torch.float64 if kind == "solve" else torch.float32)}
    if kind == "apply":
        f32 = case["op"] == "fp32"
        dtype = torch.float32 if f32 else torch.float64
        s = fb.Solver(_plan(sc), **_points(sc), precision=fb.MBC_F32 if f32 else fb.MBC_F64)
        if case["op"] == "int8":
            s.set_fp64_matvec("int8").prepare()
        return {"kind": kind, "solver": s, "V": _block(seed, sc.n, case["cols"], dtype),
                "W": _block(seed + 1, sc.nf, case["cols"], dtype)}
    s = fb.Solver(_plan(sc), **_points(sc), precision=fb.MBC_F32)
    return {"kind": kind, "solver": s, "X": _block(seed, sc.n, 6 * case["bodies"], torch.float32),
            "weights": sc.weights(), "body_ptr": sc.body_ptr(), "centers": sc.centers,
            "accel": np.random.default_rng(seed).standard_normal(6 * case["bodies"])}


def run(state):
    kind = state["kind"]
    if kind == "op":
        A = ops.MinvF_float_fastGrad(state["M"], state["F"], state["S"], 3.0, 2000, 1e-10)
        gM, gF = torch.autograd.grad(A, (state["M"], state["F"]), state["G"])
        return {"A": A.detach(), "grad_M": gM, "grad_F": gF}
    if kind == "assemble":
        M, rhs = mesh.assemble(state["V"], state["F"], state["S"], state["face_body"], state["body_pos"])
        return {"M": M, "rhs": rhs}
    if kind == "solve":
        s = fb.Solver(state["plan"], **state["points"], precision=fb.MBC_F64).factor()
        return s.solve(state["F"], out_dtype=torch.float32, tol=1e-10, max_iters=4000)[0]
    if kind == "many":
        solvers = [fb.Solver(p, **pts, precision=fb.MBC_F32) for p, pts in zip(state["plans"], state["points"])]
        res = fb.solve_many(solvers, state["F"], out_dtype=torch.float32, tol=1e-10, max_iters=4000)
        return [X for X, _ in res]
    if kind == "boxes":
        s = fb.Solver(state["plan"], **state["points"], precision=fb.MBC_F32).factor()
        return s.solve(state["F"], out_dtype=torch.float32, tol=1e-10, max_iters=4000)[0]
    if kind == "step":
        p = state["points"]
        ts = TrajectorySolver(p["coef"], mode="mixed", fp64_matvec="int8")
        s = ts.solver(state["plan"], p["x"], p["nx"], p["y"])
        return s.solve(state["F"], X0=state["X0"], out_dtype=torch.float32, tol=ts.tol, max_iters=ts.max_iters,
                       check_every=ts.check_every, schedule=ts.schedule, fp64_recursion=1)[0]
    if kind == "apply":
        s = state["solver"]
        return {"KV": s.apply_K(state["V"]), "KTW": s.apply_KT(state["W"])}
    Mf, forces = state["solver"].added_mass(state["X"], state["weights"], state["body_ptr"], state["centers"], 1.0,
                                            state["accel"])
    return {"Mf": Mf, "forces": forces}


# --------------------------------------------------------------------------
# what a pass cannot do without
# --------------------------------------------------------------------------

# products with K and with K^T that a solve is counted with: what a well
# conditioned scene takes at least, whatever the preconditioner
_PRODUCTS = 2 * 10


def work(case):
    kind = case["kind"]
    if kind in ("op", "assemble"):
        n = case["bodies"] * (10 * 4 ** case["subdiv"] + 2)
        nf = case["bodies"] * 20 * 4 ** case["subdiv"]
        R = 6 * case["bodies"]
        if kind == "assemble":
            return {"bytes": 4.0 * nf * (n + R) + 12.0 * (2 * nf + 2 * n), "flops": 60.0 * nf * n}
        # M read for the solves and for the gradient, grad_M written; the solves' products and the gradient's
        return {"bytes": 4.0 * nf * n * 2 + 4.0 * R * (2 * nf + 3 * n), "flops": (2 * _PRODUCTS + 4) * 2.0 * nf * n * R}
    if kind == "many":
        pts = _uneven(case)
        return {"bytes": sum(p * (36.0 + 8 * 6) for p in pts), "flops": sum(_PRODUCTS * 2.0 * p * p * 6 for p in pts)}
    n = case["bodies"] * (6 * case["grid"] ** 2 if kind == "boxes" else case["pts"])
    cols = case.get("cols", 6 * case["bodies"])
    if kind == "boxes":
        n += case["floor_x"] * case["floor_y"]
    if kind == "apply":
        size = 4.0 if case["op"] == "fp32" else 8.0
        return {"bytes": 36.0 * n + 4 * size * n * cols, "flops": 2 * n * n * (20.0 + 2.0 * cols)}
    if kind == "mass":
        return {"bytes": n * (40.0 + 4 * cols) + 8.0 * cols * cols, "flops": n * n * (12.0 + 2.0 * cols)}
    return {"bytes": n * (36.0 + 12.0 * cols), "flops": _PRODUCTS * n * n * (20.0 + 2.0 * cols)}


# --------------------------------------------------------------------------
# the results in 64 bits
# --------------------------------------------------------------------------

_ROWS = 2048  # rows of a matrix that are formed at a time


def _kernel_rows(sc, i0, i1):
    """Rows i0 .. i1 of K in FP64: coef ((x - y) . n) / |x - y|^3."""
    d64 = torch.float64
    x, nx, y = _dev(sc.x[i0:i1], d64), _dev(sc.nx[i0:i1], d64), _dev(sc.y, d64)
    dot, r2 = 0.0, 0.0
    for k in range(3):
        d = x[:, k, None] - y[None, :, k]
        r2 = r2 + d * d
        dot = dot + d * nx[:, k, None]
    return sc.coef * dot / (r2 * r2.sqrt())


def _matrix(sc):
    return torch.cat([_kernel_rows(sc, i, min(i + _ROWS, sc.nf)) for i in range(0, sc.nf, _ROWS)])


def _strengths(sc):
    """The strengths of all rigid modes: K is square and K X = F."""
    return torch.linalg.solve(_matrix(sc), _dev(sc.rhs(), torch.float64))


def _solid_angles(m):
    """M in FP64: 2 atan2(R1 . (R2 x R3), l1 l2 l3 + (R1.R2) l3 + (R1.R3) l2 + (R2.R3) l1)."""
    V, S = _dev(m["V"], torch.float64), _dev(m["S"], torch.float64)
    F = _dev(m["F"], torch.int64)
    out = torch.empty(F.shape[0], S.shape[0], dtype=torch.float64, device="cuda")
    for i in range(0, F.shape[0], _ROWS):
        r = [V[F[i:i + _ROWS, k]][:, None, :] - S[None] for k in range(3)]
        ln = [t.norm(dim=-1) for t in r]
        dot = lambda a, b: (r[a] * r[b]).sum(-1)
        num = (r[0] * torch.linalg.cross(r[1], r[2])).sum(-1)
        den = ln[0] * ln[1] * ln[2] + dot(0, 1) * ln[2] + dot(0, 2) * ln[1] + dot(1, 2) * ln[0]
        out[i:i + _ROWS] = 2.0 * torch.atan2(num, den)
    return out


def _mesh_rhs(m):
    V, F = _dev(m["V"], torch.float64), _dev(m["F"], torch.int64)
    v = [V[F[:, k]] for k in range(3)]
    s = torch.linalg.cross(v[1] - v[0], v[2] - v[0]) / 2
    body = _dev(m["face_body"], torch.int64)
    r = (v[0] + v[1] + v[2]) / 3 - _dev(m["body_pos"], torch.float64)[body]
    out = torch.zeros(F.shape[0], m["body_pos"].shape[0], 6, dtype=torch.float64, device="cuda")
    out[torch.arange(F.shape[0], device="cuda"), body] = torch.cat([s, torch.linalg.cross(r, s)], 1)
    return out.reshape(F.shape[0], -1)


def exact(case, seed):
    kind = case["kind"]
    if kind == "assemble":
        m = _mesh(case, seed)
        return {"M": _solid_angles(m), "rhs": _mesh_rhs(m)}
    if kind == "op":
        # the operator's input is the FP32 matrix: the results in 64 bits are those of these FP32 values
        s = prepare(case, seed)
        M, F, G = (s[k].detach().double() for k in ("M", "F", "G"))
        L = torch.linalg.cholesky(M.T @ M)
        A = torch.cholesky_solve(M.T @ F, L)
        A = A + torch.cholesky_solve(M.T @ (F - M @ A), L)
        P = torch.cholesky_solve(G, L)
        P = P + torch.cholesky_solve(G - M.T @ (M @ P), L)
        return {"A": A, "grad_M": (F - M @ A) @ P.T - (M @ P) @ A.T, "grad_F": M @ P}
    if kind == "many":
        return [_strengths(sc) for sc in _isolated(case, seed)]
    if kind == "step":
        return _strengths(_moving(case, seed)[-1])
    sc = _scene(case, seed)
    if kind in ("solve", "boxes"):
        return _strengths(sc)
    if kind == "apply":
        dtype = torch.float32 if case["op"] == "fp32" else torch.float64
        V = _block(seed, sc.n, case["cols"], dtype).double()
        W = _block(seed + 1, sc.nf, case["cols"], dtype).double()
        KV, KTW = torch.empty(sc.nf, V.shape[1], dtype=V.dtype, device="cuda"), torch.zeros_like(V)
        for i in range(0, sc.nf, _ROWS):
            K = _kernel_rows(sc, i, min(i + _ROWS, sc.nf))
            KV[i:i + _ROWS] = K @ V
            KTW += K.T @ W[i:i + _ROWS]
        return {"KV": KV, "KTW": KTW}
    X = _block(seed, sc.n, 6 * case["bodies"], torch.float32).double()
    y = _dev(sc.y, torch.float64)
    phi = torch.empty(sc.nf, X.shape[1], dtype=torch.float64, device="cuda")
    for i in range(0, sc.nf, _ROWS):
        x = _dev(sc.x[i:i + _ROWS], torch.float64)
        r2 = sum((x[:, k, None] - y[None, :, k]) ** 2 for k in range(3))
        phi[i:i + _ROWS] = r2.rsqrt() @ X / (4 * math.pi)
    phi, w, ptr = phi.cpu().numpy(), sc.weights(), sc.body_ptr()
    Mf = np.empty((6 * sc.n_bodies, X.shape[1]))
    for a in range(sc.n_bodies):
        k = slice(ptr[a], ptr[a + 1])
        N = np.concatenate([sc.nx[k], np.cross(sc.x[k] - sc.centers[a], sc.nx[k])], 1)
        Mf[6 * a:6 * a + 6] = -(N * w[k, None]).T @ phi[k]
    accel = np.random.default_rng(seed).standard_normal(6 * case["bodies"])
    return {"Mf": Mf, "forces": -Mf @ accel}
