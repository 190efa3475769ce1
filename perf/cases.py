"""The calls whose speed is tracked: what a program that uses fluidlets_gb300 has it do.

Each case is a plain dict; ``family`` says which public entry point it goes through and the other
entries are its sizes and options.  The listed sizes are those of the package's own benchmark
configurations, tests and serving mix, or ragged sizes near them; ``draw`` spreads others over the
same ranges.

``sum``      ``evaluate`` / ``evaluate_grid``: the velocity that given forces induce (plain FP64,
             the default, and the mixed-precision far field), real and complex, any kernel.
``assemble`` ``assemble``: the dense mobility matrix for a program that solves by itself.
``resist``   ``resistance``: forces on a body moving with given velocities, by the dense LU (FP64
             or tensor-core LU with FP64 refinement) or by matrix-free GMRES.
``swim``     ``swimming_problem``: one instant of a free swimmer, NumPy in and out as the callers
             (an ODE integrator) have it.
``serve``    ``SolveServer``: a burst of requests to a running server, waited for together.
"""
from __future__ import annotations

import atexit
import math

import numpy as np
import torch

import fluidlets_gb300 as fl
from fluidlets_gb300.geometry import biflagellate_shape, fibonacci_sphere_device
from fluidlets_gb300.serve import ResistanceRequest, SolveServer, SwimmerRequest

# flops of one pair interaction, by kernel (real strengths), and of one matrix block
PAIR_FLOPS = {"stokeslet": 31, "wall": 106, "brinkman": 60, "brinkman_c": 180}


def listed():
    return [
        # the velocity of a small swimmer's points at its own points (biflagellate model, 226
        # points): called once per stage by an integrator, so latency is what counts
        {"name": "sum_small", "family": "sum", "kernel": "stokeslet", "m": 226, "n": 226, "precision": "fp64",
         "strengths": "real", "layout": "points"},
        # the flow field around towers on a wall on the 32^3 grid of the legacy data set
        {"name": "sum_grid_wall", "family": "sum", "kernel": "wall", "m": 32768, "n": 1003, "precision": "fp64",
         "strengths": "real", "layout": "grid"},
        # oscillatory flow: complex alpha, complex strengths (one matvec of the complex GMRES)
        {"name": "sum_oscillatory", "family": "sum", "kernel": "brinkman_c", "m": 4099, "n": 2500,
         "precision": "fp64", "strengths": "complex", "layout": "points"},
        # an ordinary mixed-precision sum, where the plan of the near field weighs as much as the sum
        {"name": "sum_wall_mixed", "family": "sum", "kernel": "wall", "m": 8191, "n": 6145, "precision": "mixed",
         "strengths": "real", "layout": "points"},
        # the benchmark's kernel sum: 262,144 free and 16,384 wall targets, 262,144 sources
        {"name": "sum_wall_large", "family": "sum", "kernel": "wall", "m": 278528, "n": 262144,
         "precision": "mixed", "strengths": "real", "layout": "points"},
        # a rectangular mobility matrix near a wall (targets other than the sources)
        {"name": "assemble_wall", "family": "assemble", "kernel": "wall", "m": 1501, "n": 2003},
        # the default resistance call on the 1,536-point sphere: FP64 LU of 4,608 unknowns
        {"name": "resist_lu", "family": "resist", "kernel": "stokeslet", "n": 1536, "method": "auto",
         "precision": "fp64", "lu": "tf32", "alpha": 0.0},
        # the same solve in mixed precision
        {"name": "resist_mixed", "family": "resist", "kernel": "stokeslet", "n": 1536, "method": "lu",
         "precision": "mixed", "lu": "tf32", "alpha": 0.0},
        # a large body near the wall: BF16 LU of 24,576 unknowns refined in FP64
        {"name": "resist_mixed_wall", "family": "resist", "kernel": "wall", "n": 8192, "method": "lu",
         "precision": "mixed", "lu": "bf16", "alpha": 0.0},
        # matrix-free: porous medium (Brinkman), 49,152 unknowns
        {"name": "resist_gmres", "family": "resist", "kernel": "brinkman", "n": 16384, "method": "auto",
         "precision": "mixed", "lu": "tf32", "alpha": 1.0},
        # one instant of the biflagellate swimmer: 684 unknowns, FP64 LU
        {"name": "swim_instant", "family": "swim", "body": 96, "segments": 64, "precision": "fp64"},
        # twelve solves of uneven size that reach a running server together
        {"name": "serve_burst", "family": "serve", "requests": 12, "n_max": 2048},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    family = rng.choice(["sum", "sum", "sum", "assemble", "resist", "resist", "resist", "swim", "serve"])
    if family == "sum":
        precision = rng.choice(["fp64", "fp64", "mixed"])
        kernel = rng.choice(["stokeslet", "wall", "brinkman", "brinkman_c"])
        strengths = rng.choice(["real", "real", "complex"])
        if precision == "fp64":
            return {"family": "sum", "kernel": kernel, "m": _log_int(rng, 1, 40000), "n": _log_int(rng, 16, 5000),
                    "precision": precision, "strengths": strengths, "layout": "points"}
        return {"family": "sum", "kernel": kernel, "m": _log_int(rng, 1000, 100000), "n": _log_int(rng, 1000, 100000),
                "precision": precision, "strengths": strengths, "layout": "points"}
    if family == "assemble":
        return {"family": "assemble", "kernel": rng.choice(["stokeslet", "wall", "brinkman"]),
                "m": _log_int(rng, 64, 2300), "n": _log_int(rng, 64, 2300)}
    if family == "resist":
        how = rng.choice(["lu", "mixed", "gmres"])
        if how == "lu":
            return {"family": "resist", "kernel": rng.choice(["stokeslet", "wall"]), "n": _log_int(rng, 64, 2000),
                    "method": "auto", "precision": "fp64", "lu": "tf32", "alpha": 0.0}
        if how == "mixed":
            return {"family": "resist", "kernel": rng.choice(["stokeslet", "wall"]), "n": _log_int(rng, 64, 8192),
                    "method": "lu", "precision": "mixed", "lu": rng.choice(["tf32", "bf16"]), "alpha": 0.0}
        return {"family": "resist", "kernel": "brinkman", "n": _log_int(rng, 2100, 16384), "method": "auto",
                "precision": "mixed", "lu": "tf32", "alpha": rng.choice([0.0, 1.0, 10.0])}
    if family == "swim":
        return {"family": "swim", "body": _log_int(rng, 32, 400), "segments": _log_int(rng, 16, 128),
                "precision": rng.choice(["fp64", "mixed"])}
    return {"family": "serve", "requests": rng.randint(4, 12), "n_max": _log_int(rng, 400, 2048)}


# ---- inputs -----------------------------------------------------------------------------------
ALPHA_SUM = {"brinkman": 2.0, "brinkman_c": (1 + 1j) * math.sqrt(0.5)}  # (1 + i) sqrt(omega / 2) at omega = 1


def _kernel(name, alpha=None):
    if name == "stokeslet":
        return fl.Stokeslet3D()
    if name == "wall":
        return fl.WallStokeslet3D()
    return fl.Brinkmanlet3D(ALPHA_SUM[name] if alpha is None else alpha)


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _box(g, n):
    """n points uniform in [-1, 1]^2 x [0.02, 2], above the wall z = 0."""
    lo = torch.tensor([-1.0, -1.0, 0.02], dtype=torch.float64, device="cuda")
    hi = torch.tensor([1.0, 1.0, 2.0], dtype=torch.float64, device="cuda")
    return lo + (hi - lo) * torch.rand((n, 3), dtype=torch.float64, device="cuda", generator=g)


def _strengths(g, n, kind):
    f = torch.randn((n, 3), dtype=torch.float64, device="cuda", generator=g)
    if kind == "complex":
        f = torch.complex(f, torch.randn((n, 3), dtype=torch.float64, device="cuda", generator=g))
    return f


def _sum_inputs(case, seed):
    """Targets (points, or grid axes), sources, strengths, blob width.  Large target sets end with
    1/17 of them on the wall, as in the benchmark's 278,528 = 262,144 + 16,384."""
    g = _gen(seed)
    m, n = case["m"], case["n"]
    eps = 0.01 if n > 20000 else 0.25 * (8.0 / n) ** (1 / 3)
    Y = _box(g, n)
    f = _strengths(g, n, case["strengths"])
    if case["layout"] == "grid":
        k = round(m ** (1 / 3))
        shift = 0.05 * torch.rand(3, dtype=torch.float64, device="cuda", generator=g)
        t = torch.linspace(0.0, 1.0, k, dtype=torch.float64, device="cuda")
        return (-1.0 + 2 * t + shift[0], -1.0 + 2 * t + shift[1], 2 * t + shift[2]), Y, f, eps
    X = _box(g, m)
    if case["kernel"] == "wall" and m > 100000:
        X[m - m // 17:, 2] = 0.0
    return X, Y, f, eps


def _body(case, seed):
    """A sphere of radius 1 (1.05 above the wall for the wall kernel) and a rigid motion of it."""
    g = _gen(seed)
    n = case["n"]
    X = fibonacci_sphere_device(n)
    q, _ = torch.linalg.qr(torch.randn((3, 3), dtype=torch.float64, device="cuda", generator=g))
    X = X @ q.T
    if case["kernel"] == "wall":
        X = X + torch.tensor([0.0, 0.0, 1.05], dtype=torch.float64, device="cuda")
    U = torch.randn(3, dtype=torch.float64, device="cuda", generator=g)
    W = torch.randn(3, dtype=torch.float64, device="cuda", generator=g)
    V = U + torch.linalg.cross(W.expand(n, 3), X - X.mean(0))
    eps = 0.25 * math.sqrt(4 * math.pi / n)  # a quarter of the mean spacing
    return X.contiguous(), V.contiguous(), eps


def _shape(t1, t2, n_body=96, segments=64):
    """The biflagellate swimmer with its second flagellum out of phase (at t2, the first at t1), so
    that it also turns."""
    a, b = (biflagellate_shape(t, n_body=n_body, segments=segments, amplitude=0.08) for t in (t1, t2))
    i, j = n_body + segments, 4 * (n_body + segments)
    return fl.SwimmerShape(np.vstack([a.x[:i], b.x[i:]]), np.vstack([a.v[:i], b.v[i:]]),
                           np.vstack([a.X[:j], b.X[j:]]))


def _swimmer(case, seed):
    rng = np.random.default_rng(seed)
    shape = _shape(rng.uniform(0, 0.5), rng.uniform(0.5, 1), case["body"], case["segments"])
    B = np.linalg.qr(rng.normal(size=(3, 3)))[0]
    return shape, rng.normal(size=3), B * np.sign(np.linalg.det(B))


def _requests(case, seed):
    """The serving mix: rigid bodies of log-uniform size in free space or near a wall, and a
    quarter swimmers."""
    rng = np.random.default_rng(seed)
    sizes = np.random.default_rng(case["requests"])  # the same sizes for every seed: the same plans
    reqs = []
    for k in range(case["requests"]):
        n = int(round(math.exp(sizes.uniform(math.log(256), math.log(case["n_max"])))))
        B = np.linalg.qr(rng.normal(size=(3, 3)))[0]
        B = B * np.sign(np.linalg.det(B))
        if k % 4 == 3:
            reqs.append(SwimmerRequest(_shape(rng.uniform(0, 0.5), rng.uniform(0.5, 1)), np.zeros(3), B, 0.02))
            continue
        X = fibonacci_sphere_device(n).cpu().numpy() * np.array([sizes.uniform(1, 3), 1.0, 1.0]) @ B.T
        wall = k % 2 == 1
        if wall:
            X = X + np.array([0, 0, -X[:, 2].min() + 0.3])
        eps = 0.25 * math.sqrt(4 * math.pi / n)
        V = rng.normal(size=3) + np.cross(rng.normal(size=3), X - X.mean(0))
        reqs.append(ResistanceRequest(fl.WallStokeslet3D() if wall else fl.Stokeslet3D(), X, V, eps))
    return reqs


_server = None


def _the_server():
    """The one server that a program keeps running (its tensor-core mode fixed, so that a result
    does not depend on which mode a timing picked)."""
    global _server
    if _server is None:
        _server = SolveServer(slots=6, hbm_budget_gb=20.0, lu="tf32")
        atexit.register(_server.close)
    return _server


def prepare(case, seed):
    fam = case["family"]
    if fam == "sum":
        X, Y, f, eps = _sum_inputs(case, seed)
        return {"case": case, "kernel": _kernel(case["kernel"]), "X": X, "Y": Y, "f": f, "eps": eps}
    if fam == "assemble":
        g = _gen(seed)
        return {"case": case, "kernel": _kernel(case["kernel"]), "X": _box(g, case["m"]), "Y": _box(g, case["n"]),
                "eps": 0.25 * (8.0 / case["n"]) ** (1 / 3)}
    if fam == "resist":
        X, V, eps = _body(case, seed)
        return {"case": case, "kernel": _kernel(case["kernel"], case["alpha"]), "X": X, "V": V, "eps": eps}
    if fam == "swim":
        shape, x0, B = _swimmer(case, seed)
        return {"case": case, "shape": shape, "x0": x0, "B": B}
    return {"case": case, "server": _the_server(), "requests": _requests(case, seed)}


def run(state):
    c = state["case"]
    fam = c["family"]
    if fam == "sum":
        if c["layout"] == "grid":
            return fl.evaluate_grid(state["kernel"], state["X"], state["Y"], state["f"], state["eps"],
                                    precision=c["precision"])
        return fl.evaluate(state["kernel"], state["X"], state["Y"], state["f"], state["eps"],
                           precision=c["precision"])
    if fam == "assemble":
        return fl.assemble(state["kernel"], state["X"], state["Y"], state["eps"])
    if fam == "resist":
        forces, _ = fl.resistance(state["kernel"], state["X"], state["V"], state["eps"], method=c["method"],
                                  precision=c["precision"], lu=c["lu"])
        return forces
    if fam == "swim":
        s = fl.swimming_problem(state["shape"], state["x0"], state["B"], 0.02, precision=c["precision"])
        return {"U": s.U, "Omega": s.Omega, "forces": s.forces, "x": s.x, "X": s.X, "nearest": s.nearest}
    futures = [state["server"].submit(r) for r in state["requests"]]
    values = [fut.result().value for fut in futures]
    return [{"forces": v} if isinstance(v, np.ndarray) else {"forces": v.forces, "U": v.U, "Omega": v.Omega}
            for v in values]


def _flops(case):
    fam = case["family"]
    if fam == "sum":
        return case["m"] * case["n"] * PAIR_FLOPS[case["kernel"]] * (2 if case["strengths"] == "complex" else 1)
    if fam == "assemble":
        return case["m"] * case["n"] * PAIR_FLOPS[case["kernel"]]
    if fam == "resist":
        n = 3 * case["n"]
        if case["method"] == "auto" and n > fl.DENSE_MAX:
            return 12 * case["n"] ** 2 * PAIR_FLOPS[case["kernel"]]  # a dozen operator applications
        return 2 * n**3 / 3 + case["n"] ** 2 * PAIR_FLOPS[case["kernel"]]
    if fam == "swim":
        n = 3 * (case["body"] + 2 * case["segments"]) + 6
        return 2 * n**3 / 3 + 4 * n * n / 9 * PAIR_FLOPS["stokeslet"]
    return case["requests"] * 2 * (3 * math.sqrt(256 * case["n_max"])) ** 3 / 3


def work(case):
    """Inputs read once and outputs written once, in bytes, and the flops of the path's algorithm."""
    fam = case["family"]
    if fam == "sum":
        w = 2 if case["strengths"] == "complex" or case["kernel"] == "brinkman_c" else 1
        b = 24 * case["m"] + 24 * case["n"] * (2 if case["strengths"] == "real" else 3) + 24 * w * case["m"]
    elif fam == "assemble":
        b = 24 * (case["m"] + case["n"]) + 72 * case["m"] * case["n"]
    elif fam == "resist":
        b = 24 * 3 * case["n"]
    elif fam == "swim":
        b = 24 * 10 * (case["body"] + 2 * case["segments"])
    else:
        b = case["requests"] * 72 * math.sqrt(256 * case["n_max"])
    return {"bytes": int(b), "flops": int(_flops(case))}


# ---- the same outputs in plain 64-bit torch -----------------------------------------------------
_C1 = [(-1.0) ** k * (1 / math.factorial(k + 2) - 1 / math.factorial(k + 1) + 1 / math.factorial(k))
       for k in range(28)]
_C2 = [(-1.0) ** (k + 1) * (3 / math.factorial(k + 2) - 3 / math.factorial(k + 1) + 1 / math.factorial(k))
       for k in range(28)]


def _blocks(name, X, Y, eps, alpha=None):
    """G(x_i, y_j) of shape (m, n, 3, 3), mu = 1."""
    d = X[:, None, :] - Y[None, :, :]
    eye = torch.eye(3, dtype=torch.float64, device=X.device)
    Q = (d * d).sum(-1) + eps * eps
    R = Q.sqrt()
    dd = d[..., :, None] * d[..., None, :]
    if name in ("stokeslet", "wall"):
        G = ((1 / R + eps * eps / (Q * R))[..., None, None] * eye + dd / (Q * R)[..., None, None]) / (8 * math.pi)
        return G if name == "stokeslet" else G + _image(X, Y, eps)
    a = ALPHA_SUM[name] if alpha is None else alpha
    z = a * R
    zz = torch.where(z.abs() < 0.5, torch.ones_like(z), z)
    E = torch.exp(-zz)
    f1 = E * (1 + 1 / zz + 1 / zz**2) - 1 / zz**2
    f2 = 3 / zz**2 - E * (1 + 3 / zz + 3 / zz**2)
    s1, s2 = torch.zeros_like(z), torch.zeros_like(z)
    for c1, c2 in zip(reversed(_C1), reversed(_C2)):
        s1 = s1 * z + c1
        s2 = s2 * z + c2
    small = z.abs() < 0.5
    f1, f2 = torch.where(small, s1, f1), torch.where(small, s2, f2)
    B = f2 / (R * Q)
    A = f1 / R + eps * eps * B
    return (A[..., None, None] * eye + B[..., None, None] * dd) / (4 * math.pi)


def _image(X, Y, eps):
    """The image system of the regularized Stokeslet above the wall z = 0 (Ainley et al. 2008)."""
    h = Y[:, 2][None, :]
    e2 = eps * eps
    d = X[:, None, :] - Y[None, :, :] * torch.tensor([1.0, 1.0, -1.0], dtype=torch.float64, device=X.device)
    Q = (d * d).sum(-1) + e2
    i1, i3, i5 = Q**-0.5, Q**-1.5, Q**-2.5
    eye = torch.eye(3, dtype=torch.float64, device=X.device)
    dd = d[..., :, None] * d[..., None, :]

    def s(v):
        return v[..., None, None]

    z = torch.diag(torch.tensor([-1.0, -1.0, 1.0], dtype=torch.float64, device=X.device))
    G = -(s(0.5 * i1 + 0.5 * e2 * i3) * eye + s(0.5 * i3) * dd)
    G = G + (s(-h * h * (i3 - 3 * e2 * i5)) * eye + s(3 * h * h * i5) * dd) @ z
    b1, b2, b3 = -h * (3 * e2 * i5 + i3), h * i3, -3 * h * i5
    r1 = 3 * h * e2 * i5
    dz = d[..., 2]
    for a in range(2):
        for b in range(2):
            G[..., a, b] += -dz * ((b2 if a == b else 0.0) + d[..., a] * d[..., b] * b3)
        G[..., a, a] += r1 * dz
        G[..., a, 2] += d[..., a] * (b2 + dz * dz * b3)
        G[..., 2, a] += -d[..., a] * (b1 + dz * dz * b3) - r1 * d[..., a]
    G[..., 2, 2] += dz * (b1 + 2 * b2 + dz * dz * b3)
    return G / (4 * math.pi)


def _matrix(name, X, Y, eps, alpha=None):
    m, n = X.shape[0], Y.shape[0]
    K = torch.empty((3 * m, 3 * n), dtype=torch.float64, device=X.device)
    step = max(1, 4_000_000 // n)
    for i in range(0, m, step):
        G = _blocks(name, X[i:i + step], Y, eps, alpha)
        K[3 * i:3 * (i + step)] = G.permute(0, 2, 1, 3).reshape(-1, 3 * n)
    return K


def _conjugate_gradients(K, b):
    """K x = b for a symmetric positive definite K, to the rounding of 64 bits."""
    x, r = torch.zeros_like(b), b.clone()
    p, rr = r.clone(), r @ r
    for _ in range(400):
        q = K @ p
        a = rr / (p @ q)
        x, r = x + a * p, r - a * q
        new = r @ r
        if new.sqrt() < 1e-14 * b.norm():
            break
        p, rr = r + (new / rr) * p, new
    r = b - K @ x
    return x, float(r.norm() / b.norm())


def exact(case, seed):
    fam = case["family"]
    if fam == "sum":
        if case["m"] * case["n"] > 1_000_000_000:
            return None  # minutes in plain torch
        X, Y, f, eps = _sum_inputs(case, seed)
        if case["layout"] == "grid":
            x, y, z = X
            X = torch.stack([v.reshape(-1) for v in reversed(torch.meshgrid(z, y, x, indexing="ij"))], 1)
        step = max(1, 4_000_000 // case["n"])
        out = []
        for i in range(0, X.shape[0], step):
            G = _blocks(case["kernel"], X[i:i + step], Y, eps)
            dt = torch.promote_types(G.dtype, f.dtype)
            out.append(torch.einsum("mnab,nb->ma", G.to(dt), f.to(dt)))
        return torch.cat(out)
    if fam == "assemble":
        g = _gen(seed)
        X, Y = _box(g, case["m"]), _box(g, case["n"])
        return _matrix(case["kernel"], X, Y, 0.25 * (8.0 / case["n"]) ** (1 / 3))
    if fam == "resist":
        X, V, eps = _body(case, seed)
        K = _matrix(case["kernel"], X, X, eps, case["alpha"])
        if K.shape[0] > 25000:
            return _conjugate_gradients(K, V.reshape(-1))[0].reshape(-1, 3)
        return torch.linalg.solve(K, V.reshape(-1)).reshape(-1, 3)
    if fam == "swim":
        return _exact_swimmer(*_swimmer(case, seed))
    out = []
    for r in _requests(case, seed):
        if isinstance(r, SwimmerRequest):
            s = _exact_swimmer(r.shape, r.x0, r.B)
            out.append({k: s[k] for k in ("forces", "U", "Omega")})
            continue
        X = torch.from_numpy(np.ascontiguousarray(r.points)).cuda()
        K = _matrix("wall" if isinstance(r.kernel, fl.WallStokeslet3D) else "stokeslet", X, X, r.eps)
        b = torch.from_numpy(np.ascontiguousarray(r.velocities)).cuda().reshape(-1)
        out.append({"forces": torch.linalg.solve(K, b).reshape(-1, 3).cpu().numpy()})
    return out


def _exact_swimmer(shape, x0, B, eps=0.02):
    """Gallagher & Smith (2018), Eq. 8: forces, U and Omega of a free swimmer."""
    x, X, v = x0 + shape.x @ B.T, x0 + shape.X @ B.T, shape.v @ B.T
    xd, Xd = torch.from_numpy(x).cuda(), torch.from_numpy(X).cuda()
    n = len(x)
    nearest = ((Xd[:, None, :] - xd[None, :, :]) ** 2).sum(-1).argmin(1)
    K = _matrix("stokeslet", xd, Xd, eps).reshape(3 * n, -1, 3)
    A = torch.zeros((3 * n + 6, 3 * n + 6), dtype=torch.float64, device="cuda")
    Kg = torch.zeros((3 * n, n, 3), dtype=torch.float64, device="cuda").index_add_(1, nearest, K)
    A[:3 * n, :3 * n] = Kg.reshape(3 * n, 3 * n)
    r = xd - torch.from_numpy(np.asarray(x0)).cuda()
    count = torch.zeros(n, dtype=torch.float64, device="cuda").index_add_(0, nearest, torch.ones_like(Xd[:, 0]))
    S = torch.zeros((n, 3), dtype=torch.float64, device="cuda").index_add_(0, nearest, Xd)

    def cross(u):  # u x (.) as (k, 3, 3)
        o = torch.zeros_like(u[:, 0])
        return torch.stack([torch.stack([o, -u[:, 2], u[:, 1]], 1), torch.stack([u[:, 2], o, -u[:, 0]], 1),
                            torch.stack([-u[:, 1], u[:, 0], o], 1)], 1)

    eye = torch.eye(3, dtype=torch.float64, device="cuda")
    A[:3 * n, 3 * n:3 * n + 3] = -eye.repeat(n, 1)
    A[:3 * n, 3 * n + 3:] = cross(r).reshape(3 * n, 3)
    A[3 * n:3 * n + 3, :3 * n] = (count[:, None, None] * eye).permute(1, 0, 2).reshape(3, 3 * n)
    A[3 * n + 3:, :3 * n] = cross(S).permute(1, 0, 2).reshape(3, 3 * n)
    b = torch.zeros(3 * n + 6, dtype=torch.float64, device="cuda")
    b[:3 * n] = torch.from_numpy(np.ascontiguousarray(v)).cuda().reshape(-1)
    s = torch.linalg.solve(A, b).cpu().numpy()
    return {"U": s[3 * n:3 * n + 3], "Omega": s[3 * n + 3:], "forces": s[:3 * n].reshape(n, 3), "x": x, "X": X,
            "nearest": None}
