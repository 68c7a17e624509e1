"""What the engine is timed on: the calls its users make, over the range of sizes they make them at.

  listed()            the cases, each a dict of plain values
  draw(rng)           one more case of the same ranges
  prepare(case, seed) what a program has in hand before the call
  run(state)          one pass through the public entry points, and its outputs
  work(case)          the bytes and operations one pass cannot do without
  exact(case, seed)   what run() returns, computed in 64 bits by plain torch

Five kinds of case:

  tets     cubes of tetrahedra (one scene, or a batch of uneven independent scenes), a frame of `steps` steps: the
           positions and velocities are set, the steps run (a fixed number of iterations, or each scene to its
           residual tolerance), positions and velocities are read back.  Options: precision, ground contact, a fixed
           bottom, strain-rate damping, surface triangles in the collision stage, the learned warm start.
  rods     Cosserat rods on one-sided fixed joints and rigid spheres on the ground, collision stage over the
           segments; the simulation goes on from pass to pass.
  contacts rods lying on a soft cube: triangle-rod narrow phase, contact pool, recoloring; goes on likewise.
  mlp      inference of the warm start's network on rows of features.
  train    mini-batch steps of its trainer, then the parameters.
"""
from __future__ import annotations

import functools
import heapq
import math

import numpy as np
import torch

DT, GRAVITY, RHO, DENSITY = 1.0 / 60.0, 9.81, 0.5, 1000.0
MU_S, MU_K = 0.4, 0.2
MLP_IN, MLP_PAD, MLP_HID, MLP_OUT, MLP_OUT_PAD = 27, 32, 128, 3, 16
NPARAMS = 39312


# ------------------------------------------------------------------ the cases
def _tets(**kw):
    c = {"kind": "tets", "scenes": 1, "n_min": 8, "n_max": 8, "precision": "fp32", "iters": 15, "tol": 0.0,
         "max_iters": 0, "ground": True, "fixed": False, "damping": 0.0, "surface": False, "learned": False, "steps": 1}
    c.update(kw)
    return c


def listed():
    return [
        # one small scene stepped interactively in full precision: 40 color phases of some 180 vertices
        _tets(name="cube8_fp64", precision="fp64", iters=10, ground=False, fixed=True),
        # one large deformable on the ground with its surface in the collision stage
        _tets(name="drop32_fp32", n_min=32, n_max=32, iters=20, surface=True),
        # an odd middle size, FP64 state with FP32 element records
        _tets(name="cube17_mixed", n_min=17, n_max=17, precision="mixed", steps=2),
        # the damped material
        _tets(name="damped12_fp32", n_min=12, n_max=12, iters=20, damping=10.0, steps=2),
        # many uneven scenes, each to its residual tolerance: the serving case, records larger than L2
        _tets(name="batch64_tol_mixed", scenes=64, n_min=4, n_max=24, precision="mixed", tol=1e-4, max_iters=100,
              steps=2),
        # the same with a fixed iteration budget
        _tets(name="batch48_fixed_mixed", scenes=48, n_min=4, n_max=24, precision="mixed", steps=2),
        # scenes whose initial guess the learned warm start corrects
        _tets(name="batch24_learned_mixed", scenes=24, n_min=4, n_max=16, precision="mixed", tol=1e-4, max_iters=100,
              learned=True, steps=2),
        # many rods and rigid bodies in single precision
        {"name": "rods256_fp32", "kind": "rods", "rods": 256, "segments": 100, "spheres": 64, "precision": "fp32",
         "iters": 20, "steps": 2},
        # a few rods in full precision: latency
        {"name": "rods12_fp64", "kind": "rods", "rods": 12, "segments": 33, "spheres": 5, "precision": "fp64",
         "iters": 10, "steps": 2},
        # changing contacts between rods and a deformable
        {"name": "contacts_rods24_cube32", "kind": "contacts", "n": 32, "rods": 24, "segments": 32,
         "precision": "fp32", "iters": 20, "steps": 1},
        # the warm start's network on a batch's vertices
        {"name": "mlp_1000003_rows", "kind": "mlp", "rows": 1000003},
        # its training loop
        {"name": "train_8192", "kind": "train", "batch": 8192, "steps": 4},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["single", "single", "batch_tol", "batch_fixed", "rods", "contacts", "mlp", "train"])
    if kind == "single":
        n = _log_int(rng, 4, 32)
        fixed = rng.random() < 0.3
        return _tets(n_min=n, n_max=n, precision=rng.choice(["fp32", "mixed", "fp64"]), iters=rng.randint(8, 20),
                     fixed=fixed, ground=not fixed, surface=rng.random() < 0.5,
                     damping=round(rng.uniform(1.0, 20.0), 2) if rng.random() < 0.2 else 0.0, steps=rng.randint(1, 2))
    if kind in ("batch_tol", "batch_fixed"):
        lo = rng.randint(3, 7)
        c = _tets(scenes=_log_int(rng, 3, 48), n_min=lo, n_max=rng.randint(lo + 1, 24))
        if kind == "batch_tol":
            c.update(precision=rng.choice(["mixed", "mixed", "fp64"]), tol=1e-4, max_iters=rng.randint(60, 100),
                     learned=rng.random() < 0.2)
        else:
            c.update(precision=rng.choice(["mixed", "mixed", "fp64"]), iters=rng.randint(8, 20))
        return c
    if kind == "rods":
        return {"kind": "rods", "rods": _log_int(rng, 1, 256), "segments": rng.randint(7, 100),
                "spheres": rng.randint(0, 64), "precision": rng.choice(["fp32", "fp64", "mixed"]),
                "iters": rng.randint(8, 20), "steps": rng.randint(1, 2)}
    if kind == "contacts":
        return {"kind": "contacts", "n": rng.randint(8, 28), "rods": rng.randint(2, 20), "segments": rng.randint(8, 32),
                "precision": rng.choice(["fp32", "mixed"]), "iters": rng.randint(10, 20), "steps": 1}
    if kind == "mlp":
        return {"kind": "mlp", "rows": _log_int(rng, 1, 1000000)}
    return {"kind": "train", "batch": 128 * _log_int(rng, 1, 64), "steps": rng.randint(2, 4)}


def _cells(case):
    """Cells per side of each scene: spread over [n_min, n_max], the largest and smallest mixed."""
    lo, span = case["n_min"], case["n_max"] - case["n_min"] + 1
    step = next(s for s in (8, 7, 5, 3, 1) if math.gcd(s, span) == 1)
    return [lo + (step * k + span // 2) % span for k in range(case["scenes"])]


# ------------------------------------------------------------------ the inputs
@functools.lru_cache(maxsize=None)
def _grid(n):
    """(n+1)^3 vertices (x fastest) and 6 tets per cell, cell by cell; rest rows Q, volumes and nodal volume."""
    m = n + 1
    a = np.arange(m) / n
    z, y, x = np.meshgrid(a, a, a, indexing="ij")
    X = np.stack([x.ravel(), y.ravel(), z.ravel()], axis=1)
    k, j, i = (v.ravel() for v in np.meshgrid(np.arange(n), np.arange(n), np.arange(n), indexing="ij"))
    unit = np.eye(3, dtype=np.int64)
    vid = lambda o: (i + o[0]) + m * ((j + o[1]) + m * (k + o[2]))  # noqa: E731
    T = []
    for p in ((0, 1, 2), (0, 2, 1), (1, 0, 2), (1, 2, 0), (2, 0, 1), (2, 1, 0)):
        T.append(np.stack([vid((0, 0, 0)), vid(unit[p[0]]), vid(unit[p[0]] + unit[p[1]]), vid((1, 1, 1))], axis=1))
    T = np.stack(T, axis=1).reshape(-1, 4)
    return (X, T) + _rest(X, T)


def _rest(X, T):
    a, b, c = X[T[:, 0]] - X[T[:, 3]], X[T[:, 1]] - X[T[:, 3]], X[T[:, 2]] - X[T[:, 3]]
    r0, r1, r2 = np.cross(b, c), np.cross(c, a), np.cross(a, b)
    det = np.einsum("ij,ij->i", a, r0)
    return np.stack([r0, r1, r2], axis=1) / det[:, None, None], np.abs(det) / 6


@functools.lru_cache(maxsize=None)
def _surface(n):
    T = _grid(n)[1]
    f = np.concatenate([T[:, [0, 1, 2]], T[:, [0, 1, 3]], T[:, [0, 2, 3]], T[:, [1, 2, 3]]])
    _, inv, cnt = np.unique(np.sort(f, axis=1), axis=0, return_inverse=True, return_counts=True)
    return f[cnt[inv.ravel()] == 1]


def _rotation(rng):
    w, x, y, z = (q := rng.normal(size=4)) / np.linalg.norm(q)
    return np.array([[1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y)],
                     [2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x)],
                     [2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)]])


def _tet_inputs(case, seed):
    """Every scene's mesh, rest state, material, positions and velocities."""
    rng = np.random.default_rng([seed, 1])
    cells = _cells(case)
    side = math.ceil(math.sqrt(len(cells)))
    out = []
    for s, n in enumerate(cells):
        X, T, Q, V = _grid(n)
        nu = rng.uniform(0.3, 0.49)
        E = 10 ** rng.uniform(4, 7) if case["scenes"] > 1 else (1e5 if case["fixed"] else 1e6)
        if case["scenes"] > 1:
            R = _rotation(rng)
            X = (X - 0.5) @ R.T + 0.5
            Q = Q @ R.T
        elif not case["fixed"]:
            X = X + rng.uniform(-0.2 / n, 0.2 / n, size=X.shape)
            Q, V = _rest(X, T)
        if case["ground"]:  # at the end of its fall, about to touch or touching
            X = X + [(s % side) * 2.0, rng.uniform(0.0, 0.03) - X[:, 1].min(), (s // side) * 2.0]
            v = np.array([0.0, -2.4, 0.0]) + rng.uniform(-0.2, 0.2, 3)
            vel = np.tile(v, (len(X), 1))
        else:
            vel = rng.uniform(-0.5, 0.5, size=X.shape)
        mass = np.bincount(T.ravel(), weights=np.repeat(0.25 * DENSITY * V, 4), minlength=len(X))
        held = np.nonzero((np.arange(len(X)) // (n + 1)) % (n + 1) == 0)[0] if case["fixed"] else np.zeros(0, np.int64)
        vel[held] = 0.0
        out.append({"n": n, "X": X, "T": T, "Q": Q, "V": V, "vel": vel, "mass": mass, "held": held,
                    "mu": E / (2 * (1 + nu)), "lam": E * nu / ((1 + nu) * (1 - 2 * nu))})
    return out


def _add_cube(ctx, b, ground=True, damping=0.0, surface=False):
    base = ctx.add_particles(b["X"], b["mass"])
    nt = len(b["T"])
    ctx.add_neo_hookean(b["T"] + base, np.full(nt, b["lam"]), np.full(nt, b["mu"]), np.full(nt, damping),
                        b["Q"].reshape(-1, 9), b["V"])
    if len(b["held"]):
        ctx.set_fixed(b["held"] + base, np.ones(len(b["held"]), np.uint8))
    if ground:
        nv = len(b["X"])
        ctx.add_ground_collision(np.arange(nv) + base, b["mass"] / DT ** 2, np.full(nv, MU_S), np.full(nv, MU_K))
    if surface:
        ctx.add_triangles(_surface(b["n"]) + base, 0)
    return base


def _context(case):
    from avbd_b200 import Context
    ctx = Context(device=torch.cuda.current_device())
    ctx.set_params(DT, GRAVITY, 1e-3)
    ctx.set_solver(case["iters"], RHO, case.get("tol", 0.0), case.get("max_iters", 0), case["precision"])
    return ctx


def _pinned(a):
    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float64)).pin_memory().numpy()


def _qmul(a, b):
    w1, x1, y1, z1 = np.moveaxis(a, -1, 0)
    w2, x2, y2, z2 = np.moveaxis(b, -1, 0)
    return np.stack([w1 * w2 - x1 * x2 - y1 * y2 - z1 * z2, w1 * x2 + x1 * w2 + y1 * z2 - z1 * y2,
                     w1 * y2 + y1 * w2 + z1 * x2 - x1 * z2, w1 * z2 + z1 * w2 + x1 * y2 - y1 * x2], axis=-1)


def _qrot(q, v):
    t = 2 * np.cross(q[..., 1:], v)
    return v + q[..., :1] * t + np.cross(q[..., 1:], t)


def _add_rods(ctx, first, q0, curvature, segments, length, radius, joint, velocity, objects):
    """Rods in lockstep: nodes along the local z axis, frames turned by the curvature; (GA, GA, EA, EI, EI, GJ)."""
    E, nu = 1e7, 0.25
    G, nr, nn = E / (2 * (1 + nu)), len(first), segments + 1
    ds = length / segments
    th = np.linalg.norm(curvature, axis=1, keepdims=True) * ds
    turn = np.concatenate([np.cos(th / 2), np.sinc(th / (2 * np.pi)) * 0.5 * ds * curvature], axis=1)
    P, Q = np.zeros((nr, nn, 3)), np.zeros((nr, nn, 4))
    p, q = first.copy(), np.broadcast_to(q0, (nr, 4)).copy()
    for k in range(nn):
        P[:, k], Q[:, k] = p, q
        p = p + _qrot(q, np.broadcast_to([0.0, 0.0, ds], (nr, 3)))
        q = _qmul(q, turn)
    area, I = np.pi * radius ** 2, np.pi * radius ** 4 / 4
    ends = np.ones(nn)
    ends[[0, -1]] = 0.5
    mass = np.tile(ends * ds * area * DENSITY, nr)
    inertia = np.tile(ends[:, None] * DENSITY * ds * np.array([I, I, 2 * I]), (nr, 1))
    base = ctx.add_oriented_particles(P.reshape(-1, 3), Q.reshape(-1, 4), mass, inertia)
    node = base + np.arange(nr * nn).reshape(nr, nn)
    seg = np.stack([node[:, :-1], node[:, 1:]], axis=-1)
    ne = nr * segments
    ctx.add_cosserat_rod(seg.reshape(-1, 2), np.tile([G * area, G * area, E * area, E * I, E * I, 2 * G * I], (ne, 1)),
                         np.full(ne, ds), np.repeat(curvature, segments, axis=0))
    if joint:
        ctx.add_one_sided_fixed_joint(node[:, 0], np.zeros((nr, 3)), np.tile([1.0, 0, 0, 0], (nr, 1)), P[:, 0], Q[:, 0])
    ctx.add_rigid_body_ground_collision(node.ravel(), np.ones(nr * nn, np.uint8), np.full(nr * nn, radius),
                                        np.tile([0.0, -radius, 0.0], (nr * nn, 1)), mass / DT ** 2,
                                        np.full(nr * nn, 0.5), np.full(nr * nn, 0.2))
    for r in range(nr):
        ctx.add_rod_segments(seg[r], radius, int(objects[r]))
    if velocity is not None:
        ctx.set_velocities(base, np.tile(velocity, (nr * nn, 1)))


def _prepare_rods(case, seed):
    rng = np.random.default_rng([seed, 2])
    ctx = _context(case)
    nr = case["rods"]
    side = math.ceil(math.sqrt(nr))
    b = rng.uniform(0.02, 0.10, nr) / (2 * np.pi)  # helices of radius 2 cm, pitch 2 to 10 cm
    a = 0.02
    curv = np.stack([a / (a * a + b * b), np.zeros(nr), b / (a * a + b * b)], axis=1)
    r = np.arange(nr)
    first = np.stack([(r % side) * 0.1, np.full(nr, 1.2), (r // side) * 0.1], axis=1)
    c = math.sqrt(0.5)
    _add_rods(ctx, first, np.array([c, c, 0, 0]), curv, case["segments"], case["segments"] * 0.01, 0.005, True, None, r)
    ns = case["spheres"]
    if ns:
        rad = rng.uniform(0.01, 0.05, ns)
        m = 4 * np.pi / 3 * rad ** 3 * DENSITY
        P = np.stack([rng.uniform(0, max(0.1, side * 0.1), ns), rad + rng.uniform(0.0, 0.02, ns),
                      side * 0.1 + 0.2 + rng.uniform(0, 1, ns)], axis=1)
        p = ctx.add_oriented_particles(P, np.tile([1.0, 0, 0, 0], (ns, 1)), m, np.repeat(0.4 * m * rad ** 2, 3).reshape(-1, 3))
        ctx.add_rigid_body_ground_collision(p + np.arange(ns), np.full(ns, 2, np.uint8), rad,
                                            np.stack([0 * rad, -rad, 0 * rad], axis=1), m / DT ** 2, np.full(ns, 0.5),
                                            np.full(ns, 0.2))
    return ctx


def _prepare_contacts(case, seed):
    rng = np.random.default_rng([seed, 3])
    ctx = _context(case)
    n, nr, length, radius = case["n"], case["rods"], 0.9, 0.01
    X, T, Q, V = _grid(n)
    E, nu = 1e6, 0.4
    mass = np.bincount(T.ravel(), weights=np.repeat(0.25 * DENSITY * V, 4), minlength=len(X))
    held = np.nonzero((np.arange(len(X)) // (n + 1)) % (n + 1) == 0)[0]
    _add_cube(ctx, {"n": n, "X": X, "T": T, "Q": Q, "V": V, "mass": mass, "held": held, "mu": E / (2 * (1 + nu)),
                    "lam": E * nu / ((1 + nu) * (1 - 2 * nu))}, ground=False, surface=True)
    z = (np.arange(nr) + 0.5) / nr + rng.uniform(-0.05, 0.05, nr) / nr
    first = np.stack([0.05 + rng.uniform(-0.02, 0.02, nr), np.full(nr, 1.0 + radius + 0.002), z], axis=1)
    c = math.sqrt(0.5)
    _add_rods(ctx, first, np.array([c, 0, c, 0]), np.zeros((nr, 3)), case["segments"], length, radius, False,
              [0.0, -0.2, 0.0], 1 + np.arange(nr))
    return ctx


def _mlp_params(seed):
    """A network as after some training: fan-in scaled layers, small biases and outputs."""
    rng = np.random.default_rng([seed, 4])
    p = np.zeros(NPARAMS, dtype=np.float32)
    at = 0
    for rows, cols, used, scale in ((MLP_HID, MLP_PAD, MLP_IN, 1.0), (MLP_HID, MLP_HID, MLP_HID, 1.0),
                                    (MLP_HID, MLP_HID, MLP_HID, 1.0), (MLP_OUT_PAD, MLP_HID, MLP_HID, 0.2)):
        live = rows if rows == MLP_HID else MLP_OUT
        w = p[at:at + rows * cols].reshape(rows, cols)
        bound = math.sqrt(6.0 / used) * scale
        w[:live, :used] = rng.uniform(-bound, bound, (live, used))
        at += rows * cols
        p[at:at + live] = rng.normal(0, 0.1, live)
        at += rows
    return p


def _rows(n, seed, k=0):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 64 + k)
    F = torch.zeros((n, MLP_PAD), dtype=torch.bfloat16, device="cuda")
    F[:, :MLP_IN] = torch.randn((n, MLP_IN), generator=g, device="cuda").to(torch.bfloat16)
    return F, g


def _batches(case, seed):
    out = []
    for k in range(case["steps"]):
        F, g = _rows(case["batch"], seed, k)
        T = torch.randn((case["batch"], 4), generator=g, device="cuda")
        T[:, 3] = torch.rand(case["batch"], generator=g, device="cuda") + 0.5
        out.append((F, T))
    return out


def prepare(case, seed):
    kind = case["kind"]
    if kind == "mlp":
        from avbd_b200 import warmstart
        return {"kind": kind, "net": warmstart.MLP(_mlp_params(seed)), "F": _rows(case["rows"], seed)[0]}
    if kind == "train":
        from avbd_b200 import warmstart
        return {"kind": kind, "trainer": warmstart.Trainer(case["batch"], _mlp_params(seed)),
                "batches": _batches(case, seed)}
    # an FP32 or MIXED context's results carry single precision: they are kept as such, FP64's as they come
    state = {"kind": kind, "steps": case["steps"],
             "type": torch.float64 if case["precision"] == "fp64" else torch.float32}
    if kind == "tets":
        ctx = _context(case)
        scenes = _tet_inputs(case, seed)
        for s, b in enumerate(scenes):
            if s:
                ctx.begin_scene()
            _add_cube(ctx, b, case["ground"], case["damping"], case["surface"])
        ctx.finalize()
        if case["learned"]:
            from avbd_b200 import warmstart
            ctx.set_warmstart(2, warmstart.load_params())
        state["x0"] = _pinned(np.concatenate([b["X"] for b in scenes]))
        state["v0"] = _pinned(np.concatenate([b["vel"] for b in scenes]))
    else:
        ctx = _prepare_rods(case, seed) if kind == "rods" else _prepare_contacts(case, seed)
        ctx.finalize()
    n = ctx.num_particles
    state.update(ctx=ctx, x=_pinned(np.zeros((n, 3))), v=_pinned(np.zeros((n, 3))), q=_pinned(np.zeros((n, 4))))
    return state


# ------------------------------------------------------------------ one pass
def run(state):
    kind = state["kind"]
    if kind == "mlp":
        return state["net"].forward(state["F"])
    if kind == "train":
        tr = state["trainer"]
        loss = [tr.step(F, T, 1e-3) for F, T in state["batches"]]
        return {"loss": torch.tensor(loss), "params": torch.from_numpy(tr.params())}
    ctx = state["ctx"]
    if kind == "tets":  # a frame from given positions and velocities
        ctx.set_positions(0, state["x0"])
        ctx.set_state(velocities=state["v0"])
    ctx.step(state["steps"])
    out = {"x": ctx.positions(out=state["x"])}
    if kind == "tets":
        out["v"] = ctx.velocities(out=state["v"])
    else:
        out["q"] = ctx.rotations(out=state["q"])
    return {k: torch.from_numpy(a).to(state["type"]) for k, a in out.items()}


# ------------------------------------------------------------------ the work of a pass
def work(case):
    kind = case["kind"]
    if kind == "mlp":
        f = 2.0 * (MLP_IN * MLP_HID + 2 * MLP_HID * MLP_HID + MLP_HID * MLP_OUT)
        return {"bytes": case["rows"] * (2.0 * MLP_PAD + 4 * MLP_OUT_PAD) + 2.0 * NPARAMS, "flops": f * case["rows"]}
    if kind == "train":
        f = 6.0 * (MLP_IN * MLP_HID + 2 * MLP_HID * MLP_HID + MLP_HID * MLP_OUT)
        n = case["batch"] * case["steps"]
        return {"bytes": n * (2.0 * MLP_PAD + 16) + case["steps"] * 24.0 * NPARAMS, "flops": f * n}
    real = 4.0 if case["precision"] == "fp32" else 8.0
    if kind == "tets":
        cells = _cells(case)
        nv, nt = sum((n + 1) ** 3 for n in cells), 6.0 * sum(n ** 3 for n in cells)
        iters = (case["max_iters"] if case["tol"] else case["iters"]) * case["steps"]
        if case["tol"]:
            iters *= 0.6  # scenes of this range that stop before the cap
        # rest shape and material of each tet, state and contact of each vertex, positions and velocities in and out
        b = nt * (16 + 12 * (4.0 if real == 4.0 or case["precision"] == "mixed" else 8.0)) + nv * (20 * real + 96)
        return {"bytes": b, "flops": iters * (4 * nt * 40 + nv * 80)}
    if kind == "contacts":
        nv, nt = (case["n"] + 1) ** 3, 6.0 * case["n"] ** 3
    else:
        nv = nt = 0.0
    no = case["rods"] * (case["segments"] + 1) + case.get("spheres", 0)
    ne = case["rods"] * case["segments"]
    iters = case["iters"] * case["steps"]
    return {"bytes": nt * 64 + nv * 20 * real + no * 60 * real + ne * 14 * real + (nv + no) * 56,
            "flops": iters * (4 * nt * 40 + nv * 80 + ne * 2 * 1500.0 + no * 400.0)}


# ------------------------------------------------------------------ the same in 64 bits
@functools.lru_cache(maxsize=None)
def _colors(n):
    """DSATUR over the grid's vertices: most colors among the neighbours, then most neighbours, then lowest index."""
    T = _grid(n)[1]
    e = np.concatenate([T[:, [a, b]] for a in range(4) for b in range(4) if a != b])
    e = np.unique(e, axis=0)
    nv = (n + 1) ** 3
    off = np.searchsorted(e[:, 0], np.arange(nv + 1)).tolist()
    nbr = e[:, 1].tolist()
    color, seen = [-1] * nv, [0] * nv  # seen: bit set of the neighbours' colors
    heap = [(0, off[v] - off[v + 1], v) for v in range(nv)]
    heapq.heapify(heap)
    while heap:
        s, _, v = heapq.heappop(heap)
        if color[v] >= 0 or -s != bin(seen[v]).count("1"):
            continue
        free = ~seen[v]
        c = (free & -free).bit_length() - 1
        color[v] = c
        for w in nbr[off[v]:off[v + 1]]:
            if color[w] < 0 and not seen[w] >> c & 1:
                seen[w] |= 1 << c
                heapq.heappush(heap, (-bin(seen[w]).count("1"), off[w] - off[w + 1], w))
    return np.array(color)


def _exact_tets(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    scenes = _tet_inputs(case, seed)
    base = np.cumsum([0] + [len(b["X"]) for b in scenes])
    nv, S = int(base[-1]), len(scenes)
    t64 = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=dev)  # noqa: E731
    t32 = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.int64, device=dev)  # noqa: E731
    T = t32(np.concatenate([b["T"] + o for b, o in zip(scenes, base)]))
    Q = t64(np.concatenate([b["Q"] for b in scenes]))
    D = torch.cat([Q, -Q.sum(1, keepdim=True)], dim=1)
    V = t64(np.concatenate([b["V"] for b in scenes]))
    per = lambda key: t64(np.concatenate([np.full(len(b["T"]), b[key]) for b in scenes]))  # noqa: E731
    lam, mu = per("lam"), per("mu")
    color = np.concatenate([_colors(b["n"]) for b in scenes])
    free = np.ones(nv, bool)
    for b, o in zip(scenes, base):
        free[b["held"] + o] = False
    x, v = t64(np.concatenate([b["X"] for b in scenes])), t64(np.concatenate([b["vel"] for b in scenes]))
    m = t64(np.concatenate([b["mass"] for b in scenes]))
    scene = t32(np.repeat(np.arange(S), np.diff(base)))
    fr = torch.as_tensor(free, device=dev)
    mg = torch.zeros(S, dtype=torch.float64, device=dev).index_add_(0, scene, torch.where(fr, m * m, 0 * m)).sqrt() * GRAVITY
    others = ((1, 2, 3), (0, 2, 3), (0, 1, 3), (0, 1, 2))
    tc = torch.as_tensor(color, device=dev)[T]
    inc = []  # per color: the vertices of the color, then their incidences
    for c in range(int(color.max()) + 1):
        ids = torch.as_tensor(np.nonzero((color == c) & free)[0], device=dev)
        slot = torch.full((nv,), -1, dtype=torch.int64, device=dev)
        slot[ids] = torch.arange(len(ids), device=dev)
        te, lo = torch.nonzero((tc == c) & fr[T], as_tuple=True)
        oth = torch.tensor(others, device=dev)[lo]
        inc.append({"ids": ids, "slot": slot[T[te, lo]], "i": T[te, lo], "o": T[te[:, None], oth], "d": D[te[:, None], oth],
                    "dw": D[te, lo], "t": te})
    k0 = (m / DT ** 2)[:, None].expand(nv, 3).clone()
    k, gl = k0.clone(), torch.zeros((nv, 3), dtype=torch.float64, device=dev)
    cprev, static = torch.zeros(nv, dtype=torch.float64, device=dev), torch.zeros(nv, dtype=torch.bool, device=dev)
    unclamped, cp = static.clone(), torch.zeros((nv, 2), dtype=torch.float64, device=dev)
    kd = case["damping"]
    mu_s, mu_k = t64(MU_S), t64(MU_K)

    def strain(xa):
        F = torch.einsum("tka,tkb->tab", xa[T] - xa[T[:, 3:4]], D)
        return 0.5 * (F.transpose(1, 2) @ F - torch.eye(3, dtype=torch.float64, device=dev))

    def block(p, xa):
        """Gradient and Hessian of the color's vertices."""
        e = xa[p["o"]] - xa[p["i"]][:, None]
        F = torch.einsum("tka,tkb->tab", e, p["d"])
        c0, c1, c2 = torch.cross(F[:, :, 1], F[:, :, 2], dim=1), torch.cross(F[:, :, 2], F[:, :, 0], dim=1), torch.cross(F[:, :, 0], F[:, :, 1], dim=1)
        J = (F[:, :, 0] * c0).sum(1)
        dw, t = p["dw"], p["t"]
        Fc = dw[:, :1] * c0 + dw[:, 1:2] * c1 + dw[:, 2:] * c2
        Fd = torch.einsum("tab,tb->ta", F, dw)
        vl, vm, q2 = V[t] * lam[t], V[t] * mu[t], (dw * dw).sum(1)
        eye = torch.eye(3, dtype=torch.float64, device=dev)
        g = (vl * (J - 1 - mu[t] / lam[t]))[:, None] * Fc + vm[:, None] * Fd
        H = vl[:, None, None] * Fc[:, :, None] * Fc[:, None, :] + (vm * q2)[:, None, None] * eye
        if kd:
            Ed = ((0.5 * (F.transpose(1, 2) @ F - eye) - Eprev[t]) / DT @ dw[:, :, None])[:, :, 0]
            w = 2 * V[t] * kd / DT
            g = g + w[:, None] * torch.einsum("tab,tb->ta", F, Ed)
            H = H + (w * (dw * Ed).sum(1))[:, None, None] * eye + (0.5 * w / DT)[:, None, None] * (
                F @ F.transpose(1, 2) * q2[:, None, None] + Fd[:, :, None] * Fd[:, None, :])
        n = len(p["ids"])
        G = torch.zeros((n, 3), dtype=torch.float64, device=dev).index_add_(0, p["slot"], g)
        HH = torch.zeros((n, 3, 3), dtype=torch.float64, device=dev).index_add_(0, p["slot"], H)
        i = p["ids"]
        if case["ground"]:
            xi = xa[i]
            ln = (k[i, 0] * (-xi[:, 1] - 0.95 * cprev[i]) + gl[i, 0]).clamp(min=0)
            lt, lb = k[i, 1] * (xi[:, 0] - cp[i, 0]) + gl[i, 1], k[i, 2] * (xi[:, 2] - cp[i, 1]) + gl[i, 2]
            mag = (lt * lt + lb * lb).sqrt()
            mx = torch.where(static[i], mu_s, mu_k) * ln
            sc = torch.where(mag > mx, mx / (mag + 1e-8), torch.ones_like(mag))
            G = G + torch.stack([lt * sc, -ln, lb * sc], dim=1)
            HH = HH + torch.diag_embed(torch.stack([k[i, 1], k[i, 0], k[i, 2]], dim=1))
        cm = m[i] / DT ** 2
        return cm[:, None] * (xa[i] - y[i]) + G, HH + cm[:, None, None] * eye

    xp, vp = x.clone(), torch.zeros_like(v)
    gvec = torch.tensor([0.0, -GRAVITY, 0.0], dtype=torch.float64, device=dev)
    Eprev = None
    for _ in range(case["steps"]):
        if kd:
            Eprev = strain(xp)
        if case["ground"]:
            cp = x[:, [0, 2]].clone()
            cprev = torch.where(gl[:, 0] > 0, -x[:, 1], cprev)
            static = static | unclamped
            gl = gl * torch.tensor([0.95 * 0.99, 0.99, 0.99], dtype=torch.float64, device=dev)
            k = torch.maximum(0.99 * k, k0)
        al = ((v - vp) / DT) @ gvec / GRAVITY
        at = (al / GRAVITY).clamp(0, 1)[:, None] * gvec
        y = torch.where(fr[:, None], x + DT * v + DT * DT * gvec, x)
        x = torch.where(fr[:, None], x + (DT * v + DT * DT * at), x)
        hist = [x.clone(), x.clone()]
        active = torch.ones(S, dtype=torch.bool, device=dev)
        om = 1.0
        n_it = (case["max_iters"] if case["tol"] else case["iters"])
        for it in range(n_it):
            om = 4 / (4 - RHO * RHO * om) if it > 2 else 2 / (2 - RHO * RHO) if it == 2 else 1.0
            r2 = torch.zeros(S, dtype=torch.float64, device=dev)
            for p in inc:
                G, H = block(p, x)
                r2.index_add_(0, scene[p["ids"]], (G * G).sum(1))
                dx = -torch.linalg.solve(H, G[:, :, None])[:, :, 0]
                live = active[scene[p["ids"]]][:, None]
                x = x.index_copy(0, p["ids"], torch.where(live, x[p["ids"]] + dx, x[p["ids"]]))
            on = active[scene]
            h = hist[it & 1]
            xn = torch.where(on[:, None], om * (x - h) + h, x)
            hist[it & 1] = torch.where(on[:, None], xn, h)
            x = xn
            if case["ground"]:
                cc = -x[:, 1] - 0.95 * cprev
                ct, cb = x[:, 0] - cp[:, 0], x[:, 2] - cp[:, 1]
                ln, lt, lb = k[:, 0] * cc + gl[:, 0], k[:, 1] * ct + gl[:, 1], k[:, 2] * cb + gl[:, 2]
                mag = (lt * lt + lb * lb).sqrt()
                l0 = ln.clamp(min=0)
                stick = mag < torch.where(static, mu_s, mu_k) * l0
                slide = torch.where(static, mu_k * ln, mu_k * l0) / (mag + 1e-8)
                kn = torch.stack([torch.where(ln > 0, k[:, 0] + 10.0 * cc.abs(), k[:, 0]),
                                  torch.where(stick, k[:, 1] + 10.0 * ct.abs(), k[:, 1]),
                                  torch.where(stick, k[:, 2] + 10.0 * cb.abs(), k[:, 2])], dim=1)
                gn = torch.stack([l0, torch.where(stick, lt, lt * slide), torch.where(stick, lb, lb * slide)], dim=1)
                k, gl = torch.where(on[:, None], kn, k), torch.where(on[:, None], gn, gl)
                unclamped = torch.where(on, stick, unclamped)
                static = torch.where(on, static & stick, static)
            if case["tol"]:
                cand = active & (r2.sqrt() <= case["tol"] * mg)
                if bool(cand.any()):
                    ex = torch.zeros(S, dtype=torch.float64, device=dev)
                    for p in inc:
                        G, _ = block(p, x)
                        ex.index_add_(0, scene[p["ids"]], (G * G).sum(1))
                    active = active & ~(cand & (ex.sqrt() <= case["tol"] * mg))
                if not bool(active.any()):
                    break
        vp, v, xp = v, (x - xp) / DT, x.clone()
    return {"v": v.cpu(), "x": x.cpu()}


def _exact_net(p):
    p = torch.as_tensor(p, dtype=torch.float64)
    at, out = 0, []
    for rows, cols in ((MLP_HID, MLP_PAD), (MLP_HID, MLP_HID), (MLP_HID, MLP_HID), (MLP_OUT_PAD, MLP_HID)):
        out += [p[at:at + rows * cols].reshape(rows, cols), p[at + rows * cols:at + rows * cols + rows]]
        at += rows * cols + rows
    return out


def _exact_forward(net, F):
    h = F
    for i in range(4):
        z = h @ net[2 * i].T + net[2 * i + 1]
        h = z * torch.sigmoid(z) if i < 3 else z
    return h


def exact(case, seed):
    kind = case["kind"]
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if kind == "mlp":
        net = [w.to(dev) for w in _exact_net(_mlp_params(seed))]
        F = _rows(case["rows"], seed)[0].double()
        return torch.cat([_exact_forward(net, f) for f in F.split(131072)])
    if kind == "train":
        net = [w.to(dev).requires_grad_() for w in _exact_net(_mlp_params(seed))]
        opt = torch.optim.Adam(net, lr=1e-3, betas=(0.9, 0.999), eps=1e-8)
        loss = []
        for F, T in _batches(case, seed):
            T = T.double()
            e = _exact_forward(net, F.double())[:, :MLP_OUT] - T[:, :MLP_OUT]
            L = (T[:, 3:] * e * e).mean()
            opt.zero_grad()
            L.backward()
            opt.step()
            loss.append(float(L))
        return {"loss": torch.tensor(loss, dtype=torch.float64),
                "params": torch.cat([w.detach().reshape(-1) for w in net]).cpu()}
    if kind == "tets" and not case["learned"]:
        return _exact_tets(case, seed)
    # rods, contacts and the learned warm start (whose network runs in BF16) have no plain 64-bit restatement here
    return None
