"""Performance cases of the MLS-MPM forward + adjoint engine.

Each case is a piece of work that a program using this package asks of it
through its public entry points (dmpm.Context, dmpm.Batch and the mesh and
surface functions): whole gradient evaluations over the range of scene sizes,
precisions and options that the package's own benchmark and tests use, single
time steps on the reference's point structs, batches of scenes, and the scene
setup and export functions.  Scenes are the package's seeded synthetic ones
(scenes.py).

Inputs are float32-representable and dt, drag, smoothing and the forces are
too, so that the float32 and the float64 engine compute from the same values
as exact(), which restates the whole rollout, loss and adjoint in torch
float64.  The float32 engine hands its results back in double arrays; the
cases narrow them to float32, as a program that feeds a float32 optimiser
does.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

_REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(_REPO, "a-differentiable-material-point-method-for-shape-morphing_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import dmpm  # noqa: E402
import optinput  # noqa: E402
import scenes  # noqa: E402

_MASS_EPS = 1.1920928955078125e-07  # node-mass threshold of the grid update
_DEV = "cuda"


# ---------------------------------------------------------------- the cases
def _gradient(name=None, shape="sphere", size=0.2, res=32, dims="", ppc=2, steps=10, precision="fp32",
              adjoint="exact", control="tied", checkpoint=1, stride=0, deterministic=False, shuffled=False,
              smoothing=0.0, drag=0.0):
    c = dict(kind="gradient", shape=shape, size=size, res=res, dims=dims, ppc=ppc, steps=steps,
             precision=precision, adjoint=adjoint, control=control, checkpoint=checkpoint, stride=stride,
             deterministic=deterministic, shuffled=shuffled, smoothing=smoothing, drag=drag)
    return dict(c, name=name) if name else c


def listed():
    return [
        # One time step of a small cloud held in the reference's point structs, in and out: what
        # SingleThreadMPM::ForwardTimeStep callers do per frame.  The smallest call; latency counts.
        {"name": "step_small", "kind": "step", "size": 0.2, "res": 12, "dims": "", "ppc": 2,
         "precision": "fp32"},
        # The small benchmark scene (sphere to cube, 32^3, 8.8k particles, 100 steps), per-layer
        # controls: a graph of short launches.
        _gradient("grad_small", size=0.2, res=32, steps=100, control="per_layer"),
        # CompGraph as the reference's callers use it: point structs up, forward, loss, the
        # reference's own adjoint (the default mode), layer 0's structs with their gradients back.
        # A non-cubic grid, drag and smoothing as the reference sets them by default.
        {"name": "compgraph_refcompat", "kind": "compgraph", "shape": "ellipsoid", "size": 1.0, "res": 64,
         "dims": "64x60x53", "ppc": 2, "steps": 10, "precision": "fp32", "smoothing": 0.125,
         "drag": 0.5},
        # The headline benchmark: ellipsoid to torus, 64^3, 267k particles, 200 steps.
        _gradient("grad_headline", shape="ellipsoid", size=1.0, res=64, ppc=3, steps=200),
        # A long rollout's storage policy: checkpointed layers, control frames every 10 layers, the
        # cloud handed over in random order and stored in cell order by the engine.
        _gradient("grad_checkpointed", shape="spheres3", size=0.75, res=128, steps=50, control="per_layer",
                  checkpoint=25, stride=10, shuffled=True),
        # Reproducible gradients (integer node sums) on the headline shape at 8 particles per cell.
        _gradient("grad_deterministic", shape="ellipsoid", size=1.0, res=64, steps=40, deterministic=True),
        # The float64 engine, which the finite-difference checks and stiff rollouts use.
        _gradient("grad_fp64", shape="ellipsoid", size=0.9, res=64, steps=20, precision="fp64",
                  control="per_layer"),
        # Many scenes of mixed size advanced together (hyper-parameter and shape sweeps).
        {"name": "batch_mixed", "kind": "batch", "count": 12, "nmin": 5000, "nmax": 60000, "smin": 20, "smax": 60},
        # The largest grid of the benchmark (256^3) with a 2M-particle sphere.
        _gradient("grad_large_grid", size=0.1535, res=256, steps=10, control="per_layer"),
        # Scene setup: the reference's lattice point cloud of a watertight mesh of about 1,150 faces.
        {"name": "mesh_points", "kind": "mesh", "around": 48, "along": 12, "point_dx": 29 / 4096},
        # Export: sphere-union field of a morphed cloud and its isosurface.
        {"name": "surface", "kind": "surface", "points": 300000, "radius": 0.025, "grid_dx": 13 / 1024, "blur": 2},
        # Export: node masses of a cloud and their interpolation onto a finer grid.
        {"name": "mass_field", "kind": "mass", "points": 1000000, "grid_dx": 0.02, "quality": 2},
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    """One more case of the ranges that listed() stands for."""
    kind = rng.choice(["gradient", "gradient", "gradient", "gradient", "fp64", "deterministic", "checkpointed", "step",
                       "compgraph", "batch", "mesh", "surface", "mass"])
    if kind == "step":
        return {"kind": "step", "size": round(_log_uniform(rng, 0.12, 0.3), 4), "res": rng.randint(9, 48),
                "dims": "", "ppc": 2, "precision": rng.choice(["fp32", "fp32", "fp64"])}
    if kind == "batch":
        lo = int(_log_uniform(rng, 2000, 10000))
        return {"kind": "batch", "count": rng.randint(3, 16), "nmin": lo, "nmax": int(lo * rng.uniform(1.5, 6)),
                "smin": rng.randint(5, 15), "smax": rng.randint(16, 50)}
    if kind == "mesh":
        return {"kind": "mesh", "around": rng.randint(12, 60), "along": rng.randint(6, 16),
                "point_dx": round(_log_uniform(rng, 37, 240)) / 4096}
    if kind == "surface":
        dx = round(_log_uniform(rng, 13, 50)) / 1024
        return {"kind": "surface", "points": int(_log_uniform(rng, 3000, 400000)), "blur": rng.randint(0, 4),
                "radius": round(dx * rng.uniform(1.0, 2.2), 5), "grid_dx": dx}
    if kind == "mass":
        return {"kind": "mass", "points": int(_log_uniform(rng, 3000, 1000000)), "quality": rng.randint(1, 3),
                "grid_dx": round(_log_uniform(rng, 0.03, 0.1), 5)}
    shape = rng.choice(["sphere", "ellipsoid", "box"])
    res = rng.choice([20, 27, 32, 41, 48, 57, 64, 75, 96])
    size = round(_log_uniform(rng, 0.55, 1.0) * {"sphere": 0.25, "ellipsoid": 1.0, "box": 0.2}[shape], 4)
    ppc = rng.choice([2, 2, 3])
    dims = rng.choice(["", "", "%dx%dx%d" % (res, res - rng.randint(0, 3), res + rng.randint(0, 3))])
    # particles of the shape, and no more particle steps than a quarter of the headline's
    frac = {"sphere": 4.19 * size ** 3, "ellipsoid": 0.0377 * size ** 3, "box": 8 * size ** 3}[shape]
    n = frac * res ** 3 * ppc ** 3
    most = 13e6 / max(n, 500.0)
    if kind == "compgraph":
        return {"kind": "compgraph", "shape": shape, "size": size, "res": res, "dims": dims, "ppc": ppc,
                "steps": int(_log_uniform(rng, 2, 12)), "precision": rng.choice(["fp32", "fp32", "fp64"]),
                "smoothing": rng.choice([0.0, 0.125]), "drag": rng.choice([0.0, 0.5])}
    steps = max(2, int(_log_uniform(rng, 4, min(100.0, max(6.0, most)))))
    c = _gradient(shape=shape, size=size, res=res, dims=dims, ppc=ppc, steps=steps,
                  control=rng.choice(["tied", "per_layer"]), shuffled=rng.random() < 0.2,
                  smoothing=rng.choice([0.0, 0.0, 0.0625]), drag=rng.choice([0.0, 0.25]))
    if kind == "fp64":
        c.update(precision="fp64", shuffled=False, steps=max(2, min(steps, int(most / 4))))
    elif kind == "deterministic":
        c["deterministic"] = True
    elif kind == "checkpointed":
        c.update(checkpoint=rng.randint(2, 9), stride=rng.choice([0, 3]), control="per_layer")
    return c


# ---------------------------------------------------------------- scenes
def _shapes(case):
    """(shape, its bounding box, target, its bounding box) in the unit box."""
    c, s = (0.5, 0.5, 0.5), case.get("size", 0.2)
    bb = scenes._bb
    kind = case.get("shape", "sphere")
    if kind == "sphere":
        return scenes.sphere(c, s), bb(c, s), scenes.cube(c, 1.6 * s), bb(c, 0.8 * s)
    if kind == "ellipsoid":
        ax = tuple(s * a for a in (0.3, 0.2, 0.15))
        return (scenes.ellipsoid(c, ax), bb(c, ax), scenes.torus(c, 0.25 * s, 0.08 * s),
                bb(c, (0.33 * s, 0.33 * s, 0.08 * s)))
    if kind == "box":
        return (scenes.box(c, s), bb(c, s), scenes.box(c, (1.2 * s, 0.8 * s, s)), bb(c, (1.2 * s, 0.8 * s, s)))
    rng = np.random.default_rng(2007)
    cs = rng.uniform(0.3, 0.7, size=(3, 3))
    rs = s * rng.uniform(0.14, 0.2, size=3)
    lo, hi = np.min(cs - rs[:, None], 0), np.max(cs + rs[:, None], 0)
    return (scenes.union(*[scenes.sphere(cs[k], rs[k]) for k in range(3)]), (lo, hi), scenes.capsule(c, 0.5, 0.15),
            bb(c, (0.4, 0.15, 0.15)))


def _scene(case, seed, v_std=0.0):
    """A seeded scene with float32-representable inputs, its volumes and its target's node masses.
    The sub-cells whose centres lie in the shape hold one jittered particle each, so that the
    particle count is the case's and not the seed's."""
    rng = np.random.default_rng(seed + 17)
    shp, box, tgt, tbox = _shapes(case)
    dims = tuple(int(d) for d in case["dims"].split("x")) if case.get("dims") else None
    sc = scenes.make_scene("case", shp, tgt, case["res"], case["ppc"], 1e4, 0.3, 5e-4, case.get("steps", 1), seed,
                           drag=case.get("drag", 0.0), smoothing=case.get("smoothing", 0.0),
                           dfc_std=0.0, bbox=box, target_bbox=tbox, dims=dims)
    sc.x = scenes.sample_points(shp, case["res"], case["ppc"], None, box)
    n = len(sc.x)
    # the material, density and time step of the reference's default input file
    opt = optinput.OptInput()
    sc.target_mp = opt.p_density / case["ppc"] ** 3
    sc.x = sc.x + (rng.random(sc.x.shape) - 0.5) / case["ppc"]
    sc.m, sc.lam, sc.mu = (np.full(n, a) for a in (sc.target_mp, opt.lam, opt.mu))
    sc.v, sc.C, sc.vol = np.zeros((n, 3)), np.zeros((n, 3, 3)), np.zeros(n)
    sc.F = np.broadcast_to(np.eye(3), (n, 3, 3)).copy()
    sc.dFc = rng.normal(0.0, 1e-3, size=(n, 3, 3))
    sc.dt = float(np.float32(opt.dt))
    sc.f_ext = np.array([0.0, -1.0, 0.0])
    if v_std:
        sc.v = rng.normal(0.0, v_std, size=(sc.n, 3))
    if case.get("shuffled"):
        p = rng.permutation(sc.n)
        for k in ("x", "v", "F", "C", "dFc", "m", "lam", "mu"):
            setattr(sc, k, np.ascontiguousarray(getattr(sc, k)[p]))
    sc = sc.float32_inputs()
    sc.vol, sc.target = _volumes_and_target(sc)
    return sc


def _round(t):
    return t.to(torch.float32).to(torch.float64)


def _volumes_and_target(sc):
    f = lambda a: torch.as_tensor(a, dtype=torch.float64, device=_DEV)  # noqa: E731
    g = _Geo(sc)
    x, m = f(sc.x), f(sc.m)
    mass = _raster(g, x, m)
    vol = torch.zeros_like(m)
    for a, b in _chunks(len(m)):
        ids, ok, w, _, _ = g.stencil(x[a:b])
        mg = (w * mass[ids] * ok).sum(1)
        vol[a:b] = torch.where(mg.abs() > _MASS_EPS, m[a:b] / mg, torch.zeros_like(mg))
    tp = f(np.asarray(sc.target_points, dtype=np.float32))
    target = _raster(g, tp, torch.full((len(tp),), sc.target_mp, dtype=torch.float64, device=_DEV))
    return _round(vol).cpu().numpy(), _round(target).cpu().numpy()


_FIELDS = {"x": (0, 3), "v": (3, 6), "F": (6, 15), "C": (15, 24), "material": (33, 37), "dFc": (37, 46),
           "dLdx": (46, 49), "dLdv": (49, 52), "dLdF": (52, 61), "dLdC": (61, 70)}


def _fields(p):
    """The fields of an array of point structs that the engine fills, as views."""
    return {k: p[:, a:b] for k, (a, b) in _FIELDS.items()}


def _points_ref(sc):
    """The scene's cloud as the reference's 118-float point structs."""
    p = np.zeros((sc.n, 118), dtype=np.float32)
    cm = scenes.to_colmajor
    for off, a in ((0, sc.x), (3, sc.v), (6, cm(sc.F)), (15, cm(sc.C)), (37, cm(sc.dFc))):
        p[:, off: off + a.shape[1]] = a
    for off, a in ((33, sc.m), (34, sc.vol), (35, sc.lam), (36, sc.mu)):
        p[:, off] = a
    return p


# ---------------------------------------------------------------- prepare and run
def _context(case, sc, **kw):
    c = dmpm.Context(case.get("precision", "fp32"))
    c.set_grid(sc.dims, sc.dx, sc.min_point)
    c.set_params(dt=sc.dt, drag=sc.drag, f_ext=sc.f_ext, smoothing=sc.smoothing, **kw)
    return c


def prepare(case, seed):
    kind = case["kind"]
    if kind == "mesh":
        V, F = _torus_mesh(case, seed)
        return {"kind": kind, "case": case, "V": V, "F": F}
    if kind == "surface":
        return {"kind": kind, "case": case, "points": _surface_cloud(case, seed)}
    if kind == "mass":
        return {"kind": kind, "case": case, "points": _torus_cloud(case["points"], seed)}
    if kind == "batch":
        return _prepare_batch(case, seed)
    if kind in ("step", "compgraph"):
        sc = _scene(case, seed, v_std=0.3 if kind == "step" else 0.0)
        c = _context(case, sc, adjoint="refcompat")
        c.set_target_mass(sc.target)
        pts = _points_ref(sc)
        return {"kind": kind, "ctx": c, "points": pts, "out": np.zeros_like(pts), "layers": case.get("steps", 1) + 1}
    sc = _scene(case, seed)
    c = _context(case, sc, adjoint=case["adjoint"], control=case["control"], checkpoint_every=case["checkpoint"],
                 control_stride=case["stride"], deterministic=case["deterministic"],
                 reorder_particles=case["shuffled"])
    c.set_particles(sc.x, sc.m, sc.lam, sc.mu, v=sc.v, F=sc.F, C=sc.C, dFc=sc.dFc, vol=sc.vol)
    c.set_target_mass(sc.target)
    c.setup(sc.steps + 1)
    # the control gradient is read into pinned memory, column-major 3x3 matrices
    return {"kind": kind, "ctx": c, "grad": torch.empty(sc.n * 9, dtype=torch.float64, pin_memory=True),
            "narrow": case["precision"] == "fp32"}


def run(state):
    kind = state["kind"]
    if kind == "gradient":
        c = state["ctx"]
        c.forward(0)
        loss = c.loss()
        c.backward(0)
        g = c.control_grad(0, out=state["grad"])
        return {"loss": np.float32(loss), "grad": g.to(torch.float32)} if state["narrow"] else {"loss": loss, "grad": g}
    if kind == "step":
        c = state["ctx"]
        c.set_points_ref(state["points"])
        c.setup(2)
        c.forward(0)
        return _fields(c.get_points_ref(1, state["out"]))
    if kind == "compgraph":
        c = state["ctx"]
        c.set_points_ref(state["points"])
        c.setup(state["layers"])
        c.forward(0)
        loss = c.loss()
        c.backward(0)
        return {"loss": np.float32(loss), **_fields(c.get_points_ref(0, state["out"]))}
    if kind == "batch":
        b = state["batch"]
        losses = b.gradient()
        return {"losses": losses.astype(np.float32),
                "grads": [b.control_grad(i).astype(np.float32) for i in range(b.count)]}
    case = state["case"]
    if kind == "mesh":
        return dmpm.mesh_lattice_points(state["V"], state["F"], case["point_dx"])
    mn, mx = (-1.0, -1.0, -1.0), (1.0, 1.0, 1.0)
    if kind == "surface":
        return dmpm.sphere_union_surface(state["points"], case["radius"], case["grid_dx"], 0.5 * case["radius"],
                                         case["blur"], mn, mx)
    dims = dmpm.surface_grid_dims(mn, mx, case["grid_dx"])
    coarse = dmpm.p2g_mass(state["points"], 1.0, dims, case["grid_dx"], mn)
    q = case["quality"]
    fine = dmpm.g2g_mass(coarse, dims, case["grid_dx"], mn, tuple(d * q for d in dims), case["grid_dx"] / q, mn)
    return {"coarse": coarse, "fine": fine}


# instances of a batch: spheres, ellipsoids and boxes of log-uniform particle counts
def _batch_cases(case):
    out = []
    for i in range(case["count"]):
        rng = np.random.default_rng(1000 * case["nmin"] + i)
        res = int(rng.choice([32, 64]))
        n = math.exp(rng.uniform(math.log(case["nmin"]), math.log(case["nmax"])))
        shape = ["sphere", "ellipsoid", "box"][int(rng.integers(0, 3))]
        ppc = 2 if n / 8 <= 0.1 * res ** 3 else 3
        frac = n / (ppc ** 3 * res ** 3)
        size = (frac / {"sphere": 4.19, "ellipsoid": 0.0377, "box": 8.0}[shape]) ** (1 / 3)
        size = min(size, {"sphere": 0.35, "ellipsoid": 1.25, "box": 0.3}[shape])
        out.append({"shape": shape, "size": size, "res": res, "ppc": ppc,
                    "steps": int(rng.integers(case["smin"], case["smax"] + 1))})
    return out


def _batch_scenes(case, seed):
    return [_scene(c, 1000 * seed + i) for i, c in enumerate(_batch_cases(case))]


def _prepare_batch(case, seed):
    scs = _batch_scenes(case, seed)
    b = dmpm.Batch([{"n": s.n, "dims": s.dims, "dx": s.dx, "min_point": tuple(s.min_point), "steps": s.steps}
                    for s in scs])
    b.set_params(scs[0].dt, f_ext=scs[0].f_ext, adjoint="exact")
    for i, s in enumerate(scs):
        b.set_particles(i, s.x, s.m, s.lam, s.mu, v=s.v, F=s.F, C=s.C, dFc=s.dFc, vol=s.vol)
        b.set_target_mass(i, s.target)
    b.set_launch(use_graph=True)
    b.setup()
    return {"kind": "batch", "batch": b}


def _rotation(rng):
    q, r = np.linalg.qr(rng.normal(size=(3, 3)))
    q = q * np.sign(np.diag(r))
    return q if np.linalg.det(q) > 0 else q[:, ::-1]


def _torus_mesh(case, seed):
    """A watertight, outward-oriented torus mesh, tilted: around x along quads, split.  The seed
    places it.  Vertices, spacing and place are multiples of a power of two, so that the lattice
    moves with the mesh without rounding and every place keeps the same number of points."""
    rng = np.random.default_rng(7)
    R, r = 0.42 * rng.uniform(0.95, 1.05), 0.16 * rng.uniform(0.9, 1.1)
    nu, nv = case["around"], case["along"]
    u, v = np.meshgrid(2 * np.pi * np.arange(nu) / nu, 2 * np.pi * np.arange(nv) / nv, indexing="ij")
    P = np.stack([(R + r * np.cos(v)) * np.cos(u), (R + r * np.cos(v)) * np.sin(u), r * np.sin(v)], -1).reshape(-1, 3)
    place = np.random.default_rng(seed + 3).integers(-512, 513, size=3) / 1024.0
    V = (np.round(P @ _rotation(rng).T * 65536.0) / 65536.0 + place).astype(np.float32)
    i, j = np.meshgrid(np.arange(nu), np.arange(nv), indexing="ij")
    a, b = i * nv + j, ((i + 1) % nu) * nv + j
    c, d = ((i + 1) % nu) * nv + (j + 1) % nv, i * nv + (j + 1) % nv
    F = np.concatenate([np.stack([a, b, c], -1).reshape(-1, 3), np.stack([a, c, d], -1).reshape(-1, 3)])
    return V, np.ascontiguousarray(F, dtype=np.int32)


def _torus_cloud(n, seed, R=0.6, r=0.22):
    """n points spread evenly through a solid torus in a seeded orientation, in a spatial order."""
    rng = np.random.default_rng(seed + 5)
    p = np.empty((0, 3))
    while len(p) < n:
        q = rng.uniform(-1.0, 1.0, size=(int(n * 2.2) + 64, 3)) * (R + r, R + r, r)
        p = np.concatenate([p, q[(np.hypot(q[:, 0], q[:, 1]) - R) ** 2 + q[:, 2] ** 2 <= r * r]])
    p = p[:n] @ _rotation(rng).T
    cell = np.floor((p + 1.0) * 20).astype(np.int64)
    return np.ascontiguousarray(p[np.lexsort((cell[:, 2], cell[:, 1], cell[:, 0]))], dtype=np.float32)


def _surface_cloud(case, seed):
    """A cloud whose points, like the grid, lie on multiples of a power of two, moved by whole grid
    cells as the seed says: its isosurface moves with it and keeps its vertex and triangle counts."""
    p = np.round(_torus_cloud(case["points"], 11, 0.42, 0.18) * 65536.0) / 65536.0
    dx = case["grid_dx"]
    room = int((1.0 - 0.6 - case["radius"]) / dx) - case["blur"] - 2
    return (p + dx * np.random.default_rng(seed + 9).integers(-room, room + 1, size=3)).astype(np.float32)


# ---------------------------------------------------------------- work
def _count(case):
    s, r, p = case["size"], case["res"], case["ppc"]
    frac = {"sphere": 4.19 * s ** 3, "ellipsoid": 0.0377 * s ** 3, "box": 8.0 * s ** 3,
            "spheres3": 3 * 4.19 * (0.17 * s) ** 3}[case.get("shape", "sphere")]
    return frac * r ** 3 * p ** 3


def _rollout_work(case, backward=True):
    """Per particle and step: the state and controls read, the next state written; backward: the
    state, the adjoint and the controls read, the adjoint written; each covered node's record
    written once and read once in each direction.  Operations: 64-node sums of the four stencil
    stages, the polar decomposition and its derivative."""
    n, steps, w = _count(case), case.get("steps", 1), 8.0 if case.get("precision") == "fp64" else 4.0
    nodes = n / case["ppc"] ** 3
    per = w * (24 + 9 + 4 + 24) + (w * (24 + 9 + 4 + 24 + 24) if backward else 0.0)
    node = 4 * w * 2 * (2 if backward else 1)
    return {"bytes": steps * (n * per + nodes * node), "flops": steps * n * (11000.0 if backward else 4500.0)}


def work(case):
    kind = case["kind"]
    if kind == "gradient":
        return _rollout_work(case)
    if kind in ("step", "compgraph"):
        w = _rollout_work(case, kind == "compgraph")
        w["bytes"] += 2 * 472.0 * _count(case)
        return w
    if kind == "batch":
        ws = [_rollout_work(c) for c in _batch_cases(case)]
        return {k: sum(w[k] for w in ws) for k in ("bytes", "flops")}
    if kind == "mesh":
        # every lattice point's mask and every kept point written; every lattice point against every face
        lattice = (1.16 / case["point_dx"]) ** 2 * (0.8 / case["point_dx"])
        faces = 2.0 * case["around"] * case["along"]
        return {"bytes": lattice + 12 * 0.2 * lattice, "flops": 60.0 * lattice * faces}
    nodes = (2.0 / case["grid_dx"]) ** 3
    if kind == "surface":
        return {"bytes": 12.0 * case["points"] + 4 * nodes + 36.0 * nodes ** (2 / 3) * 6,
                "flops": 10.0 * case["points"] * 8 * (case["radius"] / case["grid_dx"]) ** 3 + 27.0 * case["blur"] * nodes}
    q = case["quality"]
    return {"bytes": 12.0 * case["points"] + 4 * nodes * (2 + q ** 3),
            "flops": 192.0 * case["points"] + 192.0 * nodes * q ** 3}


# ---------------------------------------------------------------- exact values in torch float64
def _chunks(n, size=1 << 16):
    return [(a, min(n, a + size)) for a in range(0, n, size)]


class _Geo:
    def __init__(self, sc):
        self.dims, self.dx = tuple(sc.dims), float(sc.dx)
        self.mn = torch.as_tensor(np.asarray(sc.min_point), dtype=torch.float64, device=_DEV)
        self.nodes = int(np.prod(self.dims))
        k = torch.arange(4, device=_DEV)
        self.off = torch.stack(torch.meshgrid(k, k, k, indexing="ij"), -1).reshape(64, 3)

    def stencil(self, x):
        """Node ids (0 outside the grid), in-grid flags, weights, offsets x_g - x and weight gradients."""
        r = (x - self.mn) / self.dx
        base = torch.floor(r).to(torch.int64) - 1
        id3 = base[:, None, :] + self.off[None]
        lim = torch.tensor(self.dims, device=_DEV)
        ok = ((id3 >= 0) & (id3 < lim)).all(-1)
        ids = torch.where(ok, (id3[..., 0] * self.dims[1] + id3[..., 1]) * self.dims[2] + id3[..., 2], 0)
        q = base[:, None, :].to(torch.float64) + torch.arange(4, device=_DEV)[None, :, None] - r[:, None, :]  # [n,4,3]
        a = q.abs()
        N = torch.where(a < 1, 0.5 * a ** 3 - a * a + 2.0 / 3.0,
                        torch.where(a < 2, (2 - a) ** 3 / 6.0, torch.zeros_like(a)))
        S = torch.where(a < 1, 1.5 * q * a - 2 * q,
                        torch.where(a < 2, (-0.5 * a + 2 - 2 / a.clamp_min(1e-300)) * q, torch.zeros_like(a)))
        o = self.off
        n0, n1, n2 = N[:, o[:, 0], 0], N[:, o[:, 1], 1], N[:, o[:, 2], 2]
        s0, s1, s2 = S[:, o[:, 0], 0], S[:, o[:, 1], 1], S[:, o[:, 2], 2]
        w = n0 * n1 * n2
        gw = torch.stack([s0 * n1 * n2, n0 * s1 * n2, n0 * n1 * s2], -1) * (-1.0 / self.dx)
        d = torch.stack([q[:, o[:, 0], 0], q[:, o[:, 1], 1], q[:, o[:, 2], 2]], -1) * self.dx
        return ids, ok.to(torch.float64), w, d, gw


def _raster(g, x, m):
    out = torch.zeros(g.nodes, dtype=torch.float64, device=_DEV)
    for a, b in _chunks(len(m)):
        ids, ok, w, _, _ = g.stencil(x[a:b])
        out.index_add_(0, ids.reshape(-1), (w * ok * m[a:b, None]).reshape(-1))
    return out


def _det(A):
    return (A[:, 0] * torch.linalg.cross(A[:, 1], A[:, 2])).sum(-1)


def _inv_t(A):
    c = torch.stack([torch.linalg.cross(A[:, 1], A[:, 2]), torch.linalg.cross(A[:, 2], A[:, 0]),
                     torch.linalg.cross(A[:, 0], A[:, 1])], 1)
    return c / _det(A)[:, None, None]


def _polar(F):
    X = F
    for _ in range(12):
        c = _det(X).abs().pow(1.0 / 3.0)[:, None, None]
        X = 0.5 * (X / c + c * _inv_t(X))
    low = (_det(F) < 0.05).nonzero()[:, 0]
    if len(low):  # flattened or inverted: U V^T with the sign of det F on the smallest singular value
        U, _, Vt = torch.linalg.svd(F[low])
        U, Vt = U.clone(), Vt.clone()
        U[:, :, 2] *= torch.det(U)[:, None]
        Vt[:, 2, :] *= torch.det(Vt)[:, None]
        X = X.index_copy(0, low, U @ Vt)
    S = X.transpose(1, 2) @ F
    return X, 0.5 * (S + S.transpose(1, 2))


def _pk(Fe, R, lam, mu):
    J = _det(Fe).clamp_min(1e-6)
    return 2 * mu[:, None, None] * (Fe - R) + (lam * (J - 1) * J)[:, None, None] * _inv_t(Fe)


def _pk_derivative(Fe, R, S, lam, mu, dF):
    """dP/dF applied to dF; J = max(det Fe, 1e-6) has no derivative where it is clamped."""
    J, Fit = _det(Fe), _inv_t(Fe)
    c = torch.where(J > 1e-6, (Fit * dF).sum((1, 2)), 0.0)
    J = J.clamp_min(1e-6)
    W = R.transpose(1, 2) @ dF - dF.transpose(1, 2) @ R
    eye = torch.eye(3, dtype=torch.float64, device=_DEV)
    A = S.diagonal(dim1=1, dim2=2).sum(-1)[:, None, None] * eye - S
    t = torch.stack([W[:, 2, 1], W[:, 0, 2], W[:, 1, 0]], -1)
    x = (_inv_t(A).transpose(1, 2) @ t[..., None])[..., 0]  # X S + S X = W for the axial vector x of X
    z = torch.zeros_like(x[:, 0])
    X = torch.stack([torch.stack([z, -x[:, 2], x[:, 1]], -1), torch.stack([x[:, 2], z, -x[:, 0]], -1),
                     torch.stack([-x[:, 1], x[:, 0], z], -1)], 1)
    k = lambda s: s[:, None, None]  # noqa: E731
    return (2 * k(mu) * (dF - R @ X) + k(lam * J * J * c) * Fit +
            k(lam * (J - 1) * J) * (k(c) * Fit - Fit @ dF.transpose(1, 2) @ Fit))


class _Exact:
    """The rollout, loss and adjoint of one scene, per-layer state kept."""

    def __init__(self, sc):
        f = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=_DEV)  # noqa: E731
        self.g, self.sc = _Geo(sc), sc
        self.m, self.vol, self.lam, self.mu, self.dfc = f(sc.m), f(sc.vol), f(sc.lam), f(sc.mu), f(sc.dFc)
        self.f, self.target = f(sc.f_ext), f(sc.target)
        self.layers = [(f(sc.x), f(sc.v), f(sc.F), f(sc.C))]
        self.grids = []
        self.k3 = 3.0 / self.g.dx ** 2
        self.eye = torch.eye(3, dtype=torch.float64, device=_DEV)

    def affine(self, a, b, F, C):
        Fe = F[a:b] + self.dfc[a:b]
        R, S = _polar(Fe)
        P = _pk(Fe, R, self.lam[a:b], self.mu[a:b])
        G = (-self.k3 * self.sc.dt * self.vol[a:b])[:, None, None] * (P @ Fe.transpose(1, 2))
        return Fe, R, S, P, G + self.m[a:b, None, None] * C[a:b]

    def step(self):
        x, v, F, C = self.layers[-1]
        g, dt, s = self.g, self.sc.dt, self.sc.smoothing
        node = torch.zeros(g.nodes, 4, dtype=torch.float64, device=_DEV)
        Fes = torch.empty_like(F)
        for a, b in _chunks(len(x)):
            ids, ok, w, d, _ = g.stencil(x[a:b])
            Fes[a:b], _, _, _, G = self.affine(a, b, F, C)
            mom = (self.m[a:b, None] * v[a:b] * (1 - dt * self.sc.drag))[:, None, :] + d @ G.transpose(1, 2)
            wt = (w * ok)[..., None]
            val = torch.cat([wt * mom, wt * self.m[a:b, None, None]], -1)
            node.index_add_(0, ids.reshape(-1), val.reshape(-1, 4))
        occ = node[:, 3:].abs() > _MASS_EPS
        vg = torch.where(occ, node[:, :3] / torch.where(occ, node[:, 3:], 1.0) + dt * self.f, 0.0)
        vn, Cn = torch.empty_like(v), torch.empty_like(C)
        for a, b in _chunks(len(x)):
            ids, ok, w, d, _ = g.stencil(x[a:b])
            wv = (w * ok)[..., None] * vg[ids]
            vn[a:b] = wv.sum(1)
            Cn[a:b] = self.k3 * (wv.transpose(1, 2) @ d)
        self.grids.append((vg, node[:, 3].clone(), occ))
        self.layers.append((x + dt * vn, vn, (1 - s) * (self.eye + dt * Cn) @ Fes + s * F, Cn))

    def loss(self):
        """The reference's log-mass loss and the last layer's adjoint."""
        x = self.layers[-1][0]
        mass = _raster(self.g, x, self.m)
        e = 1.0 + 1e-4
        lg = torch.log(mass + e) - torch.log(self.target + e)
        low = (1e-3 - mass).clamp_min(0.0)
        dl = lg / (mass + e) - 20.0 * low
        ax = torch.empty_like(x)
        for a, b in _chunks(len(x)):
            ids, ok, _, _, gw = self.g.stencil(x[a:b])
            ax[a:b] = self.m[a:b, None] * ((dl[ids] * ok)[..., None] * gw).sum(1)
        z = torch.zeros_like(self.layers[0][2])
        return float((0.5 * lg * lg + 10.0 * low * low).sum()), (ax, torch.zeros_like(ax), z, z.clone())

    def adjoint_step(self, i, adj, exact):
        """Adjoint of layer i from layer i + 1's; also dL/d dFc of layer i."""
        x, v, F, C = self.layers[i]
        Cnext = self.layers[i + 1][3]
        vg, mass, occ = self.grids[i]
        ax, av, aF, aC = adj
        sc, g, k3 = self.sc, self.g, self.k3
        dt, s, damp = sc.dt, sc.smoothing, 1.0 - sc.dt * sc.drag
        gdv = torch.zeros(g.nodes, 3, dtype=torch.float64, device=_DEV)
        vn = dt * ax + av
        Cn = ((1 - s) * dt if exact else dt) * (aF @ (F + self.dfc).transpose(1, 2)) + aC
        for a, b in _chunks(len(x)):
            ids, ok, w, d, _ = g.stencil(x[a:b])
            val = (w * ok)[..., None] * (vn[a:b, None, :] + k3 * (d @ Cn[a:b].transpose(1, 2)))
            gdv.index_add_(0, ids.reshape(-1), val.reshape(-1, 3))
        im = torch.where(occ, 1.0 / torch.where(occ, mass[:, None], 1.0), 0.0)
        gdp = gdv * im
        vm = torch.where(occ, vg - dt * self.f, 0.0) if exact else vg
        gdm = -(im[:, 0]) * (vm * gdv).sum(-1)
        out = [torch.empty_like(t) for t in (ax, av, aF, aC, aF)]
        for a, b in _chunks(len(x)):
            ids, ok, w, d, gw = g.stencil(x[a:b])
            Fe, R, S, P, G = self.affine(a, b, F, C)
            m = self.m[a:b]
            o = gdp[ids] * ok[..., None]
            vgp = vg[ids] * ok[..., None]
            wo = w[..., None] * o
            M = d.transpose(1, 2) @ wo
            u, z = wo.sum(1), (w[..., None] * vgp).sum(1)
            mvp = m[:, None] * v[a:b] * (damp if exact else 1.0)
            sig = (m[:, None] * gdm[ids] * ok + (o * (mvp[:, None, :] + d @ G.transpose(1, 2))).sum(-1) +
                   (vgp * (vn[a:b, None, :] + k3 * (d @ Cn[a:b].transpose(1, 2)))).sum(-1))
            X = (sig[..., None] * gw).sum(1)
            kk = (-k3 * dt * self.vol[a:b])[:, None, None]
            dP = kk * (M.transpose(1, 2) @ Fe)
            Tr = (self.eye + dt * Cnext[a:b]).transpose(1, 2) @ aF[a:b]
            rest = kk * (M @ P) + _pk_derivative(Fe, R, S, self.lam[a:b], self.mu[a:b], dP)
            out[0][a:b] = (X - (G.transpose(1, 2) @ u[..., None])[..., 0] -
                           k3 * (Cn[a:b].transpose(1, 2) @ z[..., None])[..., 0] + ax[a:b])
            out[1][a:b] = m[:, None] * damp * u
            if exact:
                out[4][a:b] = (1 - s) * Tr + rest
                out[2][a:b] = out[4][a:b] + s * aF[a:b]
            else:
                out[2][a:b] = (1 - s) * Tr + s * aF[a:b] + rest + Tr
                out[4][a:b] = out[2][a:b]
            out[3][a:b] = m[:, None, None] * M.transpose(1, 2)
        return tuple(out[:4]), out[4]


def _exact_gradient(sc, adjoint="exact", tied=True):
    """(loss, dL/d dFc -- of layer 0, or summed over the layers -- and layer 0's adjoint)."""
    e = _Exact(sc)
    for _ in range(sc.steps):
        e.step()
    loss, adj = e.loss()
    total = torch.zeros_like(e.dfc)
    for i in range(sc.steps - 1, -1, -1):
        adj, g = e.adjoint_step(i, adj, adjoint == "exact")
        total = total + g if tied else g
    return loss, total, adj


def _colmajor(t):
    return t.transpose(1, 2).reshape(-1, 9)


def exact(case, seed):
    kind = case["kind"]
    if kind == "surface":
        # the isosurface's vertex list follows which float32 node values lie above the level,
        # so a 64-bit field has another list: no value of its own
        return None
    if kind in ("gradient", "compgraph") and case["steps"] * _count(case) > 60e6:
        return None
    with torch.no_grad():
        if kind == "gradient":
            loss, g, _ = _exact_gradient(_scene(case, seed), case["adjoint"], case["control"] == "tied")
            return {"loss": loss, "grad": _colmajor(g).reshape(-1).cpu()}
        if kind == "step":
            sc = _scene(case, seed, v_std=0.3)
            e = _Exact(sc)
            e.step()
            x, v, F, C = e.layers[1]
            out = np.zeros((sc.n, 118))
            for off, a in ((0, x), (3, v), (6, _colmajor(F)), (15, _colmajor(C)), (37, _colmajor(e.dfc))):
                out[:, off: off + a.shape[1]] = a.cpu().numpy()
            for off, a in ((33, sc.m), (34, sc.vol), (35, sc.lam), (36, sc.mu)):
                out[:, off] = a
            return _fields(out)
        if kind == "compgraph":
            sc = _scene(case, seed)
            loss, _, (ax, av, aF, aC) = _exact_gradient(sc, "refcompat", False)
            out = _points_ref(sc).astype(np.float64)
            for off, a in ((46, ax), (49, av), (52, _colmajor(aF)), (61, _colmajor(aC))):
                out[:, off: off + a.shape[1]] = a.cpu().numpy()
            return {"loss": loss, **_fields(out)}
        if kind == "batch":
            res = [_exact_gradient(sc) for sc in _batch_scenes(case, seed)]
            return {"losses": np.array([r[0] for r in res]), "grads": [r[1].cpu() for r in res]}
        if kind == "mass":
            return _exact_mass(case, seed)
        return _exact_mesh(case, seed)


class _Grid:
    """A cubic grid of the export functions, as _Geo takes it."""

    def __init__(self, n, dx):
        self.dims, self.dx, self.min_point = (n, n, n), dx, np.full(3, -1.0)


def _exact_mass(case, seed):
    n, q = int(math.ceil(np.float32(2.0) / np.float32(case["grid_dx"]))), case["quality"]
    dx = float(np.float32(case["grid_dx"]))
    g = _Geo(_Grid(n, dx))
    x = torch.as_tensor(_torus_cloud(case["points"], seed), device=_DEV).to(torch.float64)
    coarse = _raster(g, x, torch.ones(len(x), dtype=torch.float64, device=_DEV))
    fdx = float(np.float32(case["grid_dx"] / q))
    # node positions as the float32 product and sum that place them
    ax = torch.as_tensor((np.float32(-1.0) + np.arange(n * q, dtype=np.float32) * np.float32(fdx)).astype(np.float64),
                         device=_DEV)
    fine = torch.empty((n * q) ** 3, dtype=torch.float64, device=_DEV)
    yz = torch.stack(torch.meshgrid(ax, ax, indexing="ij"), -1).reshape(-1, 2)
    plane = len(yz)
    for i in range(n * q):
        for a, b in _chunks(plane):
            p = torch.cat([ax[i].expand(b - a, 1), yz[a:b]], 1)
            ids, ok, w, _, _ = g.stencil(p)
            fine[i * plane + a: i * plane + b] = (w * ok * coarse[ids]).sum(1)
    return {"coarse": coarse.cpu(), "fine": fine.cpu()}


def _exact_mesh(case, seed):
    """The lattice points (float32 by definition) whose winding number is at least 1/2."""
    V, F = _torus_mesh(case, seed)
    f32 = np.float32
    mn, mx = V.min(0), V.max(0)
    dx = f32(case["point_dx"])
    d = [int(math.ceil(float(f32(f32(mx[a] - mn[a]) / dx)))) + 1 for a in range(3)]
    idx = np.stack(np.meshgrid(*[np.arange(k) for k in d], indexing="ij"), -1).reshape(-1, 3)
    pts = mn + (dx * idx.astype(f32))
    T = torch.as_tensor(V[F], device=_DEV).to(torch.float64)  # [faces, 3, 3]
    P = torch.as_tensor(pts.astype(np.float64), device=_DEV)
    keep = torch.empty(len(P), dtype=torch.bool, device=_DEV)
    for a, b in _chunks(len(P), 1 << 15):
        A, B, C = (T[None, :, k, :] - P[a:b, None, :] for k in range(3))
        la, lb, lc = A.norm(dim=-1), B.norm(dim=-1), C.norm(dim=-1)
        det = (A * torch.linalg.cross(B, C)).sum(-1)
        den = la * lb * lc + (A * B).sum(-1) * lc + (B * C).sum(-1) * la + (C * A).sum(-1) * lb
        keep[a:b] = torch.atan2(det, den).sum(1) / (2 * math.pi) >= 0.5
    return P[keep].cpu()
