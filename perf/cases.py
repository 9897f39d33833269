"""The work that users of this library have it do, as cases that can be timed and compared.

A pass is one 60 Hz frame of a scene (or of everything resident), one ChainMail run, one
splatted image or one shape writeback, called through the package's public entry points.
Sizes are those of the repository's configurations (2 thousand to 1 million Gaussians, 8-
and 12-neighbour graphs, 64- and 128-member clusters, 4 to 20 iterations), round and ragged.

Scenes are uniform ellipsoids with a symmetric nearest-neighbour graph, made on the GPU
from the seed.  Grippers and plates swing about their start (a sine of the frame number),
so a state can be stepped any number of frames and every frame costs about the same.

``exact`` restates the step in FP64 torch, from the equations, for the cases whose result
has a value independent of an order of evaluation.
"""
import ctypes
import importlib
import math
import types

import numpy as np
import torch

pkg = importlib.import_module("3dgs-isaac-sim-xpbd_b200")
scenes, bridge = pkg.scenes, pkg.bridge

SUBSTEPS = 10
SWING, PERIOD = 4.0, 24.0     # amplitude in frames of the gripper's motion, frames per period


def _case(kind, n, **kw):
    """Every case has the same keys; `n` is the Gaussians of the scene, or of the largest object."""
    c = dict(kind=kind, n=n, objects=1, knn=8, members=64, iters=4, substeps=SUBSTEPS, shape=True, robust=True,
             contact=False, blocking=False)
    c.update(kw)
    return c


def listed():
    return [
        # the smallest object of a batch on its own, through the reference's blocking ABI: all latency
        dict(name="plain_2k", **_case("scene", 2000, blocking=True)),
        # the plain small scene (20,000 Gaussians, two grippers), as the reference's bridge drives it
        dict(name="plain_20k", **_case("scene", 20000, blocking=True)),
        # the float polar decomposition, asynchronous frames, a ragged size
        dict(name="float_polar_61k", **_case("scene", 60997, robust=False)),
        # the large scene's settings (self-collision, twisting grippers) at an ordinary, odd size
        dict(name="contact_200k", **_case("scene", 200003, contact=True)),
        # the large scene itself: 1,000,000 Gaussians
        dict(name="large_1m", **_case("scene", 1000000, contact=True)),
        # dense contact: two plates, 12 neighbours, 128 members, 20 iterations; two substeps a pass
        dict(name="plates_250k", **_case("plates", 250007, knn=12, members=128, iters=20, substeps=2, contact=True)),
        # independent objects of uneven size packed into one scene
        dict(name="batch_16", **_case("batch", 60000, objects=16)),
        # served sessions resident in one arena, positions read back after the tick
        dict(name="serve_8", **_case("serve", 60000, objects=8)),
        # the Isaac runtime's own frame: 16 iterations, one step, contact shapes, ground, object shape
        dict(name="runtime_30k", **_case("runtime", 30011, members=2048, iters=16, substeps=1, shape=False,
                                         blocking=True)),
        # a ChainMail wave: seeds, 20 propagation and 6 relax sweeps, arrival times read back
        dict(name="chainmail_300k", **_case("chainmail", 300007, substeps=1)),
        # a 1080p image of the deformed Gaussians, degree-3 colours, kept on the device
        dict(name="splat_250k", **_case("splat", 250000, members=16, substeps=1)),
        # deformed scales and rotations of every Gaussian, read back (the runtime's writeback)
        dict(name="shapes_102k", **_case("shapes", 102363, members=16, substeps=1)),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["scene"] * 5 + ["plates", "batch", "serve", "runtime", "chainmail", "splat", "shapes"])
    if kind == "scene":
        n = _log_int(rng, 2000, 700000)
        return _case(kind, n, iters=rng.choice([4, 4, 6]) if n < 400000 else 4, members=rng.choice([32, 64, 64]),
                     robust=rng.random() < 0.8, shape=rng.random() < 0.9, contact=rng.random() < 0.5,
                     blocking=n < 50000 and rng.random() < 0.5, knn=rng.choice([8, 8, 10]))
    if kind == "plates":
        return _case(kind, _log_int(rng, 20000, 250000), knn=12, members=128, iters=rng.choice([10, 20]), substeps=2,
                     contact=True)
    if kind in ("batch", "serve"):
        return _case(kind, _log_int(rng, 10000, 60000), objects=rng.randint(2, 16 if kind == "batch" else 8))
    if kind == "runtime":
        return _case(kind, _log_int(rng, 4000, 30000), members=2048, iters=16, substeps=1, shape=False, blocking=True)
    return _case(kind, _log_int(rng, 20000, 300000), members=16 if kind != "chainmail" else 64, substeps=1)


# ------------------------------------------------------------------ scenes
def _grid_candidates(p, cell, chunk=65536):
    """For chunks of the points ``p`` (N, 3): (rows, candidates, valid), the points in the 27
    cells of edge ``cell`` around each row's own, as padded index lists."""
    n = p.shape[0]
    c = torch.floor((p - p.min(0).values) / cell).long()
    dim = c.max(0).values + 3
    c = c + 1
    key = (c[:, 2] * dim[1] + c[:, 1]) * dim[0] + c[:, 0]
    key_s, order = torch.sort(key, stable=True)
    dz, dy = torch.meshgrid(torch.arange(-1, 2, device=p.device), torch.arange(-1, 2, device=p.device), indexing="ij")
    shift = ((dz * dim[1] + dy) * dim[0]).reshape(-1)
    for b in range(0, n, chunk):
        rows = order[b:b + chunk]
        base = key[rows][:, None] + shift[None]
        lo = torch.searchsorted(key_s, base - 1, right=False)
        hi = torch.searchsorted(key_s, base + 1, right=True)
        width = int((hi - lo).max())
        at = lo[:, :, None] + torch.arange(width, device=p.device)
        ok = at < hi[:, :, None]
        cand = order[torch.where(ok, at, torch.zeros_like(at))]
        yield rows, cand.reshape(len(rows), -1), ok.reshape(len(rows), -1)


def _scene(n, seed, knn, radii=scenes.DEFAULT_RADII):
    """The arrays of ``XPBD.create`` for one object: centres uniform in an ellipsoid, edges to
    each centre's ``knn`` nearest among the 27 cells around it (both directions, once)."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)

    def randn(*s):
        return torch.randn(*s, generator=g, device="cuda")

    d = randn(n, 3)
    d = d / d.norm(dim=1, keepdim=True)
    u = torch.rand(n, generator=g, device="cuda") ** (1.0 / 3.0)
    pos = d * u[:, None] * torch.tensor(radii, device="cuda")
    q = randn(n, 4)
    q = q / q.norm(dim=1, keepdim=True)
    scales = torch.exp(randn(n, 3) * 0.3 - 4.0)
    volume = 4.0 / 3.0 * math.pi * radii[0] * radii[1] * radii[2]
    keys = []
    for rows, cand, ok in _grid_candidates(pos, (volume * 0.8 * knn / n) ** (1.0 / 3.0)):
        d2 = ((pos[cand] - pos[rows][:, None]) ** 2).sum(-1)
        d2 = torch.where(ok & (cand != rows[:, None]), d2, torch.full_like(d2, math.inf))
        v, k = torch.topk(d2, min(knn, d2.shape[1]), dim=1, largest=False)
        a, b = rows[:, None].expand_as(k), torch.gather(cand, 1, k)
        keep = torch.isfinite(v)
        keys.append((torch.minimum(a, b) * n + torch.maximum(a, b))[keep])
    key = torch.unique(torch.cat(keys))
    edges = torch.stack([key // n, key % n], 1)
    rest = (pos[edges[:, 0]].double() - pos[edges[:, 1]].double()).norm(dim=1).float()

    def host(t):
        return np.ascontiguousarray(t.cpu().numpy())

    return {"pos": host(pos), "scales": host(scales), "rots": host(q), "opacity": np.full(n, 0.9, np.float32),
            "edges": host(edges.int()), "rest": host(rest), "stiff": np.ones(len(edges), np.float32)}


def _swing(t):
    return SWING * math.sin(2.0 * math.pi * (t - 1.0) / PERIOD)


def _swinging(gripper):
    """The gripper with its motion swinging about the start instead of going on for good."""
    straight = type(gripper).pose
    gripper.pose = lambda t: straight(gripper, _swing(t))
    return gripper


def _grippers(scene, rng, radii=scenes.DEFAULT_RADII, count=2):
    """Capsules at the x extremes that pull along x and twist, each holding what is inside it
    and its 20 nearest Gaussians."""
    out = []
    for side in (-1.0, 1.0)[:count]:
        centre = (side * 0.85 * radii[0], 0.0, 0.0)
        vel = (side * float(rng.uniform(0.005, 0.01)), float(rng.uniform(-0.003, 0.003)), 0.0)
        twist = math.radians(float(rng.uniform(-1.0, 1.0)))
        g = scenes.Gripper(scene["pos"], centre, 20, vel, twist)
        inside = scenes.Gripper(scene["pos"], centre, 0, vel, twist, pin_radius=0.055)
        g.idx = np.union1d(g.idx, inside.idx).astype(np.int32)
        g.rel = scene["pos"][g.idx].astype(np.float64) - g.centre
        out.append(_swinging(g))
    return out


def _options(case):
    return dict(substeps=SUBSTEPS, iters=case["iters"], shape=case["shape"], self_collision=case["contact"],
                max_members=case["members"], shape_robust=case["robust"])


def _scenario(case, seed):
    rng = np.random.default_rng(seed)
    scene = _scene(case["n"], seed, case["knn"])
    if case["kind"] == "plates":
        z = scene["pos"][:, 2].astype(np.float64)
        plates = []
        for side in (1.0, -1.0):
            p = scenes.Plate(side, float((side * z).max()) - 0.004 * float(rng.uniform(0.5, 1.5)), 0.0025, math.inf)
            still = type(p).centre
            p.centre = types.MethodType(lambda self, t, still=still: still(self, _swing(t)), p)
            plates.append(p)
        return scenes.Scenario(scene, plates, **_options(case))
    return scenes.Scenario(scene, _grippers(scene, rng), **_options(case))


def _objects(case, seed):
    """Objects with log-spaced, ragged sizes up to n, each with 1 or 2 grippers."""
    rng = np.random.default_rng(seed)
    k, out = case["objects"], []
    lo = max(500.0, case["n"] / 30.0)
    for i in range(k):
        n = int(lo * (case["n"] / lo) ** (i / max(k - 1, 1)))
        radii = tuple(float(r) for r in rng.uniform(0.3, 1.5, 3))
        scene = _scene(n, seed * 1000 + i + 1, case["knn"], radii)
        out.append((scene, _grippers(scene, rng, radii, 1 + i % 2)))
    return out


# ------------------------------------------------------------------ states
class _Owner:
    """Closes an engine or an arena when nothing refers to it any more."""

    def __init__(self, what):
        self.what = what

    def __del__(self):
        self.what.close()


class _Memory:
    """Float32 device memory of an engine, which lives on while a tensor over it does."""

    def __init__(self, ptr, shape, owner):
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f4", "data": (ptr, False), "version": 3}
        self.owner = owner


def _view(ptr, shape, owner):
    return torch.as_tensor(_Memory(ptr, shape, owner), device="cuda")


class State:
    """What a program keeps between frames."""

    def __init__(self, case):
        self.case = case
        self.frame = 0


def _solver(state):
    s = pkg.XPBD(instance=True)
    state.owner = _Owner(s)
    return s


def _set_positions(solver, pos):
    f = solver.raw.xpbd_b200_set_positions
    f.argtypes = [ctypes.c_void_p, ctypes.c_int]
    f.restype = ctypes.c_int
    p = np.ascontiguousarray(pos, np.float32)
    if solver.lib.xpbd_b200_set_positions(p.ctypes.data, len(p)) != 0:
        raise RuntimeError(solver.last_error())


def _at_rest(solver, scen):
    """Scene on the device, topology built, state at rest; the pins act from the next substep on."""
    scen.setup(solver)
    solver.step()
    solver.reset()
    scen.k = scen.substeps


def _bent(pos, seed):
    """Smoothly twisted and stretched positions."""
    rng = np.random.default_rng(seed)
    p = pos.astype(np.float64)
    a = float(rng.uniform(0.5, 1.0)) * p[:, 0]
    s = 1.0 + 0.2 * np.sin(2.0 * p[:, 0] + float(rng.uniform(0, 6)))
    y, z = p[:, 1] * s, p[:, 2] / s
    return np.stack([p[:, 0] * 1.1, np.cos(a) * y - np.sin(a) * z, np.sin(a) * y + np.cos(a) * z], 1).astype(np.float32)


class _SwingingPads(scenes.RuntimeScenario):
    """The runtime's frame with the lift going up and down after the grasp."""

    def pad_centre(self, side, frame):
        t = min(frame, self.close)
        c = self.pad0[side] + self.pad_dir[side] * (self.close_speed * t)
        lift = SWING * math.sin(2.0 * math.pi * max(0, frame - self.close) / PERIOD)
        return c + np.array([0.0, 0.0, self.lift_speed * lift])


def prepare(case, seed):
    state = State(case)
    kind = case["kind"]
    if kind in ("scene", "plates"):
        state.solver, state.scen = _solver(state), _scenario(case, seed)
        _at_rest(state.solver, state.scen)
    elif kind == "batch":
        state.solver = _solver(state)
        state.scen = pkg.batch.Batch(_objects(case, seed), **_options(case))
        raw, ptr = state.solver.raw, ctypes.c_void_p   # an engine of its own needs the types on the library
        raw.xpbd_b200_step_async.argtypes = [ctypes.c_int]
        raw.xpbd_b200_set_colliders_many.argtypes = [ctypes.c_int, ptr, ptr, ptr, ptr, ctypes.c_float, ctypes.c_float]
        _at_rest(state.solver, state.scen)
    elif kind == "serve":
        objects = _objects(case, seed)
        rows = sum(sc["pos"].shape[0] for sc, _ in objects)
        state.arena = bridge.Arena(pkg.library_path(), rows, 16 * rows, 66 * rows, 68 * rows)
        state.owner = _Owner(state.arena)
        state.sessions = []
        for sc, grippers in objects:
            scen = scenes.Scenario(sc, grippers, **_options(case))
            s = bridge.XPBD(pkg.library_path(), instance=True)
            _at_rest(s, scen)
            state.sessions.append((state.arena.admit(s), scen))
            s.close()
    elif kind == "runtime":
        state.solver = _solver(state)
        state.scen = _SwingingPads(_scene(case["n"], seed, case["knn"]))
        state.scen.setup(state.solver)
        state.scen.advance(state.solver, state.scen.close + 1)
    else:
        state.solver, scene = _solver(state), _scene(case["n"], seed, case["knn"])
        rng = np.random.default_rng(seed)
        scene["opacity"] = rng.uniform(0.02, 1.0, case["n"]).astype(np.float32)
        scen = scenes.Scenario(scene, [], ring_k=1, max_members=case["members"])
        _at_rest(state.solver, scen)
        if kind == "chainmail":
            p = scene["pos"].astype(np.float64)
            state.seeds = [np.argsort(np.linalg.norm(p - np.array([0.9 * s, 0.0, 0.0]), axis=1))[:30].astype(np.int32)
                           for s in (-1.0, 1.0)]
            state.push = np.tile(np.float32([float(rng.uniform(0.004, 0.006)), 0.0, 0.0]), (30, 1))
        else:
            bent = _bent(scene["pos"], seed)
            _set_positions(state.solver, bent)
            if kind == "splat":
                state.camera = pkg.splat.Camera.framing(bent, 1920, 1080)
                state.solver.render_set_colors(pkg.splat.synthetic_colors(case["n"], 3, seed), 3)
                state.solver.render(state.camera, to_host=False)      # its buffers and the image's place
                state.image = _view(state.solver.render_device_ptr(), (3, 1080, 1920), state.owner)
    if hasattr(state, "solver") and not case["blocking"] and kind in ("scene", "plates", "batch", "chainmail"):
        # the committed positions, float3 in the caller's order, where the solver keeps them
        state.positions = _view(state.solver.positions_device_ptr(), (state.solver.n, 3), state.owner)
    return state


def run(state):
    case, kind = state.case, state.case["kind"]
    if kind == "serve":
        parts, slots, pins = [], [], []
        for slot, scen in state.sessions:
            parts.append(scen.frame_inputs(case["substeps"]))
            slots.append(np.full(len(parts[-1][0]), slot, np.int32))
            pins.append(np.full(len(parts[-1][3]), slot, np.int32))
            scen.k += case["substeps"]
        cat = np.concatenate
        state.arena.step(case["substeps"], cat([p[0] for p in parts]), cat([p[1] for p in parts], axis=1),
                         cat([p[2] for p in parts]), cat(slots), cat(pins), cat([p[3] for p in parts]),
                         cat([p[4] for p in parts], axis=1))
        state.arena.sync()
        return [state.arena.positions(slot, scen.n) for slot, scen in state.sessions]
    if kind == "batch":
        state.scen.advance(state.solver, case["substeps"], blocking=False)
        return state.positions
    if kind == "runtime":
        state.scen.advance(state.solver, 1)
        return state.solver.positions()
    if kind == "chainmail":
        end, sign = state.frame % 2, (1.0, -1.0)[(state.frame // 2) % 2]
        state.frame += 1
        state.solver.chainmail_seed(state.seeds[end], state.push * np.float32(sign * (1.0, -1.0)[end]))
        state.solver.chainmail_run(**scenes.CHAINMAIL_DEFAULTS)
        return {"positions": state.positions, "times": state.solver.chainmail_times()}
    if kind == "splat":
        _, pairs = state.solver.render(state.camera, deform_eps=1e-2, bg=(0.1, 0.2, 0.3), to_host=False)
        return {"image": state.image, "pairs": pairs}
    if kind == "shapes":
        sc, q, count = state.solver.shapes(1e-2)
        return {"scales": sc, "rotations": q, "deformed": count}
    if case["blocking"]:
        state.scen.advance(state.solver, case["substeps"])
        return state.solver.positions()
    state.scen.advance_async(state.solver, case["substeps"])
    return state.positions


def _sizes(case):
    if case["kind"] in ("batch", "serve"):
        lo = max(500.0, case["n"] / 30.0)
        k = case["objects"]
        return sum(int(lo * (case["n"] / lo) ** (i / max(k - 1, 1))) for i in range(k))
    return case["n"]


def work(case):
    """What an iteration cannot do without, once per iteration: positions read and written, each
    directed edge's neighbour, rest length and stiffness read and its multiplier read and
    written, each cluster member's index read.  Per substep the state (positions and
    velocities) in and out; per pass the result out."""
    n, d = _sizes(case), 1.17 * case["knn"]
    if case["kind"] == "chainmail":
        return {"bytes": 26.0 * n * (32 + 8 + 12 * d) + 16.0 * n, "flops": 26.0 * n * 30 * d}
    if case["kind"] == "splat":   # per Gaussian: two positions, shape in, colours, neighbours; the image out
        return {"bytes": n * (32 + 28 + 192 + 4 * d) + 12.0 * 1920 * 1080, "flops": n * (600 + 60 * d)}
    if case["kind"] == "shapes":
        return {"bytes": n * (32 + 28 + 28 + 4 * d), "flops": n * (600 + 60 * d)}
    members = min(case["members"], 230 if case["kind"] == "runtime" else case["members"])
    share = 0.4 if case["kind"] == "runtime" else 1.0        # clusters per Gaussian (leader spacing 2)
    per_iter = 32 + 20 * d + 4 * members * share + (32 + 4 * d if case["shape"] else 0)
    flops = 25 * d + 60 * members * share + (30 * d + 300 if case["shape"] else 0)
    steps = case["substeps"]
    return {"bytes": float(n * (steps * (64 + case["iters"] * per_iter) + 12)),
            "flops": float(n * steps * case["iters"] * flops)}


# ------------------------------------------------------------------ exact values
def _f(v):
    """The value a float argument has after the ABI's single precision."""
    return float(np.float32(v))


def _ball3(nbr, rows):
    """Sorted, unique nodes within three hops of each row (itself excluded), padded with -1."""
    def uniq(x):
        x = torch.sort(x, dim=1, descending=True).values
        x[:, 1:][x[:, 1:] == x[:, :-1]] = -1
        x = torch.sort(x, dim=1, descending=True).values
        return x[:, :int((x >= 0).sum(1).max())]

    def step(x):
        y = nbr[x.clamp(min=0)]
        y = torch.where(x[:, :, None] >= 0, y, torch.full_like(y, -1)).reshape(len(x), -1)
        return uniq(torch.cat([x, y], 1))

    ball = step(step(uniq(nbr[rows])))
    ball[ball == rows[:, None]] = -1
    return ball


def _clusters(pos, nbr, cap):
    """Member lists (n, cap), -1 where none: the three-hop ball, thinned to ``cap`` by farthest
    points in single precision (the choice is discrete; its arithmetic is the library's)."""
    n = pos.shape[0]
    out = torch.full((n, cap), -1, dtype=torch.long, device=pos.device)
    size = max(1, min(n, 20000))

    def dist2(a, b):
        d = a - b
        d = d * d
        return (d[..., 0] + d[..., 1]) + d[..., 2]

    for b in range(0, n, size):
        rows = torch.arange(b, min(n, b + size), device=pos.device)
        ball = _ball3(nbr, rows)
        ok = ball >= 0
        p = pos[ball.clamp(min=0)]
        small = ok.sum(1) <= cap
        none = torch.full(ok.shape, -1.0, device=pos.device)
        md = torch.where(ok, dist2(p, pos[rows][:, None]), none)
        cur = md.argmax(1)
        picked = torch.empty(len(rows), cap, dtype=torch.long, device=pos.device)
        for t in range(cap):
            picked[:, t] = torch.gather(ball, 1, cur[:, None])[:, 0]
            md.scatter_(1, cur[:, None], -1.0)
            at = torch.gather(p, 1, cur[:, None, None].expand(-1, 1, 3))
            md = torch.where(md >= 0, torch.minimum(md, dist2(p, at)), md)
            cur = md.argmax(1)
        whole = torch.full_like(picked, -1)
        w = min(cap, ball.shape[1])
        whole[:, :w] = torch.sort(ball, dim=1, descending=True).values[:, :w]
        out[rows] = torch.where(small[:, None], whole, picked)
    return out


def _collide(x, free, types_, pose, dims, obj, owner):
    """Points inside a capsule or a box go onto its surface, collider by collider."""
    for c in range(len(types_)):
        R = torch.tensor(pose[c, :9].reshape(3, 3), dtype=torch.float64, device=x.device)
        t = torch.tensor(pose[c, 9:], dtype=torch.float64, device=x.device)
        h = [float(v) for v in dims[c]]
        l = (x - t) @ R
        if types_[c] == 1:
            e = l.abs() - torch.tensor(h, dtype=torch.float64, device=x.device)
            dist, axis = e.max(1)
            nrm = torch.zeros_like(l).scatter_(1, axis[:, None], 1.0) * torch.where(l >= 0, 1.0, -1.0)
        else:
            a = l.clone()
            a[:, 2] = l[:, 2] - l[:, 2].clamp(-h[1], h[1])
            rad = a.norm(dim=1)
            dist = rad - h[0]
            nrm = a / rad[:, None].clamp(min=1e-20)
        hit = free & (dist < 0)
        if owner is not None:
            hit = hit & (obj == int(owner[c]))
        x = torch.where(hit[:, None], x - (nrm @ R.T) * dist[:, None], x)
    return x


def _near_pairs(p, rest, search, excl):
    """Directed pairs closer than ``search`` now and at least ``excl`` apart at rest."""
    a, b = [], []
    for rows, cand, ok in _grid_candidates(p, search * 1.01, 16384):
        d = (p[rows][:, None] - p[cand]).norm(dim=-1)
        q = (rest[rows][:, None] - rest[cand]).norm(dim=-1)
        i, k = torch.nonzero(ok & (cand != rows[:, None]) & (d < search) & (q >= excl), as_tuple=True)
        a.append(rows[i])
        b.append(cand[i, k])
    return torch.cat(a), torch.cat(b)


def _frame(scen, owner=None, obj=None):
    """Positions after the substeps of the scenario's first frame, from rest, in FP64."""
    dev, f64 = "cuda", torch.float64
    sc = scen.scene
    rest32 = torch.tensor(sc["pos"], device=dev)
    rest, n = rest32.double(), scen.n
    e = torch.tensor(sc["edges"].astype(np.int64), device=dev)
    src, dst = torch.cat([e[:, 0], e[:, 1]]), torch.cat([e[:, 1], e[:, 0]])
    order = torch.argsort(src, stable=True)
    src, dst = src[order], dst[order]
    length = torch.tensor(sc["rest"], device=dev).double().repeat(2)[order]
    deg = torch.bincount(src, minlength=n)
    start = torch.cumsum(deg, 0) - deg
    nbr = torch.full((n, int(deg.max())), -1, dtype=torch.long, device=dev)
    nbr[src, torch.arange(len(src), device=dev) - start[src]] = dst

    def scatter(idx, val, size=n):
        return torch.zeros((size,) + val.shape[1:], dtype=f64, device=dev).index_add_(0, idx, val)

    mem = _clusters(rest32, nbr, scen.max_members)
    lead = torch.arange(n, device=dev)
    mem = torch.cat([lead[:, None], mem], 1)
    mok = mem >= 0
    count = mok.sum(1).double()
    midx = mem.clamp(min=0)

    def moments(x, parts=8):
        c = torch.empty(n, 3, dtype=f64, device=dev)
        s = torch.empty(n, 3, 3, dtype=f64, device=dev)
        for r in lead.chunk(parts):
            d = x[midx[r]] * mok[r][:, :, None]
            c[r] = d.sum(1) / count[r][:, None]
            d = (x[midx[r]] - c[r][:, None]) * mok[r][:, :, None]
            s[r] = d.transpose(1, 2) @ d / count[r][:, None, None]
        return c, s

    eye = torch.eye(3, dtype=f64, device=dev)
    _, s0 = moments(rest)
    det0 = torch.linalg.det(s0)
    ev = torch.cat([torch.linalg.eigvalsh(m) for m in s0.split(16384)])
    solid = (count >= 5) & (ev[:, 0] / ev[:, 2] > _f(0.05))
    shortest = torch.full((n,), math.inf, dtype=f64, device=dev).scatter_reduce_(
        0, src, (rest[src] - rest[dst]).norm(dim=1), "amin")
    shortest = torch.where(torch.isfinite(shortest), shortest, torch.zeros_like(shortest))
    # shape matching at rest: centroid of the ring, and the Gaussians that take part
    ring = (deg + 1).double()
    com0 = (rest + scatter(src, rest[dst])) / ring[:, None]
    arm = rest[dst] - com0[src]
    bias = scatter(src, arm / arm.norm(dim=1, keepdim=True)).norm(dim=1) / deg.clamp(min=1)
    shaped = (deg >= 4) & (bias <= _f(0.4))

    dt, relax, damp = _f(scen.dt), _f(scen.under_relax), _f(scen.vel_damping)
    dt2 = max(dt * dt, 1e-8)
    soft_d, soft_v, soft_s = _f(scen.dist_compliance) / dt2, _f(scen.vol_compliance) / dt2, \
        _f(scen.shape_compliance) / dt2
    x, v = rest.clone(), torch.zeros_like(rest)
    spacing = float(torch.sort(torch.full((n,), math.inf, dtype=f64, device=dev).scatter_reduce_(
        0, src, length, "amin")).values[n // 2]) if scen.self_collision else 0.0
    dc = _f(_f(1.5) * spacing)
    cols, poses, dims, pin, targets = scen.frame_inputs(scen.exact_substeps, k0=scen.substeps)
    for s in range(scen.exact_substeps):
        w = torch.ones(n, dtype=f64, device=dev)
        if len(pin):
            held = torch.tensor(pin.astype(np.int64), device=dev)
            x[held] = torch.tensor(targets[s], device=dev).double()
            v[held] = 0.0
            w[held] = 0.0
        free = w > 0
        x0, x = x, x + v * dt
        if scen.self_collision:
            pa, pb = _near_pairs(x, rest, _f(_f(1.5) * dc), _f(2.0 * dc))
        lam = torch.zeros(len(src), dtype=f64, device=dev)
        lamv = torch.zeros(n, dtype=f64, device=dev)
        for _ in range(scen.iters):
            d = x[src] - x[dst]
            dl = d.norm(dim=1)
            step = (-(dl - length) - soft_d * lam) / (w[src] + w[dst] + soft_d)
            lam = lam + step
            push = scatter(src, d / dl[:, None] * (step * w[src])[:, None]) / deg.clamp(min=1)[:, None]
            x = x + push * relax * free[:, None]
            # volume
            c, sg = moments(x)
            scale = sg.diagonal(dim1=1, dim2=2).mean(1)
            hat = torch.linalg.det(sg / scale[:, None, None])
            J = (scale ** 3 * hat / det0).clamp(min=0).sqrt().clamp(_f(0.333), 3.0)
            valid = solid & (hat > _f(1e-6)) & ((J - 1).abs() >= _f(1e-4))
            sr = sg + (_f(0.06) * scale * (hat < _f(0.2)))[:, None, None] * eye
            inv = torch.linalg.inv(torch.where(valid[:, None, None], sr, eye))
            gs = J / count
            den = torch.empty(n, dtype=f64, device=dev)
            for r in lead.chunk(8):
                g = ((x[midx[r]] - c[r][:, None]) @ inv[r]) * gs[r][:, None, None]
                den[r] = ((g * g).sum(-1) * w[midx[r]] * mok[r]).sum(1)
            dlv = torch.where(valid, (-(J - 1) - soft_v * lamv) / (den + soft_v), torch.zeros_like(den))
            lamv = lamv + dlv
            total, got = torch.zeros_like(x), torch.zeros(n, dtype=f64, device=dev)
            for r in lead.chunk(8):
                use = mok[r] & valid[r][:, None]
                g = ((x[midx[r]] - c[r][:, None]) @ inv[r]) * (dlv[r] * gs[r])[:, None, None]
                total.index_add_(0, midx[r][use], g[use])
                got.index_add_(0, midx[r][use], torch.ones(int(use.sum()), dtype=f64, device=dev))
            avg = total / got.clamp(min=1)[:, None]
            ln = avg.norm(dim=1)
            cut = (0.25 * shortest / ln.clamp(min=1e-300)).clamp(max=1.0)
            cut = torch.where(shortest > 1e-12, cut, torch.ones_like(cut))
            x = x + avg * (cut * relax * free)[:, None]
            if scen.shape:
                com = (x + scatter(src, x[dst])) / ring[:, None]
                dq, dr = x[dst] - com[src], rest[dst] - com0[src]
                A = scatter(src, dq[:, :, None] * dr[:, None, :]) + \
                    (x - com)[:, :, None] * (rest - com0)[:, None, :]
                usv = [torch.linalg.svd(m) for m in torch.where(shaped[:, None, None], A, eye).split(16384)]
                U, Vh = torch.cat([m[0] for m in usv]), torch.cat([m[2] for m in usv])
                flip = torch.ones(n, 3, dtype=f64, device=dev)
                flip[:, 2] = torch.sign(torch.linalg.det(U @ Vh))
                R = (U * flip[:, None, :]) @ Vh
                goal = com + (R @ (rest - com0)[:, :, None])[:, :, 0]
                pull = _f(0.1) * (w / (w + soft_s))
                x = torch.where((free & shaped)[:, None], x + (goal - x) * pull[:, None], x)
            if scen.self_collision:
                d = x[pa] - x[pb]
                dl = d.norm(dim=1)
                hit = (dl < dc) & (w[pa] > 0)
                share = w[pa] / (w[pa] + w[pb]).clamp(min=1e-30)
                val = d * ((dc - dl) / dl.clamp(min=1e-30) * share * hit)[:, None]
                x = x + scatter(pa, val) / scatter(pa, hit.double()).clamp(min=1)[:, None]
            x = _collide(x, free, cols, poses[s].astype(np.float64), dims, obj, owner)
        v = (x - x0) / dt * (1.0 - damp)
        v = torch.where((free & ((x - x0).norm(dim=1) >= 1e-9))[:, None], v, torch.zeros_like(v))
    return x


def exact(case, seed):
    kind = case["kind"]
    # a wave's arrival times tie and the runtime's covers, the deformed shapes' axes and the
    # image's thresholds are choices: those have no value but the library's
    if kind not in ("scene", "plates", "batch", "serve") or _sizes(case) > 300000:
        return None
    if kind in ("scene", "plates"):
        scen = _scenario(case, seed)
        scen.exact_substeps = case["substeps"]
        return _frame(scen)
    parts = []
    for sc, grippers in _objects(case, seed):
        scen = scenes.Scenario(sc, grippers, **_options(case))
        scen.exact_substeps = case["substeps"]
        parts.append(_frame(scen))
    return parts if kind == "serve" else torch.cat(parts)
