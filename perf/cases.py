"""Performance cases of the XPBD cloth library.

Each case is one call sequence that a program using the library makes, through
``xpbd_gb300.native``, ``xpbd_gb300.diff`` and ``xpbd_gb300.scene``:

* ``sim``   -- one cloth solver: the timeline jumps (reset, the cached positions
  uploaded), then a few frames run, each with this frame's pin targets and
  moving colliders uploaded, one step, and the positions downloaded, as the
  add-on's frame handler does.
* ``batch`` -- many cloths in one batch handle, the same sequence.
* ``diff``  -- a rollout with one compliance per constraint, a loss on the final
  positions and the gradients of both compliance arrays.
* ``prep``  -- constraint inputs of a cloth from its mesh.

Every pass starts from the same uploaded state, so repeated passes do the same
work.  Frames have 10 substeps of 2 iterations, as everywhere in this
repository's scenes.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ssbl-cuda-xpbd_gb300"))

from xpbd_gb300 import native, scene  # noqa: E402

SUBSTEPS, ITERATIONS = 10, 2
NO_TRIANGLES = np.empty((0, 3, 3), np.float32)


def listed():
    """`n`: vertices per side of the (square) cloth; `mode`: self collision off
    (0), fast (1) or strict (2); `pose`: the uploaded positions; `hard`: the
    add-on's hardness slider (hard stretch solve, from 0.5 on with tethers)."""
    return [
        # the smallest call: a preview cloth hanging from two animated corners
        sim("plain-32", 32, 8, pins=True),
        # a finely meshed curtain without self collision, launch per stage
        sim("plain-180", 180, 4, pins=True),
        # an odd-sized small garment part in strict self collision: latency
        sim("strict-37", 37, 3, mode=2, pose="pleats", sphere=True),
        # the headline drop scene: 10k vertices on a sphere and a 64^3 SDF, pleated as after a drop
        sim("drop-100-strict", 100, 3, mode=2, pose="pleats", sphere=True, sdf=True),
        # the same cloth in the fast mode, lying folded on itself: every query finds contacts
        sim("drop-100-fast", 100, 3, mode=1, pose="fold", sphere=True, sdf=True),
        # a large serving request: 200k vertices at 1 cm spacing, strict
        sim("serve-450-strict", 450, 2, mode=2, pose="pleats", sphere=True, spacing=0.01),
        # the add-on's hardness slider at full: CG stretch solve, caps, tethers
        sim("hard-32", 32, 4, pins=True, hard=1.0),
        # a mid-size stiff cloth: CG stretch solve alone
        sim("hard-100", 100, 3, pins=True, hard=0.4),
        # animated mesh and particles hitting a falling cloth, uploaded every frame
        sim("dynamic-64", 64, 4, dynamic=True),
        # the benchmark's batch: 256 uneven cloths, fast and strict mixed
        {"name": "batch-256", "kind": "batch", "count": 256, "lo": 16, "hi": 128, "self": True, "frames": 3},
        # material fitting: rollout and adjoint of the 64 x 64 cloth
        {"name": "diff-64", "kind": "diff", "n": 64, "frames": 20},
        # import of a 250k-vertex garment
        {"name": "prep-500", "kind": "prep", "n": 500},
    ]


def sim(name, n, frames, mode=0, pose="rest", sphere=False, sdf=False, pins=False, hard=0.0, dynamic=False, spacing=0.0):
    """`spacing`: vertex spacing in metres (0: a 1 m cloth)."""
    return {"name": name, "kind": "sim", "n": n, "frames": frames, "mode": mode, "pose": pose, "sphere": sphere,
            "sdf": sdf, "pins": pins, "hard": hard, "dynamic": dynamic, "spacing": spacing}


def _log_int(rng, lo, hi):
    return min(max(int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))), lo), hi)


def draw(rng):
    kind = rng.choice(["plain", "plain", "self", "self", "self", "hard", "dynamic", "batch", "batch", "diff", "prep"])
    if kind == "batch":
        collide = rng.random() < 0.6
        if collide:
            c = {"kind": "batch", "count": _log_int(rng, 8, 200), "lo": rng.randint(8, 24), "hi": rng.randint(32, 128)}
        else:
            c = {"kind": "batch", "count": _log_int(rng, 8, 200), "lo": rng.randint(4, 12), "hi": rng.randint(16, 64)}
        return dict(c, self=collide, frames=rng.randint(1, 3))
    if kind == "diff":
        return {"kind": "diff", "n": _log_int(rng, 12, 110), "frames": rng.randint(2, 20)}
    if kind == "prep":
        return {"kind": "prep", "n": _log_int(rng, 24, 500)}
    if kind == "plain":
        c = sim("", _log_int(rng, 8, 300), rng.randint(1, 8), pins=rng.random() < 0.7)
    elif kind == "self":
        mode = rng.choice([1, 2])
        wide = rng.random() < 0.3
        c = sim("", _log_int(rng, 60, 420) if wide else _log_int(rng, 12, 160), rng.randint(1, 3), mode=mode,
                pose=rng.choice(["pleats", "fold"]), sphere=rng.random() < 0.7, sdf=rng.random() < 0.4,
                spacing=0.01 if wide else 0.0)
    elif kind == "hard":
        c = sim("", _log_int(rng, 12, 140), rng.randint(1, 4), pins=True, hard=rng.choice([0.2, 0.4, 0.7, 1.0]))
    else:
        c = sim("", _log_int(rng, 16, 120), rng.randint(1, 4), dynamic=True, mode=rng.choice([0, 0, 2]))
    del c["name"]
    return c


# ------------------------------------------------------------------ inputs --
_MESHES: dict = {}


def _mesh(n, side, pins, tether_slack):
    """Rest mesh and constraints (the same for every seed, like a garment's
    file); `pins`: the two corners of the y = +side/2 edge are hard-pinned."""
    key = (n, side, pins, tether_slack)
    if key not in _MESHES:
        pos, tris = scene.grid_mesh(n, side, 0.0)
        w = np.zeros(n * n, np.float32)
        if pins:
            w[(n - 1) * n] = w[n * n - 1] = 1.0
        _MESHES[key] = scene.build_cloth(pos, tris, 0.2, w, tether_slack=tether_slack)
    return _MESHES[key]


def _pose(rest, n, pose, rng):
    """Positions of an n x n cloth: at rest, in pleats, or folded once, with a
    jitter well under the contact distance."""
    p = rest.astype(np.float64).copy()
    side = float(np.ptp(p[:, 0]))
    d = side / (n - 1)
    if pose == "pleats":
        # an arc-length preserving meander along x whose loops nearly touch
        wave = max(0.2, 16.0 * d)
        top, phase = rng.uniform(1.85, 2.1), rng.uniform(0.0, 1.0)
        fine = 64
        s = (np.arange((n - 1) * fine + 1)) * (d / fine)
        a = top * np.sin(2.0 * np.pi * (s / wave + phase))
        x = np.concatenate([[0.0], np.cumsum(np.cos(a[:-1]))])[::fine] * (d / fine)
        z = np.concatenate([[0.0], np.cumsum(np.sin(a[:-1]))])[::fine] * (d / fine)
        col = np.tile(np.arange(n), n)
        p[:, 0] = (x - x.mean())[col]
        p[:, 2] = (z - z.min())[col] + 0.305
        p += rng.uniform(-2.0e-4, 2.0e-4, p.shape)
    elif pose == "fold":
        right = p[:, 0] > 0.0
        p[right, 0] = -p[right, 0] + 0.001
        p[right, 2] += rng.uniform(0.0012, 0.0025)
        p[:, 2] += 0.301
        p[:, :2] += rng.uniform(-2.0e-4, 2.0e-4, (len(p), 2))
    else:
        p[:, 2] += rng.uniform(-1.0e-3, 1.0e-3, len(p))
    return np.ascontiguousarray(p, np.float32)


def _options(case, cloth):
    opt = scene.SolverOptions(dt=1.0 / 60.0, damping=0.99, stretch_compliance=1.0e-7, bend_compliance=1.0e-4,
                              collision_margin=0.005, use_ground=True, ground_height=-1.0)
    mode = case["mode"]
    if mode or case["sphere"] or case["sdf"]:
        opt.collision_margin = opt.cloth_thickness = 0.002
        opt.contact_friction = 0.3
        opt.static_sdf_max_resolution = 64
    if case["sphere"]:
        opt.use_sphere, opt.sphere_radius = True, 0.3
    if mode:
        opt.self_collision, opt.self_collision_mode = True, mode
        opt.self_collision_interval = 2 if mode == 1 else 1
        opt.max_self_collision_neighbors = 32 if mode == 1 else 64
    if case["dynamic"]:
        opt.cloth_thickness, opt.contact_friction = 0.002, 0.2
    if case["hard"]:
        h = scene.derive_hardness(case["hard"])
        opt.stretch_compliance, opt.bend_compliance = h["stretch_compliance"], h["bend_compliance"]
        opt.stretch_optimization_enabled = h["stretch_optimization_enabled"]
        opt.stretch_optimization_strength = h["stretch_optimization_strength"]
        opt.lra_compliance = h["hidden_tether_compliance"] if len(cloth.lra_edges) else 0.0
    return opt


def _cloth(case):
    n = case["n"]
    side = (n - 1) * case["spacing"] if case["spacing"] else 1.0
    h = scene.derive_hardness(case["hard"])
    slack = h["hidden_tether_slack"] if case["hard"] and h["hidden_tether_enabled"] else None
    return _mesh(n, side, case["pins"], slack)


def _sim_inputs(case, seed):
    """Cloth, options, start positions, pin targets and colliders per frame."""
    rng = np.random.default_rng(seed)
    cloth = _cloth(case)
    opt = _options(case, cloth)
    start = _pose(cloth.positions_world, case["n"], case["pose"], rng)
    frames = case["frames"]
    pins, moving = [], []
    way = rng.uniform(-0.004, 0.004, (max(len(cloth.pin_indices), 1), 3))
    for f in range(frames):
        pins.append((cloth.pin_targets_world + (f + 1) * way[: len(cloth.pin_indices)]).astype(np.float32))
    if case["dynamic"]:
        center = np.array([rng.uniform(-0.2, 0.2), rng.uniform(-0.2, 0.2), -0.16])
        ball, faces = scene.icosphere((0.0, 0.0, 0.0), 0.15, 3)
        grit, radii = scene.particle_stream(500, (0.25, -0.2, -0.05), 0.2, 0.02, seed=int(rng.integers(1 << 30)))
        for f in range(frames):
            shift = np.array([0.003 * f, 0.0, 0.006 * f])
            moving.append(((ball + center + shift).astype(np.float32), faces, (grit + 0.5 * shift).astype(np.float32), radii))
    return cloth, opt, start, pins, moving


def prepare(case, seed):
    kind = case["kind"]
    if kind == "sim":
        cloth, opt, start, pins, moving = _sim_inputs(case, seed)
        static = scene.collider_meshes() if case["sdf"] else NO_TRIANGLES
        return {"case": case, "solver": native.NativeXpbdSolver(cloth, opt, static), "start": start,
                "pin_indices": cloth.pin_indices, "pins": pins, "moving": moving}
    if kind == "batch":
        # sizes, materials and pins come from the scene's own fixed draw, the state from the seed
        scs = _batch_scenes(case)
        rng = np.random.default_rng(seed)
        start = []
        for k, s in enumerate(scs):
            pose = ("pleats", "rest", "fold")[k % 3] if case["self"] else "rest"
            start.append(_pose(s.cloth.positions_world, s.meta["side"], pose, rng))
            if len(s.cloth.pin_indices):
                start[-1][s.cloth.pin_indices] = s.cloth.pin_targets_world
        return {"case": case, "solver": native.NativeXpbdBatch([(s.cloth, s.options, s.static_triangles) for s in scs]),
                "start": start}
    if kind == "diff":
        from xpbd_gb300.diff import DiffCloth

        sc = scene.diff_scene(case["n"], case["frames"]) if ("diff", case["n"]) not in _MESHES else _MESHES["diff", case["n"]]
        _MESHES["diff", case["n"]] = sc
        ks, kb, target = _diff_inputs(case, sc.cloth, seed)
        return {"case": case, "cloth": DiffCloth(sc.cloth, sc.options),
                "ks": torch.from_numpy(ks).cuda().requires_grad_(), "kb": torch.from_numpy(kb).cuda().requires_grad_(),
                "target": torch.from_numpy(target).cuda()}
    pos, tris, hard = _prep_inputs(case, seed)
    return {"case": case, "positions": pos, "triangles": tris, "hard": hard}


def _batch_scenes(case):
    key = ("batch", case["count"], case["lo"], case["hi"], case["self"])
    if key not in _MESHES:
        scs = scene.batched_scenes(case["count"], 0, 120, (case["lo"], case["hi"]))
        if not case["self"]:
            for s in scs:
                s.options.self_collision = False
        _MESHES[key] = scs
    return _MESHES[key]


def _diff_inputs(case, cloth, seed):
    rng = np.random.default_rng(seed)
    ks = scene.compliance_field(len(cloth.edges), 1.0e-5, 1.0, int(rng.integers(1 << 30)))
    kb = scene.compliance_field(len(cloth.bends), 1.0e-3, 1.0, int(rng.integers(1 << 30)))
    target = cloth.positions_world + rng.uniform(-0.05, 0.05, cloth.positions_world.shape)
    return ks, kb, target.astype(np.float32)


def _prep_inputs(case, seed):
    n = case["n"]
    pos, tris = scene.grid_mesh(n, 0.01 * (n - 1), 0.0)
    rng = np.random.default_rng(seed)
    pos = (pos + rng.uniform(-1.0e-3, 1.0e-3, pos.shape)).astype(np.float32)
    flip = rng.random(len(tris)) < 0.5  # imported meshes list their triangles from any corner
    tris[flip] = np.roll(tris[flip], 1, axis=1)
    hard = np.zeros(len(pos), bool)
    hard[[0, n - 1]] = True
    return pos, tris, hard


# --------------------------------------------------------------------- run --
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "sim":
        s, out = state["solver"], []
        s.reset()
        s.update_positions(state["start"])
        for f in range(case["frames"]):
            if case["pins"]:
                s.update_pin_targets(state["pin_indices"], state["pins"][f])
            if case["dynamic"]:
                ball, faces, grit, radii = state["moving"][f]
                s.update_dynamic_colliders(indexed=(ball, faces, f == 0), particles=(grit, radii))
            s.step(SUBSTEPS, ITERATIONS, diagnostics=False, synchronize=False)
            out.append(s.download_positions().copy())
        return out
    if kind == "batch":
        s = state["solver"]
        s.reset()
        for k, p in enumerate(state["start"]):
            s.update_cloth_positions(k, p)
        for _ in range(case["frames"]):
            s.step(SUBSTEPS, ITERATIONS, diagnostics=False, synchronize=False)
            out = s.download_positions()
        return out
    if kind == "diff":
        from xpbd_gb300.diff import rollout

        x = rollout(state["ks"], state["kb"], state["cloth"], case["frames"], SUBSTEPS, ITERATIONS)
        gs, gb = torch.autograd.grad(((x - state["target"]) ** 2).sum(), (state["ks"], state["kb"]))
        return x.detach(), gs, gb
    edges, rest, inv, bends, bend_rest = scene.cloth_inputs_device(state["positions"], state["triangles"], 0.2, state["hard"])
    return {"edges": edges, "rest": rest, "inv": inv, "bends": bends, "bend_rest": bend_rest}


def _counts(case):
    """(vertices, edges, bends, triangles) of a case's cloths."""
    sides = [s.meta["side"] for s in _batch_scenes(case)] if case["kind"] == "batch" else [case["n"]]
    v = sum(n * n for n in sides)
    t = sum(2 * (n - 1) ** 2 for n in sides)
    e = sum(2 * n * (n - 1) + (n - 1) ** 2 for n in sides)
    b = sum(2 * n * (n - 1) + (n - 1) ** 2 - 4 * (n - 1) for n in sides)
    return v, e, b, t


def work(case):
    """Mesh, state and uploads read once and positions written once per pass;
    operations of the constraints (about 40 per edge and iteration, 60 per
    vertex and substep) and, with self collision, of one edge-box walk and one
    closest-point test per primitive and pass."""
    v, e, b, t = _counts(case)
    if case["kind"] == "prep":
        return {"bytes": v * 12 + t * 12 + v + e * 12 + v * 4 + b * 12, "flops": t * 30 + (e + b) * 8}
    frames = case["frames"]
    steps = frames * SUBSTEPS
    mesh = v * 16 + e * 12 + b * 12
    flops = steps * (ITERATIONS * 40 * e + 60 * v) + frames * 40 * b
    if case["kind"] == "diff":
        # forward, its replay and the adjoint; the state at each frame written and read
        return {"bytes": 3 * mesh + 2 * frames * v * 36 + (e + b) * 8 + v * 24, "flops": 4 * flops}
    both = case["kind"] == "batch" and case["self"]
    if both or case.get("mode"):
        passes = 4 * steps * (0.75 if both else (0.5 if case["mode"] == 1 else 1.0))
        mesh += t * 12
        flops += passes * (v * 60 + e * 100)
    return {"bytes": mesh + v * 12 + frames * v * 12, "flops": flops}


# ------------------------------------------------------------------- exact --
EPS = 1.0e-7


def _stretch(x, prev, w, i, j, rest, k, dt):
    """Snapshot-Jacobi stretch pass in 64 bits."""
    d = x[j] - x[i]
    length = (d * d).sum(1).clamp_min(EPS).sqrt()
    c = length - rest
    ww = w[i] + w[j]
    a = k.clamp_min(0.0) / max(dt * dt, EPS)
    s = torch.where(ww > 0.0, -0.18 * c / (ww + a).clamp_min(1e-300) / length.clamp_min(EPS), torch.zeros_like(c))
    corr = d * s[:, None]
    size = (corr.detach() * corr.detach()).sum(1).sqrt()
    cap = torch.clamp(torch.clamp(rest * 0.10, max=0.025), min=0.0025)
    over = size > cap
    n = corr / (corr * corr).sum(1).clamp_min(1e-60).sqrt()[:, None]
    corr = torch.where(over[:, None], n * cap[:, None], corr)
    pull = (c > 0.0).to(x.dtype)[:, None] * 0.08
    di, dj = corr * (-w[i])[:, None], corr * w[j][:, None]
    x2 = x.index_add(0, i, di).index_add(0, j, dj)
    p2 = prev.index_add(0, i, di * pull).index_add(0, j, dj * pull)
    return x2, p2


def _bend(x, prev, w, i, j, rest, k, thickness, dt):
    """One bend colour (no vertex twice) in 64 bits."""
    d = x[j] - x[i]
    sq = (d * d).sum(1)
    length = sq.clamp_min(1e-30).sqrt()
    c = length - rest
    ww = w[i] + w[j]
    a = k.clamp_min(0.0) / max(dt * dt, EPS)
    use = (ww > 0.0) & (rest > EPS) & (sq > 1e-10) & (c.abs() > 1e-6)
    corr = d * (0.10 * -c / (ww + a).clamp_min(EPS) / length)[:, None]
    size = (corr.detach() * corr.detach()).sum(1).sqrt()
    cap = torch.clamp(torch.clamp(rest, min=thickness) * 0.08, min=2.5e-4, max=0.020)
    n = corr / (corr * corr).sum(1).clamp_min(1e-60).sqrt()[:, None]
    corr = torch.where((size > cap)[:, None], n * cap[:, None], corr)
    corr = torch.where(use[:, None], corr, torch.zeros_like(corr))
    di, dj = corr * (-w[i])[:, None], corr * w[j][:, None]
    return (x.index_add(0, i, di).index_add(0, j, dj), prev.index_add(0, i, di * 0.06).index_add(0, j, dj * 0.06))


def _velocity(x, prev, vel, w, thickness, dt):
    measured = (x - prev) / dt
    proj = measured - vel
    scale = torch.where((proj * vel).sum(1) > 0.0, 0.9, 1.0).to(x.dtype)
    fb = proj * scale[:, None]
    speed = (fb.detach() * fb.detach()).sum(1).sqrt()
    top = max(2.0e-4, max(thickness, 0.0) * 0.35) / dt
    n = fb / (fb * fb).sum(1).clamp_min(1e-60).sqrt()[:, None]
    fb = torch.where(((scale < 1.0) & (speed > top))[:, None], n * top, fb)
    return torch.where((w > 0.0)[:, None], vel + fb, torch.zeros_like(vel))


def _simulate(cloth, opt, start, ks, kb, frames, targets):
    """Contact-free frames in 64 bits: the positions after each frame."""
    f64 = lambda a: torch.from_numpy(np.asarray(a, np.float64))  # noqa: E731
    dt = float(np.float32(np.float32(opt.dt) / np.float32(SUBSTEPS)))
    g = f64(np.float32(opt.gravity))
    damping, thickness = float(np.float32(opt.damping)), float(np.float32(opt.cloth_thickness))
    w, rest = f64(cloth.inv_mass), f64(cloth.positions_world)
    i, j = (torch.from_numpy(cloth.edges[:, q].astype(np.int64)) for q in (0, 1))
    bi, bj = (torch.from_numpy(cloth.bends[:, q].astype(np.int64)) for q in (0, 1))
    edge_rest, bend_rest = f64(cloth.edge_rest_lengths), f64(cloth.bend_rest_lengths)
    free = (w > 0.0)[:, None]
    x, vel, got = f64(start), torch.zeros_like(rest), []
    pins = torch.from_numpy(cloth.pin_indices.astype(np.int64))
    for f in range(frames):
        goal = f64(targets[f])

        def pin(a):
            return a.index_copy(0, pins, goal) if len(pins) else a

        def still(a):
            return a.index_copy(0, pins, torch.zeros_like(goal)) if len(pins) else a

        for s in range(SUBSTEPS):
            vel = torch.where(free, (vel + g * dt) * damping, torch.zeros_like(vel))
            prev = x
            x = torch.where(free, x + vel * dt, rest)
            x, prev, vel = pin(x), pin(prev), still(vel)
            for it in range(ITERATIONS):
                x, prev = _stretch(x, prev, w, i, j, edge_rest, ks, dt)
                if s == SUBSTEPS - 1 and it == ITERATIONS - 1:
                    for a, b in zip(cloth.bend_color_offsets[:-1], cloth.bend_color_offsets[1:]):
                        x, prev = _bend(x, prev, w, bi[a:b], bj[a:b], bend_rest[a:b], kb[a:b], thickness, dt)
                x, prev, vel = pin(x), pin(prev), still(vel)
            vel = _velocity(x, prev, vel, w, thickness, dt)
        got.append(x)
    return got


def exact(case, seed):
    """Frames without contacts or the CG solve, the rollout with its gradients,
    and the lengths and masses of the preprocessing; the contact paths have no
    plain 64-bit form (their candidate sets are integers of the hash)."""
    if case["kind"] == "sim":
        if case["mode"] or case["sphere"] or case["sdf"] or case["hard"] or case["dynamic"]:
            return None
        cloth, opt, start, pins, _ = _sim_inputs(case, seed)
        ks = torch.full((len(cloth.edges),), float(np.float32(opt.stretch_compliance)), dtype=torch.float64)
        kb = torch.full((len(cloth.bends),), float(np.float32(opt.bend_compliance)), dtype=torch.float64)
        with torch.no_grad():
            return _simulate(cloth, opt, start, ks, kb, case["frames"], pins)
    if case["kind"] == "diff":
        if case["n"] ** 2 * case["frames"] > 100_000:
            return None
        sc = scene.diff_scene(case["n"], case["frames"])
        ks, kb, target = _diff_inputs(case, sc.cloth, seed)
        ks = torch.from_numpy(ks.astype(np.float64)).requires_grad_()
        kb = torch.from_numpy(kb.astype(np.float64)).requires_grad_()
        pins = [sc.cloth.pin_targets_world] * case["frames"]
        x = _simulate(sc.cloth, sc.options, sc.cloth.positions_world, ks, kb, case["frames"], pins)[-1]
        gs, gb = torch.autograd.grad(((x - torch.from_numpy(target.astype(np.float64))) ** 2).sum(), (ks, kb))
        return x.detach(), gs, gb
    if case["kind"] == "prep":
        pos, tris, hard = _prep_inputs(case, seed)
        p = pos.astype(np.float64)
        pairs = np.sort(np.concatenate([tris[:, [0, 1]], tris[:, [1, 2]], tris[:, [2, 0]]]), axis=1).astype(np.int64)
        key = np.unique(pairs[:, 0] * len(p) + pairs[:, 1])
        rest = np.linalg.norm(p[key % len(p)] - p[key // len(p)], axis=1)
        a, b, c = (p[tris[:, q]] for q in range(3))
        share = 0.5 * np.linalg.norm(np.cross(b - a, c - a), axis=1) * float(np.float32(0.2)) / 3.0
        mass = np.zeros(len(p))
        for q in range(3):
            np.add.at(mass, tris[:, q], share)
        inv = 1.0 / mass
        inv[hard] = 0.0
        return {"edges": None, "rest": rest, "inv": inv, "bends": None, "bend_rest": None}
    return None
