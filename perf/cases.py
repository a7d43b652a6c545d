"""What a user of this framework has it do, as cases that can be timed.

Every case authors worlds (or inputs) from a seed, brings them to the state
in which such a program spends its time, and then runs one pass through the
public entry points: a frame of a game or controller loop, a few steps of a
resident simulation, a differentiable rollout with its gradients, or one
allocation-free pair query.  Sizes are those of the benchmark
configurations (1,000 boxes; 131,072 mixed bodies; 4,096 scenes; 1,024 x 64
differentiable boxes; 32,768 bodies with cooked hulls) or lie between them.

The stepping cases run worlds that have landed and keep moving in place
(sleeping off, or velocities written back each frame, which wakes every
body), so that every pass does the same kind of work; `resting` is the
default world after most of it has fallen asleep.  The rollouts rewind to the same
start each pass, so they cover the fall and the landing.
"""
from __future__ import annotations

import ctypes
import importlib
import math

import numpy as np
import torch

fyzz = importlib.import_module("fyzzxyzzy-sdk_b200")
scenes = importlib.import_module("fyzzxyzzy-sdk_b200.scenes")
autograd = importlib.import_module("fyzzxyzzy-sdk_b200.autograd")

DT = 1.0 / 120.0


def listed():
    return [
        # One small interactive scene: a kinematic platform moved to a new
        # target each frame with boxes riding on it; the host sets the
        # target, steps and reads every body back.  Launch and host latency.
        {"name": "platform_60", "kind": "platform", "n": 60},
        # The plain scene (1,000 random boxes) as an application with
        # gameplay callbacks runs it: each frame steps, then reads the
        # contact events, the force-threshold stream and the bodies.
        {"name": "boxes_1000_events", "kind": "boxes", "n": 1000},
        # Machines: chains of boxes on every joint kind, a third of them
        # hung from the floor; four substeps a frame, bodies read back.
        {"name": "mechanisms_300x4", "kind": "mechanisms", "n": 300, "links": 4, "steps": 4},
        # One mid-sized settled pile of an odd size (boxes, spheres,
        # compounds, distance joints), four resident substeps.
        {"name": "pile_20011", "kind": "pile", "n": 20011, "scenes": 1, "steps": 4, "loop": False},
        # The plain method at scale: 131,072 mixed bodies in one settled
        # pile, stepped with its inputs and outputs resident.
        {"name": "pile_131072", "kind": "pile", "n": 131072, "scenes": 1, "steps": 4, "loop": False},
        # The same pile in a host loop: each frame steps once, reads every
        # body to pinned host memory and writes every velocity back.
        {"name": "pile_131072_loop", "kind": "pile", "n": 131072, "scenes": 1, "steps": 1, "loop": True},
        # A level of scattered props that has come to rest, sleeping on (the
        # default): three bodies in four asleep, eight substeps, bodies read
        # back.
        {"name": "resting_40000", "kind": "resting", "n": 40000, "steps": 8},
        # Batched forward: 4,096 independent scenes of 16 to 512 bodies
        # (piles and stacks of unit cubes), as a trainer steps them.
        {"name": "batch_4096", "kind": "batch", "n": 4096, "high": 512, "steps": 4},
        # Cooked convex hulls with boxes and spheres among them.
        {"name": "hulls_32768", "kind": "hulls", "n": 32768, "steps": 4},
        # Differentiable batched rollout: 1,024 scenes of 64 boxes, 128
        # steps, checkpoints every 16; gradients of a centre-target loss
        # with respect to velocities, masses and friction.
        {"name": "rollout_1024x64", "kind": "rollout", "n": 1024, "boxes": 64, "steps": 128, "every": 16},
        # Differentiable mixed scenes of uneven size (boxes, spheres,
        # compounds, distance joints), 64 steps, checkpoints every 8.
        {"name": "rollout_mixed_2000", "kind": "rollout_mixed", "n": 2000, "high": 256, "steps": 64, "every": 8},
        # The allocation-free pair query at its largest size.
        {"name": "sap_8192", "kind": "sap", "n": 8192},
    ]


def draw(rng):
    def log(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    kind = rng.choice(["platform", "boxes", "mechanisms", "pile", "pile", "pile_loop", "resting", "batch", "hulls",
                       "rollout", "rollout_mixed", "sap"])
    if kind == "platform":
        return {"kind": kind, "n": log(8, 200)}
    if kind == "boxes":
        return {"kind": kind, "n": log(100, 4000)}
    if kind == "mechanisms":
        return {"kind": kind, "n": log(8, 1000), "links": rng.randint(2, 6), "steps": rng.randint(1, 4)}
    if kind == "pile":
        return {"kind": kind, "n": log(500, 131072), "scenes": rng.choice([1, 1, 2, 3]), "steps": rng.randint(1, 4),
                "loop": False}
    if kind == "pile_loop":
        return {"kind": "pile", "n": log(500, 131072), "scenes": 1, "steps": 1, "loop": True}
    if kind == "resting":
        return {"kind": kind, "n": log(1000, 40000), "steps": rng.randint(1, 8)}
    if kind == "batch":
        return {"kind": kind, "n": log(16, 4000), "high": rng.randint(64, 512), "steps": rng.randint(1, 4)}
    if kind == "hulls":
        return {"kind": kind, "n": log(200, 32768), "steps": rng.randint(1, 4)}
    if kind == "rollout":
        return {"kind": kind, "n": log(16, 1000), "boxes": rng.randint(8, 64), "steps": rng.randint(16, 64),
                "every": rng.choice([8, 16])}
    if kind == "rollout_mixed":
        return {"kind": kind, "n": log(32, 1500), "high": rng.randint(16, 256), "steps": rng.randint(8, 48),
                "every": 8}
    return {"kind": kind, "n": log(64, 8192)}


# ---- authoring ----
def _mixed(n, seed, side, height, boxes=0.7, compounds=0.1, joined=0.02):
    """scenes.mixed_scale's distributions (boxes, spheres, box + sphere
    compounds, distance-joined pairs), assembled without a loop over the
    bodies and with counts that follow from n alone; x, z in a square of the
    given side, y in [0.5, 0.5 + height]."""
    rng = np.random.Generator(np.random.PCG64(seed))
    pos = np.stack([rng.uniform(-side / 2, side / 2, n), rng.uniform(0.5, 0.5 + height, n),
                    rng.uniform(-side / 2, side / 2, n)], 1)
    joined = rng.permutation(n)[: 2 * int(round(n * joined / 2))].reshape(-1, 2)
    d = rng.standard_normal((joined.shape[0], 3))
    d *= rng.uniform(0.8, 1.5, (joined.shape[0], 1)) / np.linalg.norm(d, axis=1, keepdims=True)
    d[:, 1] = np.abs(d[:, 1])
    pos[joined[:, 1]] = pos[joined[:, 0]] + d
    bodies = np.zeros((n, 14), np.float32)
    bodies[:, 0:3] = pos
    bodies[:, 3:7] = scenes.random_quaternions(rng, n)
    bodies[:, 7:10] = rng.standard_normal((n, 3))
    bodies[:, 13] = 1000.0
    kind = rng.permutation(n) / n
    compound = kind >= 1.0 - compounds
    owner = np.repeat(np.arange(n), 1 + compound)
    second = np.zeros(owner.size, bool)
    second[1:] = owner[1:] == owner[:-1]
    sphere = second | ((kind >= boxes) & ~compound)[owner]
    size = rng.uniform(0.05, 0.3, (owner.size, 3))
    geom = np.zeros((owner.size, 4), np.float32)
    geom[:, :3] = np.where(sphere[:, None], size * np.array([1, 0, 0]), size)
    local = np.tile(scenes.IDENTITY, (owner.size, 1))
    local[second, :3] = rng.uniform(-0.25, 0.25, (int(second.sum()), 3))
    mu = rng.uniform(0.3, 0.8, n)[owner]
    start = bodies[:, :3]
    return scenes.SceneSpec(
        bodies=bodies, shape_body=owner.astype(np.uint32), shape_type=sphere.astype(np.uint32), shape_geom=geom,
        shape_local=local, shape_mat=np.stack([mu, mu, 0 * mu], 1).astype(np.float32),
        joints=joined.astype(np.uint32),
        joint_dist=np.linalg.norm(start[joined[:, 0]] - start[joined[:, 1]], axis=1).astype(np.float32)).validate()


def _pile(n, seed):
    """A pile of the plain scene's density a square metre (131,072 bodies on
    200 x 200 m), dropped from a few metres so that it lands in two seconds."""
    return _mixed(n, seed, math.sqrt(n / 3.28), 5.0)


def _sizes(n, low, high):
    """Body counts of n scenes, log-uniform in [low, high], from the case alone."""
    rng = np.random.Generator(np.random.PCG64(n * 1000 + high))
    return np.exp(rng.uniform(math.log(low), math.log(high + 1), n)).astype(int).clip(low, high)


def _batch(n, high, seed):
    """scenes.batched_scenes: random piles and stacks of unit cubes in turn."""
    out = []
    for k, size in enumerate(_sizes(n, 16, high)):
        scale = (size / 1000.0) ** (1.0 / 3.0)
        out.append(scenes.box_stack_scene(int(size), seed=seed + k) if k % 2 else
                   scenes.random_boxes(int(size), seed=seed + k, xz=10.0 * scale, y=(1.0, 1.0 + 20.0 * scale)))
    return out


def _batch_mixed(n, high, seed):
    """scenes.mixed_batched: small mixed scenes with joined pairs."""
    return [_mixed(int(size), seed + k, 20.0 * (size / 1000.0) ** (1.0 / 3.0), 20.0 * (size / 1000.0) ** (1.0 / 3.0),
                   boxes=0.6, compounds=0.15, joined=0.05) for k, size in enumerate(_sizes(n, 8, high))]


def _world(specs, settle, sleeping=False):
    w = fyzz.World(0)
    if not sleeping:
        w.set_sleeping(False)
    for s in specs:
        w.add_scene(s)
    w.step(DT, settle)
    return w


class _Resident:
    """A device array of the world's state, seen by torch without a copy."""

    def __init__(self, world, pointer, n):
        self.world = world
        self.__cuda_array_interface__ = {"shape": (n, 4), "typestr": "<f4", "data": (pointer, False), "version": 3}


def _resident(world):
    v = world.device_view()
    return {name: torch.as_tensor(_Resident(world, getattr(v, name), v.n_bodies), device="cuda")
            for name in ("position", "orientation", "velocity", "angular_velocity")}


def _host_states(world):
    return torch.zeros((world.counts()["bodies"], 14), dtype=torch.float32, pin_memory=True).numpy()


def _encoded(x):
    """Order-preserving integers of float32 values, as the broadphase's bounds hold them."""
    b = x.to(torch.float32).contiguous().view(torch.int32)
    return torch.where(b < 0, ~b, b ^ torch.tensor(-(1 << 31), dtype=torch.int32, device=x.device))


def _sap_inputs(n, seed):
    """n shapes at the density of a landed pile, one in eight of a static
    body, one in five sharing its body with its neighbour."""
    g = torch.Generator().manual_seed(seed)
    side = math.sqrt(n / 20.0)
    centre = torch.rand((n, 3), generator=g) * torch.tensor([side, 1.5, side])
    half = 0.05 + 0.3 * torch.rand((n, 3), generator=g)
    bounds = torch.cat([_encoded(centre - half), _encoded(centre + half)], 1)
    body = torch.arange(n, dtype=torch.int64)
    shared = torch.rand(n, generator=g) < 0.2
    shared[0] = False
    body = torch.where(shared, body - 1, body)
    dynamic = torch.rand(n, generator=g) < 0.875
    dynamic = torch.where(shared, dynamic.roll(1), dynamic)
    body = (body | (dynamic.to(torch.int64) << 31)).numpy().astype(np.uint32).view(np.int32)
    return bounds, torch.from_numpy(body)


def prepare(case, seed):
    kind, n = case["kind"], case["n"]
    if kind == "sap":
        bounds, body = _sap_inputs(n, seed)
        return {"kind": kind, "n": n, "bounds": bounds.cuda(), "body": body.cuda(), "cap": 64 * n,
                "pairs": torch.zeros((64 * n, 2), dtype=torch.int32, device="cuda"),
                "count": torch.zeros(1, dtype=torch.int32, device="cuda")}
    s = {"kind": kind, "steps": case.get("steps", 1)}
    if kind == "platform":
        spec = scenes.random_boxes(n + 1, seed=seed, xz=0.11 * math.sqrt(n) + 0.4, y=(1.0, 3.0), half=(0.1, 0.2))
        spec.bodies[0, 0:7] = [0, 0.6, 0, 0, 0, 0, 1]
        spec.shape_geom[0, :3] = [0.25 * math.sqrt(n) + 1.0, 0.1, 0.25 * math.sqrt(n) + 1.0]
        w = fyzz.World(0)
        s["platform"] = w.add_scene(spec)
        w.set_body_kinematic(s["platform"], True)
        w.step(DT, 150)
        s["frame"] = 0
    elif kind == "boxes":
        scale = (n / 1000.0) ** (1.0 / 3.0)
        w = fyzz.World(0)
        w.set_sleeping(False)
        first = w.add_scene(scenes.random_boxes(n, seed=seed, xz=10.0 * scale, y=(1.0, 1.0 + 6.0 * scale)))
        w.set_contact_notifications(True)
        for i in range(n):
            w.set_body_contact_report_threshold(first + i, 5000.0)
        w.step(DT, 240)
        # the application keeps the frame's reports, column by column, in buffers of its own
        s["reports"] = {group + "." + name: np.zeros((size, *dtype[name].shape), dtype[name].base)
                        for group, dtype, size in (("events", fyzz.EVENT_DTYPE, 8 * n),
                                                   ("points", fyzz.EVENT_POINT_DTYPE, 16 * n),
                                                   ("changes", fyzz.THRESHOLD_DTYPE, 4 * n))
                        for name in dtype.names}
    elif kind == "mechanisms":
        w = _world([scenes.joint_mechanisms(n, seed=seed, links=case["links"])], 60)
    elif kind == "pile":
        w = _world([_pile(n // case["scenes"], seed + k) for k in range(case["scenes"])], 240)
        s["loop"] = case["loop"]
    elif kind == "resting":
        w = _world([_mixed(n, seed, math.sqrt(n / 0.6), 3.0)], 900, sleeping=True)
    elif kind == "batch":
        w = _world(_batch(n, case["high"], 100_000 * (seed % 10_000)), 200)
    elif kind == "hulls":
        w = _world([scenes.convex_pile(n, seed=seed, xz=0.5 * math.sqrt(n / 2.3), y=(0.5, 4.0))], 200)
    elif kind in ("rollout", "rollout_mixed"):
        base = 100_000 * (seed % 10_000)
        specs = (scenes.loose_piles(n, case["boxes"], base_seed=base) if kind == "rollout"
                 else _batch_mixed(n, case["high"], base))
        w = fyzz.World(0)
        first = [w.add_scene(x) for x in specs]
        w.step(DT, 60)
        w.fit_pair_budget(1.5)
        bodies = w.counts()["bodies"]
        moving = np.concatenate([f + np.arange(x.n_bodies) for f, x in zip(first, specs)])
        rng = np.random.Generator(np.random.PCG64(seed))
        start = np.zeros((bodies, 6), np.float32)
        start[moving] = rng.normal(0, 0.5, (moving.size, 6))
        mass = np.zeros(bodies, np.float32)
        mass[moving] = [1.0 / w.body_mass_properties(int(b))[0] for b in moving]
        friction = np.concatenate([np.concatenate([[x.floor_mat[0]], x.shape_mat[:, 0]]) for x in specs])
        target = w.read_mass_frames()[0] + rng.uniform(-1, 1, (bodies, 3))
        leaf = lambda x: torch.from_numpy(np.ascontiguousarray(x, np.float32)).requires_grad_()  # noqa: E731
        s.update(every=case["every"], start=[leaf(start[:, :3]), leaf(start[:, 3:]), leaf(mass), leaf(friction)],
                 target=torch.from_numpy(target.astype(np.float32)), moving=torch.from_numpy(moving), ran=False)
    s["world"] = w
    s["states"] = _host_states(w)
    return s


def run(s):
    kind = s["kind"]
    if kind == "sap":
        message = ctypes.create_string_buffer(256)
        status = fyzz.lib().fyzz_b200_sap_pairs_static_scratch(
            s["bounds"].data_ptr(), s["body"].data_ptr(), s["n"], s["pairs"].data_ptr(), s["cap"],
            s["count"].data_ptr(), torch.cuda.current_stream().cuda_stream, message, len(message))
        if status:
            raise RuntimeError(message.value.decode())
        return {"pairs": s["pairs"], "count": s["count"]}
    w = s["world"]
    if kind in ("rollout", "rollout_mixed"):
        if s["ran"]:
            w.rollout_rewind()
        s["ran"] = True
        c, v, av = autograd.rollout(w, *s["start"], steps=s["steps"], every=s["every"])
        at = s["moving"]
        if kind == "rollout":
            loss = ((c - s["target"])[at] ** 2).sum(1).mean()
        else:
            loss = c[at, 1].mean() + 0.5 * (v[at] ** 2).sum(1).mean()
        grads = torch.autograd.grad(loss, s["start"])
        return {"centre": c, "velocity": v, "angular": av, "grads": grads}
    if kind == "platform":
        s["frame"] = (s["frame"] + 1) % 4096
        t = 2.0 * math.pi * s["frame"] / 512.0
        w.set_body_kinematic_target(s["platform"], [0.3 * math.sin(t), 0.6 + 0.1 * math.sin(2 * t), 0.0,
                                                    0.0, math.sin(0.2 * math.sin(t)), 0.0, math.cos(0.2 * math.sin(t))])
        w.step(DT)
        return w.read_bodies(s["states"])
    if kind == "boxes":
        w.step(DT)
        events, points = w.contact_events()
        for group, a in (("events", events), ("points", points), ("changes", w.force_threshold_changes())):
            for name in a.dtype.names:
                column = s["reports"][group + "." + name]
                column[: len(a)] = a[name]
                column[len(a):] = 0
        return {"states": w.read_bodies(s["states"]), **s["reports"]}
    w.step(DT, s["steps"])
    if kind == "pile" and s["loop"]:
        w.read_bodies(s["states"])
        w.write_states(s["states"])
        return s["states"]
    if kind in ("mechanisms", "resting"):
        return w.read_bodies(s["states"])
    return _resident(w)


def exact(case, seed):
    """The pair query is integer work and has one answer.  A stepped world
    has none in 64 bits: its contacts, branches and the order of its solver
    make the 32-bit trajectory part from any other arithmetic's within a few
    steps of the hundreds that lead to the state the cases start from."""
    if case["kind"] != "sap":
        return None
    n = case["n"]
    bounds, body = _sap_inputs(n, seed)
    b = bounds.numpy().view(np.uint32)
    flags = body.numpy().view(np.uint32)
    owner, dynamic = flags & 0x7FFFFFFF, flags >> 31
    found = []
    for a in range(n):
        o = slice(a + 1, n)
        hit = (owner[o] != owner[a]) & ((dynamic[o] | dynamic[a]) != 0)
        for k in range(3):
            hit &= (b[o, k] <= b[a, 3 + k]) & (b[a, k] <= b[o, 3 + k])
        p = np.flatnonzero(hit) + a + 1
        found.append(np.stack([np.full(p.size, a), p], 1))
    found = np.concatenate(found)
    pairs = np.zeros((64 * n, 2), np.int32)
    pairs[: len(found)] = found[: 64 * n]
    return {"pairs": torch.from_numpy(pairs), "count": torch.tensor([len(found)], dtype=torch.int32)}


# A body's state in and out (13 floats each way) with its mass and limits; a
# shape's geometry, pose and material; an overlap pair's key and manifold
# from the last step and for the next (4 points of 10 floats, its poses, 2
# friction anchors); the solver's row arithmetic (4 + 1 passes over about
# two contact points and two friction rows a touching pair, 60 operations a
# row) and contact generation (about 600 a pair).
_BODY, _SHAPE, _PAIR = 104 + 44, 60, 2 * (8 + 224 + 56)
_PAIR_OPS = 5 * 4 * 60 + 600


def work(case):
    kind, n = case["kind"], case["n"]
    if kind == "sap":   # bounds and body of each shape, its pairs (about three)
        return {"bytes": n * (24 + 4 + 3 * 8), "flops": 0}
    steps, pairs, shapes = case.get("steps", 1), 3.0, 1.0
    bodies = n
    if kind == "mechanisms":
        bodies, pairs = n * case["links"], 1.5
    elif kind == "pile":
        shapes = 1.1
    elif kind == "batch":
        bodies = n * (case["high"] - 16) / math.log(case["high"] / 16.0)
    elif kind == "rollout":
        bodies = n * case["boxes"]
    elif kind == "rollout_mixed":
        bodies, shapes = n * (case["high"] - 8) / math.log(case["high"] / 8.0), 1.15
    unit = _BODY + shapes * _SHAPE + pairs * _PAIR
    ops = pairs * _PAIR_OPS
    if kind in ("rollout", "rollout_mixed"):   # the forward, its recompute and the adjoint of each step
        unit, ops = 3 * unit, 4 * ops
    host = 56 * bodies * (2 if case.get("loop") else 1) if kind in ("platform", "boxes", "mechanisms", "resting") or \
        case.get("loop") else 0
    return {"bytes": bodies * steps * unit + host, "flops": bodies * steps * ops}
