"""The work that the framework is timed on: steps of single worlds, steps of
batches of worlds and differentiable rollouts, each through its public entry
points, with the sizes, scenes and time steps of this repository's benchmark
and tests.

A world's case steps one ``GpuWorld`` once a pass with ``step_io`` on pinned
host arrays (poses out, and for worlds that float, forces in): the call of a
simulation loop.  Its scene has come to its steady state in ``prepare`` (a
settled pile, resting boxes, bodies that coast without gravity), so a pass
does the same work however many came before it.  A batch's case steps all
worlds of a ``GpuBatch``.  A rollout's case is one gradient of a loss through
``rollout_function()``: forward and adjoint from the same initial state.
"""
from __future__ import annotations

import pathlib
import sys
import types

import numpy as np
import torch

_PACKAGE = str(pathlib.Path.cwd() / "phys-engine_gb300")
if _PACKAGE not in sys.path:
    sys.path.insert(0, _PACKAGE)

_SELECTORS = {"sap": 0, "grid": 1, "tree": 2}


def listed():
    return [
        # The smallest world a game or a test steps: ten boxes at rest on a
        # floor.  Latency, launches and the host path are all there is.
        {"name": "boxes_10", "kind": "world", "scene": "plane", "bodies": 10, "selector": "sap", "dt": 1 / 120,
         "iterations": 8, "settle": 120, "sleeping": False},
        # The benchmark's 1,000 spheres dropped on a floor, once they lie
        # there: a floor that every sphere touches, one contact point each.
        {"name": "spheres_1000", "kind": "world", "scene": "spheres", "bodies": 1000, "selector": "sap",
         "dt": 1 / 60, "iterations": 10, "settle": 2400, "sleeping": False},
        # The reference's own benchmark scene at an odd size, under the tree
        # selector: piles of spheres and boxes a few hundred contacts large.
        {"name": "field_1501_tree", "kind": "world", "scene": "field", "bodies": 1501, "selector": "tree",
         "dt": 1 / 120, "iterations": 8, "settle": 1500, "sleeping": False},
        # The same scene at the size that the reference publishes: about
        # 13,000 manifolds, islands of thousands of them.
        {"name": "field_10000", "kind": "world", "scene": "field", "bodies": 10000, "selector": "sap",
         "dt": 1 / 120, "iterations": 8, "settle": 720, "sleeping": False},
        # A large level at rest: 65,536 boxes in stacks, with sleeping on.
        {"name": "stacks_65536_asleep", "kind": "world", "scene": "stacks", "bodies": 65536, "selector": "sap",
         "dt": 1 / 120, "iterations": 8, "settle": 240, "sleeping": True},
        # The headline workload: 100,000 mixed bodies in a volume under the
        # uniform grid, forces in and poses out every step.  The step is that
        # of a control loop, so that the cloud hardly spreads while it runs.
        {"name": "mixed_100000", "kind": "world", "scene": "mixed", "bodies": 100000, "selector": "grid",
         "dt": 1 / 240, "iterations": 10, "settle": 30, "sleeping": False},
        # Sixteen pyramids under a rain of convex hulls: GJK / EPA beside the
        # box contacts, twenty iterations.
        {"name": "pyramids_hulls_16", "kind": "world", "scene": "pyramids", "bodies": 4611, "selector": "sap",
         "dt": 1 / 60, "iterations": 20, "settle": 900, "sleeping": False},
        # Batched simulation with contact-rich worlds of uneven size, as a
        # sampling controller or a learner steps them.
        {"name": "batch_field_1024", "kind": "batch", "scene": "field", "worlds": 1024, "smallest": 16,
         "largest": 512, "dt": 1 / 120, "iterations": 8, "settle": 240},
        # The benchmark's batch at half its number of worlds: uneven worlds of
        # mixed bodies in a volume, few contacts.
        {"name": "batch_mixed_2048", "kind": "batch", "scene": "mixed", "worlds": 2048, "smallest": 16,
         "largest": 2048, "dt": 1 / 240, "iterations": 10, "settle": 8},
        # Gradients for a handful of worlds: latency of one rollout.
        {"name": "rollout_plane_8", "kind": "rollout", "scene": "plane", "worlds": 8, "smallest": 33, "largest": 33,
         "steps": 20, "dt": 1 / 120, "iterations": 10, "checkpoint": 10},
        # The benchmark's differentiable worlds (64 boxes on a plane), a
        # horizon that ends inside a checkpoint interval.
        {"name": "rollout_plane_1024", "kind": "rollout", "scene": "plane", "worlds": 1024, "smallest": 64,
         "largest": 64, "steps": 24, "dt": 1 / 120, "iterations": 10, "checkpoint": 10},
        # Uneven worlds of mixed bodies: sparse contacts, long sorts.
        {"name": "rollout_mixed_512", "kind": "rollout", "scene": "mixed", "worlds": 512, "smallest": 16,
         "largest": 1024, "steps": 20, "dt": 1 / 60, "iterations": 10, "checkpoint": 10},
    ]


def _log_uniform(rng, lo, hi):
    return min(hi, max(lo, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    """One more case: a kind of work, a scene, sizes over the logarithm of
    their range, and the options that a program sets."""
    kind = rng.choice(("world", "world", "batch", "rollout", "rollout"))
    if kind == "world":
        scene = rng.choice(("plane", "spheres", "field", "stacks", "mixed", "pyramids"))
        lo, hi = {"plane": (1, 700), "spheres": (50, 1500), "field": (60, 10000), "stacks": (512, 65536),
                  "mixed": (1000, 100000), "pyramids": (211, 4611)}[scene]
        floats = scene == "mixed"
        return {"kind": "world", "scene": scene, "bodies": _log_uniform(rng, lo, hi),
                "selector": rng.choice(("grid", "tree") if floats else ("sap", "sap", "tree")),
                "dt": 1 / 240 if floats else rng.choice((1 / 120, 1 / 60)),
                "iterations": 20 if scene == "pyramids" else rng.choice((8, 10)), "settle": 30 if floats else 300,
                "sleeping": not floats and rng.random() < 0.3}
    if kind == "batch":
        scene = rng.choice(("plane", "field", "mixed"))
        smallest = _log_uniform(rng, 8, 64)
        largest = _log_uniform(rng, smallest, 400)
        return {"kind": "batch", "scene": scene, "worlds": _log_uniform(rng, 1, 800), "smallest": smallest,
                "largest": largest, "dt": 1 / 240 if scene == "mixed" else 1 / 120, "iterations": rng.choice((8, 10)),
                "settle": 8 if scene == "mixed" else 120}
    scene = rng.choice(("plane", "mixed"))
    smallest = _log_uniform(rng, 8, 64)
    largest = smallest if rng.random() < 0.5 else _log_uniform(rng, smallest, 120 if scene == "plane" else 400)
    worlds = _log_uniform(rng, 1, 500)
    steps = _log_uniform(rng, 2, 24)
    return {"kind": "rollout", "scene": scene, "worlds": worlds, "smallest": smallest, "largest": largest,
            "steps": steps, "dt": 1 / 120 if scene == "plane" else 1 / 60, "iterations": rng.choice((8, 10)),
            "checkpoint": rng.choice((5, 10))}


# ------------------------------------------------------------------ scenes ---
def _scene(kind, bodies, seed):
    from phys_gb300 import scenes

    if kind == "plane":
        return scenes.generate(scenes.BOXES_ON_PLANE, bodies, seed)
    if kind == "spheres":
        return scenes.generate(scenes.SPHERES_ON_FLOOR, bodies, seed)
    if kind == "mixed":
        return scenes.generate(scenes.MIXED_VOLUME, bodies, seed)
    if kind == "field":
        return scenes.mixed_field(bodies, seed)
    if kind == "pyramids":
        # generate(PYRAMIDS, g): g x g pyramids of 210 boxes and their share
        # of hulls; the first `bodies` bodies, the last of them fewer hulls
        g = 1
        while 288 * g * g < bodies and g < 4:
            g += 1
        sc = scenes.generate(scenes.PYRAMIDS, g, seed)
        return sc.subset(np.arange(min(bodies, sc.count)))
    if kind == "stacks":
        # tiles of 512 boxes, each stack moved by up to a centimetre
        tiles = max(1, round(bodies / 512))
        tx = max(1, int(np.sqrt(2 * tiles)))
        tz = max(1, round(tiles / tx))
        sc = scenes.box_stacks(tx, tz)
        rng = np.random.default_rng(seed)
        shift = rng.uniform(-0.01, 0.01, size=(tx * tz * 256, 2)).astype(np.float32)
        rows = np.flatnonzero(sc.is_static == 0)
        for level in (0, 1):  # a stack's two boxes follow one another
            sc.pos[rows[level::2], 0] += shift[:, 0]
            sc.pos[rows[level::2], 2] += shift[:, 1]
        return sc
    raise ValueError(kind)


def _world_sizes(case):
    rng = np.random.default_rng(case["worlds"])
    lo, hi = case["smallest"], case["largest"]
    return [int(n) for n in np.rint(lo * (hi / lo) ** rng.random(case["worlds"]))]


def _cell(scene):
    extent = np.where(scene.shape == 0, scene.dims[:, 0], np.linalg.norm(scene.dims * 0.5, axis=1))
    return float(2.0 * extent.max())


def _pinned(*shape):
    return torch.zeros(shape, dtype=torch.float32).pin_memory().numpy()


# ----------------------------------------------------------------- prepare ---
def _prepare_world(case, seed):
    from phys_gb300 import engine

    scene = _scene(case["scene"], case["bodies"], seed)
    floats = case["scene"] == "mixed"
    world = engine.GpuWorld(algo=_SELECTORS[case["selector"]],
                            cell_size=_cell(scene) if case["selector"] == "grid" else 0.0,
                            iterations=case["iterations"])
    if floats:
        world.set_gravity((0.0, 0.0, 0.0))
    if case["sleeping"]:
        world.set_sleeping_enabled(True)
    world.load_scene(scene)
    n = world.body_count()
    s = types.SimpleNamespace(kind="world", world=world, dt=case["dt"], positions=_pinned(n, 3),
                              rotations=_pinned(n, 4), forces=None, turn=0)
    if floats:
        # thrusters that push each body back and forth
        push = np.random.default_rng(seed + 1).normal(0.0, 0.1, size=(n, 3)).astype(np.float32)
        s.forces = [_pinned(n, 3), _pinned(n, 3)]
        s.forces[0][:] = push
        s.forces[1][:] = -push
    for _ in range(case["settle"]):
        world.step(case["dt"])
    return s


def _prepare_batch(case, seed):
    from phys_gb300 import engine

    sizes = _world_sizes(case)
    floats = case["scene"] == "mixed"
    batch = engine.GpuBatch([_scene(case["scene"], n, seed + w) for w, n in enumerate(sizes)],
                            iterations=case["iterations"], gravity=(0.0, 0.0, 0.0) if floats else (0.0, -9.81, 0.0))
    s = types.SimpleNamespace(kind="batch", batch=batch, dt=case["dt"], positions=_pinned(batch.n, 3),
                              rotations=_pinned(batch.n, 4))
    batch.step(case["dt"], case["settle"])
    batch.autotune(case["dt"], 3)
    batch.step(case["dt"], 2)
    return s


def _prepare_rollout(case, seed):
    from phys_gb300 import rollout

    sizes = _world_sizes(case)
    scenes_ = [_scene(case["scene"], n, seed + w) for w, n in enumerate(sizes)]
    rng = np.random.default_rng(seed)
    if case["scene"] == "mixed":
        # bodies start axis-aligned and turn as they go
        for sc in scenes_:
            sc.spin[:] = 0.0
    roll = rollout.GpuRollout(scenes_, case["steps"], case["dt"], iterations=case["iterations"],
                              checkpoint_every=case["checkpoint"])
    dev = torch.device("cuda", 0)
    x0, q0, v0, w0 = roll.initial_state()
    moving = ~roll.is_static.astype(bool)
    if case["scene"] == "plane":
        # boxes pushed along the floor
        v0[moving, 0] += rng.normal(0.0, 0.5, size=int(moving.sum())).astype(np.float32)
        v0[moving, 2] += rng.normal(0.0, 0.5, size=int(moving.sum())).astype(np.float32)
    else:
        w0[moving] = rng.normal(0.0, 1.0, size=(int(moving.sum()), 3)).astype(np.float32)
    # what was observed of each body at the end of the horizon
    initial = [torch.tensor(a, device=dev) for a in (x0, q0, v0, w0, roll.mass, roll.friction, roll.restitution)]
    observed = [t + torch.tensor(rng.normal(0.0, 0.3, size=tuple(t.shape)).astype(np.float32), device=dev)
                for t in initial[:4]]
    return types.SimpleNamespace(kind="rollout", roll=roll, function=rollout.rollout_function(), initial=initial,
                                 observed=observed, moving=torch.tensor(moving, device=dev)[:, None])


def prepare(case, seed):
    return {"world": _prepare_world, "batch": _prepare_batch, "rollout": _prepare_rollout}[case["kind"]](case, seed)


# --------------------------------------------------------------------- run ---
def _run_world(s):
    forces = None
    if s.forces is not None:
        forces = s.forces[s.turn]
        s.turn ^= 1
    s.world.step_io(s.dt, forces, s.positions, s.rotations)
    return {"positions": s.positions, "rotations": s.rotations}


def _run_batch(s):
    s.batch.step(s.dt)
    s.batch.read_poses(s.positions, s.rotations)
    return {"positions": s.positions, "rotations": s.rotations}


def _run_rollout(s):
    """Squared distance of the bodies' final states from what was observed, and
    its gradients with respect to everything that the rollout starts from, as a
    program that fits initial states and material parameters takes them."""
    leaves = [t.detach().requires_grad_(True) for t in s.initial]
    final = s.function.apply(s.roll, *leaves)
    loss = sum(((f - o) ** 2 * s.moving).sum() for f, o in zip(final, s.observed))
    loss.backward()
    return {"final": [t.detach() for t in final], "loss": loss.detach(), "gradients": [t.grad for t in leaves]}


def run(state):
    return {"world": _run_world, "batch": _run_batch, "rollout": _run_rollout}[state.kind](state)


# -------------------------------------------------------------------- work ---
# Contact manifolds and points per body in each scene's steady state (measured
# once), for the estimate of the work that a step cannot do without.
_MANIFOLDS = {"plane": 1.0, "spheres": 0.6, "field": 1.8, "stacks": 1.0, "mixed": 0.007, "pyramids": 1.5}
_POINTS = {"plane": 4.0, "spheres": 0.6, "field": 2.6, "stacks": 4.0, "mixed": 0.007, "pyramids": 3.0}
# Operations of one velocity update of a point, of preparing one, of finding
# one manifold, and of one body's integration and bounds.
_UPDATE, _PREPARE, _COLLIDE, _BODY = 130, 450, 900, 150


def work(case):
    if case["kind"] == "world":
        bodies, steps = case["bodies"], 1
    else:
        lo, hi = case["smallest"], case["largest"]
        mean = lo if lo == hi else (hi - lo) / np.log(hi / lo)
        bodies, steps = case["worlds"] * mean, case.get("steps", 1)
    # A pass reads a body's state (52 bytes), mass and material (28), shape
    # (16) and inertia (12), and writes its state; a step's poses or forces go
    # to and come from the host, and the warm start is read and written.
    warm = 44 * _POINTS[case["scene"]] * bodies
    flops = bodies * (_BODY + _COLLIDE * _MANIFOLDS[case["scene"]] +
                      (_PREPARE + _UPDATE * case["iterations"]) * _POINTS[case["scene"]])
    if case["kind"] == "rollout":
        # forward, and an adjoint that costs about three times as much; in and
        # out of a pass go the state, the parameters and their gradients
        return {"bytes": 108 * bodies + 3 * 64 * bodies, "flops": 4 * steps * flops}
    moved = 28 * bodies + (12 * bodies if case["scene"] == "mixed" and case["kind"] == "world" else 0)
    if case["sleeping"] if case["kind"] == "world" else False:
        flops = bodies * (_BODY + _COLLIDE * _MANIFOLDS[case["scene"]])
    return {"bytes": 160 * bodies + moved + 2 * warm, "flops": flops}


def exact(case, seed):
    """None: where a contact starts, which vertex a face keeps and when a
    contact slides are decided on rounded values, so a step in 64 bits is
    another trajectory and not the exact value of this one."""
    return None
