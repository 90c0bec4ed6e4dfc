"""The whole-grid sweeps of piles (the path that a world takes after 64 steps
with a pile), each time with the path asserted: the one-cluster solver stamps
its phases, the other two paths do not, and the island sweeps need several
launches more than the whole-grid ones."""
import ctypes

import numpy as np
import pytest

from oracle import cpu
from phys_gb300 import scenes
from test_gpu_parity import compare_worlds
from test_gpu_paths import sphere_scene

pytestmark = pytest.mark.gpu


def path(w):
    if np.any(w.solver_phases()):
        return "cluster"
    return "islands" if w.stats()["kernel_launches"] > 19 else "grid"


def pyramids(g):
    return scenes.generate(scenes.PYRAMIDS_BOXES_ONLY, g, 3)


def worlds(gpu, sc, iterations, sleeping=False):
    g = gpu.GpuWorld(algo=0, iterations=iterations)
    o = cpu.OracleWorld(algo=0, iterations=iterations, order_mode=1)
    for w in (g, o):
        w.set_sleeping_enabled(sleeping)
    return g, o, g.load_scene(sc), o.load_scene(sc)


@pytest.mark.parametrize("name, iterations, dt, steps, first, sleeping", [
    ("one pyramid", 20, 1 / 60, 72, "cluster", False),
    ("four pyramids with hulls", 20, 1 / 60, 72, "cluster", False),
    ("sixteen pyramids with hulls", 20, 1 / 60, 70, "islands", False),
    ("sixty-four pyramids", 4, 1 / 60, 69, "islands", False),
    ("field asleep in part", 8, 1 / 120, 220, "cluster", True),
])
def test_piles_are_swept_over_the_whole_grid(gpu, name, iterations, dt, steps, first, sleeping):
    """Few manifolds, a few thousand, one item of eight a warp, more items than
    the chip holds warps (sixty-four pyramids: 33,000 manifolds, 19,456 fit), and a
    world with sleeping on; bit for bit with the oracle after the change."""
    sc = {"one pyramid": lambda: pyramids(1), "sixty-four pyramids": lambda: pyramids(8),
          "four pyramids with hulls": lambda: scenes.generate(scenes.PYRAMIDS, 2, 3),
          "sixteen pyramids with hulls": lambda: scenes.generate(scenes.PYRAMIDS, 4, 3),
          "field asleep in part": lambda: scenes.mixed_field(1501, 11)}[name]()
    g, o, _, _ = worlds(gpu, sc, iterations, sleeping)
    for s in range(1, steps + 1):
        g.step(dt)
        o.step(dt)
        if s == 64:
            assert path(g) == first
        if s > 64 and (s < 68 or s % 40 == 0):
            compare_worlds(g, o, f"{name} step {s}")
    assert path(g) == "grid"
    compare_worlds(g, o, f"{name} step {steps}")
    for f in ("solved_contact_count", "prepared_points", "warm_start_matches", "color_count"):
        assert g.stats()[f] == o.stats()[f], f


def test_sweeps_are_left_when_the_pile_is_gone(gpu):
    """A pyramid on the whole-grid sweeps whose boxes are thrown apart goes back
    to the one-cluster solver, and a copy made in between goes on as it does."""
    g, o, hg, ho = worlds(gpu, pyramids(1), 20)
    for s in range(70):
        g.step(1 / 60)
        o.step(1 / 60)
    assert path(g) == "grid"
    n = len(hg)
    rng = np.random.default_rng(4)
    for i in range(n):
        if pyramids(1).is_static[i]:
            continue
        lin = (rng.normal(size=3) * [30.0, 0.0, 30.0] + [0.0, 15.0, 0.0]).astype(np.float32)
        g.set_velocity(gpu.Handle(int(hg[i, 0]), int(hg[i, 1])), lin, np.zeros(3, np.float32))
        o.set_velocity(int(ho[i, 0]), lin, np.zeros(3, np.float32))
    c = g.clone()
    seen = set()
    for s in range(150):
        for w in (g, o, c):
            w.step(1 / 60)
        seen.add(path(g))
        if s % 10 == 0:
            compare_worlds(g, o, f"step {s} after the throw")
            compare_worlds(c, o, f"step {s} of the copy")
    assert seen == {"grid", "cluster"} and path(g) == "cluster"


def test_wait_of_the_sweeps_runs_out(gpu):
    """A plank on 120 boxes: its last manifold waits for 119 updates, hundreds of
    turns of its wait.  With 100 turns allowed in the sweeps alone the step fails and
    the world keeps its state; with the default it goes on as the oracle does."""
    k = np.arange(120)
    pos = np.stack([k % 12 * 1.0, np.full(120, 0.49), k // 12 * 1.0], 1)
    lone = np.stack([np.arange(60) % 10 * 2.0 + 40.0, np.full(60, 0.49), np.arange(60) // 10 * 2.0], 1)
    pos = np.concatenate([[[20.0, -0.5, 5.0], [5.5, 1.17, 4.5]], pos, lone])
    n = len(pos)
    sc = sphere_scene(pos, np.full(n, 1.0), np.arange(n) == 0)
    sc.shape[:] = 1
    sc.dims[:] = [1.0, 1.0, 1.0]
    sc.dims[0], sc.dims[1] = [100.0, 1.0, 40.0], [13.0, 0.4, 11.0]
    sc.dims[2:122] = [0.6, 1.0, 0.6]
    g, o, _, _ = worlds(gpu, sc, 8)
    for s in range(70):
        g.step(1 / 120)
        o.step(1 / 120)
    compare_worlds(g, o, "before")
    assert path(g) == "grid" and g.stats()["color_count"] > 100
    before = {k: v.copy() for k, v in g.bodies().items()}
    limit = gpu.lib()._ZN2pe19setSpinLimitIslandsEj  # the sweeps' translation unit alone
    limit.argtypes, limit.restype = [ctypes.c_uint32], None
    try:
        limit(100)
        for _ in range(3):
            with pytest.raises(Exception, match="a bounded wait timed out"):
                g.step(1 / 120)
    finally:
        gpu.check(gpu.lib().pe_debug_set_spin_limit(0, 0))
    for k, v in g.bodies().items():
        assert np.array_equal(v.view(np.uint32), before[k].view(np.uint32)), k
    for s in range(4):
        g.step(1 / 120)
        o.step(1 / 120)
        compare_worlds(g, o, f"step {s} after the limit was restored")
    assert path(g) == "grid"
