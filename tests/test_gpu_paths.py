"""The kernels' own paths at the sizes where they change, against the oracle or
against another path that gives the same result by definition."""
import numpy as np
import pytest

from helpers import assert_bit_equal, assert_manifolds_equal
from oracle import cpu
from phys_gb300 import scenes

pytestmark = pytest.mark.gpu


def sphere_scene(pos, radius, static):
    n, f = len(pos), np.float32
    return scenes.Scene(shape=np.zeros(n, np.uint8), is_static=np.asarray(static, np.uint8),
                        dims=np.stack([radius, np.zeros(n), np.zeros(n)], 1).astype(f), pos=np.asarray(pos, f),
                        density=np.ones(n, f), restitution=np.zeros(n, f), friction=np.full(n, f(0.5)),
                        linvel=np.zeros((n, 3), f), spin=np.zeros((n, 3), f), hull_id=np.full(n, -1, np.int32),
                        mass=np.zeros(n, f), inv_inertia=np.zeros((n, 3), f))


@pytest.mark.parametrize("n", [2, 33, 65, 700, 4097])
@pytest.mark.parametrize("sizes", ["equal", "two_classes", "uneven"])
def test_tree_reports_each_pair_once_whatever_the_sizes(gpu, n, sizes):
    """The reporter of a pair is the box of the lower size class, or the earlier
    one of two in a class: equal boxes, sizes on both sides of a class edge,
    and sizes over a factor of thirty give the sweep's pairs."""
    rng = np.random.default_rng(n)
    radius = {"equal": np.full(n, 0.25), "two_classes": rng.choice([0.3333, 0.3334, 0.66, 0.67, 1.33, 1.34], n),
              "uneven": 10.0 ** rng.uniform(-0.6, 0.9, n)}[sizes]
    side = 1.8 * (n * np.mean(radius ** 3)) ** (1 / 3)  # 0.7 sphere volumes per unit volume
    sc = sphere_scene(rng.uniform(-side / 2, side / 2, (n, 3)), radius, rng.random(n) < 0.2)
    got = {}
    for algo in (gpu.SAP, gpu.TREE):
        w = gpu.GpuWorld(algo=algo, iterations=1)
        w.load_scene(sc)
        w.step(1e-4)
        got[algo] = w.pairs()
    assert_bit_equal(got[gpu.TREE], got[gpu.SAP], f"{n} {sizes}")


@pytest.mark.parametrize("n", [1024, 1025, 2048, 2049, 4096])
@pytest.mark.parametrize("alike", [False, True])
def test_tree_built_in_one_block(gpu, n, alike):
    """Sizes at which the block's keys a thread change (one, two, four); alike:
    an eighth of the spheres in one place, so that only the index tells their keys apart
    and a walk finds hundreds of leaves."""
    rng = np.random.default_rng(n)
    pos = rng.uniform(-12.0, 12.0, (n, 3))
    if alike:
        pos[: n // 8] = pos[0]
    sc = sphere_scene(pos, np.full(n, 0.25), np.zeros(n))
    got = {}
    for algo in (gpu.SAP, gpu.TREE):
        w = gpu.GpuWorld(algo=algo, iterations=1)
        w.load_scene(sc)
        w.step(1e-4)
        got[algo] = w.pairs()
    assert_bit_equal(got[gpu.TREE], got[gpu.SAP], f"{n} {alike}")


@pytest.mark.parametrize("algo", ["SAP", "TREE"])
@pytest.mark.parametrize("touching", [0, 8, 9, 64, 65, 2048, 2049, 4300])
def test_pair_order_by_lists(gpu, algo, touching):
    """Lists sorted by a thread (up to 8 partners), a warp (64), a block (2,048)
    and as a bitmap: a slab that touches so many spheres, first, in the middle
    or last in index order, above 4,096 bodies in small groups."""
    rng = np.random.default_rng(touching)
    groups = 1470
    cell = np.stack([np.arange(groups) % 40, np.arange(groups) // 40, np.zeros(groups)], 1) * 3.0
    pos = np.repeat(cell, 3, 0) + rng.uniform(-0.3, 0.3, (3 * groups, 3))
    near = np.argsort(pos[:, 0], kind="stable")[:touching]
    pos[near, 2] -= 40.0  # into the slab below
    for at in (0, len(pos) // 2, len(pos)):
        slab = np.arange(len(pos) + 1) == at
        sc = sphere_scene(np.insert(pos, at, [[58.0, 58.0, -40.0]], 0), np.full(len(slab), 0.4), slab)
        sc.shape[slab] = 1
        sc.dims[slab] = [140.0, 140.0, 0.2]
        ref = gpu.GpuWorld(algo=gpu.GRID, iterations=1)
        got = gpu.GpuWorld(algo=getattr(gpu, algo), iterations=1)
        for w in (ref, got):
            w.load_scene(sc)
            w.step(1e-4)
        assert np.count_nonzero(got.pairs() == at) >= touching
        assert_bit_equal(got.pairs(), ref.pairs(), f"{algo} {touching} at {at}")


@pytest.mark.parametrize("n", [1, 255, 256, 257, 515])
@pytest.mark.parametrize("offset", [0, 1, 3])
def test_batch_poses_reach_any_array(gpu, n, offset):
    """Poses of a tile's edge sizes into pinned arrays on and off 16 bytes and
    into pageable ones, with nothing written around them."""
    import torch

    sc = scenes.generate(scenes.MIXED_VOLUME, n, 7)
    b = gpu.GpuBatch([sc], iterations=2)
    b.step(1 / 60, 2)
    pos, rot, _, _ = b.bodies()
    for make in (lambda k: torch.full((k,), 7.0).pin_memory().numpy(), lambda k: np.full(k, 7.0, np.float32)):
        p, q = make(3 * n + 8), make(4 * n + 8)
        b.read_poses(p[offset:offset + 3 * n], q[offset:offset + 4 * n])
        assert_bit_equal(p[offset:offset + 3 * n].reshape(n, 3), pos, "positions")
        assert_bit_equal(q[offset:offset + 4 * n].reshape(n, 4), rot, "rotations")
        for a, k in ((p, 3), (q, 4)):
            assert np.all(a[:offset] == 7.0) and np.all(a[offset + k * n:] == 7.0)


def boxes_on_floor(n, seed):
    """n boxes pressed 2 cm into a floor and sliding (no stick-slip switch)."""
    sc = scenes.generate(scenes.BOXES_ON_PLANE, n, seed)
    rng = np.random.default_rng(seed)
    ang = rng.uniform(0, 2 * np.pi, n)
    sc.linvel[1:] = (2.0 * np.stack([np.cos(ang), np.zeros(n), np.sin(ang)], 1)).astype(np.float32)
    sc.pos[1:, 1] -= np.float32(0.02)
    return sc


@pytest.mark.parametrize("n", [1, 31, 32, 33, 37, 63, 64, 65, 200])
def test_rollout_block_paths(gpu, n):
    """One world at the sizes where the block's paths change: a group of lanes
    for every manifold or several manifolds a group (32 / 64 manifolds), 128 or
    256 threads (36 bodies).  Forward against the batched engine, bit for bit; gradients against
    the FP64 adjoint, float rounding (6e-8) grown by the 4 steps' condition: the
    1e-3 that this adjoint is held to elsewhere."""
    import torch

    from phys_gb300 import rollout

    sc = boxes_on_floor(n, 3)
    steps, dt, iters = 4, 1 / 120, 10
    roll = rollout.GpuRollout([sc], steps, dt, iterations=iters, checkpoint_every=3)
    start = roll.initial_state()
    args = [torch.tensor(a, device="cuda:0") for a in (*start, roll.mass, roll.friction, roll.restitution)]
    outs = roll.forward(*args)
    batch = gpu.GpuBatch([sc], iterations=iters)
    batch.step(dt, steps)
    for k, (o, r) in enumerate(zip(outs, batch.bodies())):
        assert_bit_equal(o.cpu().numpy(), r, f"state {k}")
    rng = np.random.default_rng(5)
    d = [rng.normal(size=tuple(o.shape)).astype(np.float32) for o in outs]
    grads = roll.backward(*[torch.tensor(a, device="cuda:0") for a in d])
    _, iinv, he = rollout.body_properties(sc)
    _, ref = rollout.fp64_rollout(sc.shape, sc.is_static, he, iinv, start, roll.mass, roll.friction, roll.restitution,
                                  steps, dt, iters, d_final=d)
    dyn = ~sc.is_static.astype(bool)
    for name, g, r in zip(("x0", "q0", "v0", "w0", "mass", "friction", "restitution"), grads, ref):
        g, r = g.cpu().numpy()[dyn], r[dyn]
        assert np.linalg.norm(g - r) <= 1e-3 * max(np.linalg.norm(r), 1e-6), name


@pytest.mark.parametrize("n", [1023, 1024, 1055])
def test_rollout_of_a_large_world_equals_its_parts(gpu, n):
    """Velocities in shared memory up to 1,024 bodies, in global memory beyond:
    boxes that touch the floor alone move in one world as they do in worlds of
    at most 31 boxes, and have the same gradients (one manifold a body: nothing
    is summed in another order)."""
    import torch

    from phys_gb300 import rollout

    sc = boxes_on_floor(n, 3)
    rows = np.arange(1, n + 1)
    parts = [np.concatenate([[0], rows[i:i + 31]]) for i in range(0, n, 31)]
    rng = np.random.default_rng(6)
    d = [rng.normal(size=(n + 1, k)).astype(np.float32) for k in (3, 4, 3, 3)]
    got = []
    for worlds in ([np.arange(n + 1)], parts):
        roll = rollout.GpuRollout([sc.subset(w) for w in worlds], 4, 1 / 120, iterations=10, checkpoint_every=3)
        args = [torch.tensor(a, device="cuda:0")
                for a in (*roll.initial_state(), roll.mass, roll.friction, roll.restitution)]
        outs = roll.forward(*args)
        pick = np.concatenate(worlds)
        grads = roll.backward(*[torch.tensor(a[pick], device="cuda:0") for a in d])
        moving = pick > 0
        got.append([t.cpu().numpy()[moving] for t in (*outs, *grads)])
    for k, (a, b) in enumerate(zip(*got)):
        assert_bit_equal(a, b, f"output {k}")


def test_rollout_of_a_pile(gpu):
    """Several colours and islands: spheres and boxes in two layers on a floor
    (bodies with many manifolds), more manifolds than the block has groups."""
    import torch

    from phys_gb300 import rollout

    sc = scenes.mixed_field(90, 4)
    sc.pos[1:] *= np.float32([0.64, 0.6, 0.64])  # neighbours overlap by a few centimetres
    steps, dt, iters = 2, 1 / 120, 8
    roll = rollout.GpuRollout([sc], steps, dt, iterations=iters, checkpoint_every=2, manifolds_per_body=8)
    start = roll.initial_state()
    args = [torch.tensor(a, device="cuda:0") for a in (*start, roll.mass, roll.friction, roll.restitution)]
    outs = roll.forward(*args)
    batch = gpu.GpuBatch([sc], iterations=iters)
    batch.step(dt, steps)
    st = batch.stats(0)
    assert st["contact_count"] > 64 and st["color_count"] > 3
    for k, (o, r) in enumerate(zip(outs, batch.bodies())):
        assert_bit_equal(o.cpu().numpy(), r, f"state {k}")
    rng = np.random.default_rng(5)
    d = [torch.tensor(rng.normal(size=tuple(o.shape)).astype(np.float32), device="cuda:0") for o in outs]
    for g in roll.backward(*d):
        assert bool(torch.isfinite(g).all())


@pytest.mark.parametrize("n, steps, sleeping", [(60, 140, False), (700, 100, False), (700, 160, True),
                                                (3000, 90, False), (16000, 80, False)])
def test_whole_grid_sweeps_match_the_oracle(gpu, n, steps, sleeping):
    """Piles long enough for the step to change to the whole-grid sweeps (64
    steps): few manifolds, one item of eight a warp, more items than warps, and
    with sleeping on; poses, velocities, pairs and manifolds with their impulses
    against the oracle, bit for bit, before and after the change."""
    from oracle import cpu
    from test_gpu_parity import compare_worlds

    sc = scenes.mixed_field(n, 5)
    g = gpu.GpuWorld(algo=0, iterations=8)
    o = cpu.OracleWorld(algo=0, iterations=8, order_mode=1)
    for w in (g, o):
        w.set_sleeping_enabled(sleeping)
        w.load_scene(sc)
    for s in range(1, steps + 1):
        g.step(1 / 120)
        o.step(1 / 120)
        if s in (60, 66, 70) or s % 20 == 0:
            compare_worlds(g, o, f"step {s}")
    for f in ("solved_contact_count", "prepared_points", "warm_start_matches", "color_count"):
        assert g.stats()[f] == o.stats()[f], f


def test_whole_grid_sweeps_survive_changes_of_path(gpu):
    """A pile is lifted apart (bodies removed until none touches another) and the
    copy of the world goes on: the paths change and the oracle agrees."""
    from oracle import cpu
    from test_gpu_parity import compare_worlds

    sc = scenes.mixed_field(200, 6)
    g = gpu.GpuWorld(algo=0, iterations=8)
    o = cpu.OracleWorld(algo=0, iterations=8, order_mode=1)
    hg, ho = g.load_scene(sc), o.load_scene(sc)
    for phase in range(3):
        for _ in range(70):
            g.step(1 / 120)
            o.step(1 / 120)
        compare_worlds(g, o, f"phase {phase}")
        c = g.clone()
        c.step(1 / 120)
        for i in range(1 + phase, 200, 3):
            g.remove_body(*hg[i, :2])
            o.remove_body(*ho[i, :2])
        g.step(1 / 120)
        o.step(1 / 120)
        compare_worlds(g, o, f"phase {phase} after the removal")


@pytest.mark.parametrize("pairs", [1, 4, 31, 32, 33, 700, 19456, 19457, 45000])
def test_narrowphase_matches_the_oracle_for_any_number_of_pairs(gpu, pairs):
    """Couples of turned boxes and spheres, each couple alone: tiles of 32 pairs
    on eight lanes each up to 19,456 pairs (on 152 SMs), a thread a pair beyond."""
    rng = np.random.default_rng(pairs)
    n = 2 * pairs
    k = np.arange(pairs)
    cell = np.stack([k % 256, k // 256, np.zeros(pairs)], 1) * 6.0
    pos = np.repeat(cell, 2, 0)
    pos[1::2] += rng.uniform(-0.45, 0.45, (pairs, 3))  # every couple's boxes overlap
    sc = sphere_scene(pos, np.full(n, 0.6), np.zeros(n))
    sc.shape[:] = rng.random(n) < 0.75
    boxes = sc.shape == 1
    sc.dims[boxes] = rng.uniform(0.5, 1.5, (int(boxes.sum()), 3))
    sc.dims[boxes & (rng.random(n) < 0.4)] = 1.0
    sc.spin[:] = rng.uniform(-20.0, 20.0, (n, 3)) * (rng.random((n, 1)) < 0.7)
    gw = gpu.GpuWorld(algo=gpu.SAP, iterations=2, order=gpu.ORDER_COLOR)
    ow = cpu.OracleWorld(algo=0, iterations=2, order_mode=1)
    for w in (gw, ow):
        w.load_scene(sc)
    for step in range(3):
        gw.step(1 / 60)
        ow.step(1 / 60)
        assert step > 0 or len(gw.pairs()) == pairs
        assert_bit_equal(gw.pairs(), ow.pairs(), f"{pairs} step {step} pairs")
        assert_manifolds_equal(gw.contacts(), ow.contacts(), what=f"{pairs} step {step}")


@pytest.mark.parametrize("n", [40, 128, 129, 1000, 1025, 2049])
def test_piles_on_one_rank_and_over_the_cluster(gpu, n):
    """Spheres heaped on a floor: manifolds that fit one block's shared memory
    (up to a few hundred points) and more; bodies at the edges of the one-block
    sweep's variants (128, 1,024 and 2,048 with the floor)."""
    sc = scenes.generate(scenes.SPHERES_ON_FLOOR, n - 1, n)
    gw = gpu.GpuWorld(algo=gpu.SAP, iterations=6, order=gpu.ORDER_COLOR)
    ow = cpu.OracleWorld(algo=0, iterations=6, order_mode=1)
    for w in (gw, ow):
        w.load_scene(sc)
    for step in range(60):
        gw.step(1 / 60)
        ow.step(1 / 60)
    assert_bit_equal(gw.pairs(), ow.pairs(), f"{n} pairs")
    assert_manifolds_equal(gw.contacts(), ow.contacts(), what=f"{n}")
    for k in ("pos", "quat", "lin", "ang"):
        assert_bit_equal(gw.bodies()[k], ow.bodies()[k], f"{n} {k}")


@pytest.mark.parametrize("n", [4097, 6143, 6144, 6145, 12289, 32767, 32768, 32769])
@pytest.mark.parametrize("rows", [False, True])
def test_sweep_order_of_tiles(gpu, n, rows):
    """Tiles of 2,048 sorted keys and their remainders, the last size placed by
    lookups and the first that is sorted in passes; rows: few different min.x,
    so that the index decides the order."""
    rng = np.random.default_rng(n)
    side = 1.1 * n ** (1 / 3)
    pos = rng.uniform(-side / 2, side / 2, (n, 3))
    if rows:
        pos[:, 0] = np.round(pos[:, 0])
    sc = sphere_scene(pos, np.full(n, 0.3), np.zeros(n))
    got = {}
    for algo in (gpu.SAP, gpu.GRID):
        w = gpu.GpuWorld(algo=algo, iterations=1)
        w.load_scene(sc)
        for _ in range(2):
            w.step(1e-3)
        got[algo] = w.pairs()
    assert_bit_equal(got[gpu.SAP], got[gpu.GRID], f"{n} {rows}")


@pytest.mark.parametrize("n", [63, 64, 511, 512, 513])
def test_batched_worlds_equal_single_ones_on_either_memory(gpu, n):
    """Worlds of up to 512 bodies are coloured and swept in shared memory, larger
    ones in global memory; beside each a slab on 150 fixed spheres (150 colours:
    two colour windows, more than the shared colour ranges hold)."""
    grid = np.stack(np.meshgrid(np.arange(15), np.arange(10)), -1).reshape(-1, 2) * 0.75
    pos = np.concatenate([np.stack([grid[:, 0], np.zeros(150), grid[:, 1]], 1), [[5.25, 0.54, 3.4]]])
    slab = sphere_scene(pos, np.full(151, 0.3), np.arange(151) < 150)
    slab.shape[150] = 1
    slab.dims[150] = [12.0, 0.5, 8.0]
    sc = [scenes.mixed_field(n - 1, n), slab]
    batch = gpu.GpuBatch(sc, iterations=6)
    worlds = []
    for x in sc:
        w = gpu.GpuWorld(algo=gpu.SAP, iterations=6, order=gpu.ORDER_COLOR)
        w.load_scene(x)
        worlds.append(w)
    for _ in range(100):
        batch.step(1 / 120)
        for w in worlds:
            w.step(1 / 120)
    assert batch.stats(0)["contact_count"] > 0 and batch.stats(1)["color_count"] > 128
    for k, w in enumerate(worlds):
        got, want = batch.world_bodies(k), w.bodies()
        for g, key in zip(got, ("pos", "quat", "lin", "ang")):
            assert_bit_equal(g, want[key], f"{n} world {k} {key}")
        assert_manifolds_equal(batch.contacts(k), w.contacts(), what=f"{n} world {k}")


@pytest.mark.parametrize("n", [4097, 6145, 32767])
def test_sweep_order_held_and_broken(gpu, n):
    """The tiles' sort is left out while the last order holds: spheres at rest
    (held), a tenth of them moved past the others (broken, then held again in
    the new order), two bodies more (other counts: 32,768 and 32,769, where the
    radix sort takes the order over)."""
    rng = np.random.default_rng(n)
    side = 1.1 * n ** (1 / 3)
    sc = sphere_scene(rng.uniform(-side / 2, side / 2, (n, 3)), np.full(n, 0.3), np.zeros(n))
    worlds, handles = [], []
    for algo in (gpu.SAP, gpu.GRID):
        w = gpu.GpuWorld(algo=algo, iterations=1)
        w.set_gravity((0.0, 0.0, 0.0))
        handles.append(w.load_scene(sc))
        worlds.append(w)
    movers = rng.choice(n, n // 10, replace=False)
    to = rng.uniform(-side / 2, side / 2, (len(movers), 3)).astype(np.float32)
    extra = rng.uniform(-side / 2, side / 2, (2, 3)).astype(np.float32)
    for phase in range(4):
        for w, h in zip(worlds, handles):
            if phase == 1:
                for i, p in zip(movers, to):
                    at = gpu.Handle(*(int(x) for x in h[i, :2]))
                    st = w.get_body(at)
                    st.position[:] = p
                    w.set_body(at, st)
            elif phase > 1:
                w.create_body(0, (0.3, 0.0, 0.0), extra[phase - 2], 1.0, False, 0.0, 0.5)
        for step in range(2):
            for w in worlds:
                w.step(1e-3)
            assert_bit_equal(worlds[0].pairs(), worlds[1].pairs(), f"{n} phase {phase} step {step}")


@pytest.mark.parametrize("lanes", [8, 4])
@pytest.mark.parametrize("beyond", [0, 1])
def test_tree_walk_with_fewer_lanes(gpu, lanes, beyond):
    """The last size with so many lanes a leaf (they fill three quarters of the
    chip's threads) and the first beyond: a floor under spheres of three sizes."""
    import torch

    n = torch.cuda.get_device_properties(0).multi_processor_count * 1536 // lanes + beyond
    rng = np.random.default_rng(n)
    side = 1.3 * n ** (1 / 3)
    pos = rng.uniform(-side / 2, side / 2, (n, 3))
    sc = sphere_scene(pos, rng.choice([0.2, 0.35, 0.6], n), np.zeros(n))
    sc.shape[0], sc.is_static[0] = 1, 1
    sc.pos[0], sc.dims[0] = [0, -side / 2, 0], [side, 1.0, side]
    got = {}
    for algo in (gpu.GRID, gpu.TREE):
        w = gpu.GpuWorld(algo=algo, iterations=1)
        w.load_scene(sc)
        w.step(1e-4)
        got[algo] = w.pairs()
    assert np.count_nonzero(got[gpu.TREE][:, 0] == 0) > 300 and len(got[gpu.TREE]) > n
    assert_bit_equal(got[gpu.TREE], got[gpu.GRID], f"{n}")
