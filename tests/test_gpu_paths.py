"""The kernels' own paths at the sizes where they change, against the oracle or
against another path that gives the same result by definition."""
import numpy as np
import pytest

from helpers import assert_bit_equal
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
