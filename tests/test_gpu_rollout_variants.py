"""The rollout kernels' register variants (worlds for every block the chip holds
at once) and the adjoint of piles, where a group of lanes takes several manifolds."""
import numpy as np
import pytest

from helpers import assert_bit_equal
from phys_gb300 import scenes
from test_gpu_paths import boxes_on_floor

pytestmark = pytest.mark.gpu

NAMES = ("x0", "q0", "v0", "w0", "mass", "friction", "restitution")


def run(sc, steps, every, iterations, directions=None, per_body=None):
    """Final states and gradients (numpy), one array each over all worlds."""
    import torch

    from phys_gb300 import rollout

    kw = {} if per_body is None else {"manifolds_per_body": per_body}
    roll = rollout.GpuRollout(sc, steps, 1 / 120, iterations=iterations, checkpoint_every=every, **kw)
    start = roll.initial_state()
    args = [torch.tensor(a, device="cuda:0") for a in (*start, roll.mass, roll.friction, roll.restitution)]
    outs = roll.forward(*args)
    if directions is None:
        rng = np.random.default_rng(5)
        directions = [rng.normal(size=tuple(t.shape)).astype(np.float32) for t in outs]
    grads = roll.backward(*[torch.tensor(a, device="cuda:0") for a in directions])
    return roll, start, directions, [t.cpu().numpy() for t in outs], [t.cpu().numpy() for t in grads]


def many(gpu, n, make):
    """More worlds of n bodies than the device has SMs (the rule's line)."""
    import torch

    count = torch.cuda.get_device_properties(0).multi_processor_count + 9
    return [make(seed) for seed in range(count)]


@pytest.mark.parametrize("boxes", [32, 63])
def test_register_variants(gpu, boxes):
    """Worlds of 33 bodies (four blocks of 128 threads an SM) and of 64 (two of
    256): forward as the batched engine, and states and gradients as worlds have
    that run alone (boxes that touch the floor alone: one manifold a body,
    nothing is summed in another order), bit for bit."""
    sc = many(gpu, boxes + 1, lambda seed: boxes_on_floor(boxes, seed))
    n = boxes + 1
    _, _, d, outs, grads = run(sc, 5, 3, 10)
    batch = gpu.GpuBatch(sc, iterations=10)
    batch.step(1 / 120, 5)
    for k, (o, r) in enumerate(zip(outs, batch.bodies())):
        assert_bit_equal(o, r, f"state {k}")
    for w in (0, 1, len(sc) // 2, len(sc) - 1):
        rows = slice(w * n, (w + 1) * n)
        _, _, _, one, grad = run([sc[w]], 5, 3, 10, [a[rows] for a in d])
        for k, (a, b) in enumerate(zip((*outs, *grads), (*one, *grad))):
            assert_bit_equal(a[rows][1:], b[1:], f"world {w} output {k}")


def pile(seed):
    """32 spheres and boxes, overlapping by a few centimetres on a floor."""
    sc = scenes.mixed_field(32, seed)
    sc.pos[1:] *= np.float32([0.64, 0.6, 0.64])
    return sc


def test_several_manifolds_a_group_as_one_a_group(gpu):
    """The same piles in blocks of 128 threads (more manifolds than groups of
    lanes: their adjoints wait in memory) and alone in blocks of 256 (a group for
    each): the same states, and gradients that differ by the order of the sums
    over a body's manifolds alone: eight terms of 6e-8, grown by the two steps'
    condition of 100."""
    sc = many(gpu, 33, pile)
    assert all(s.count <= 33 for s in sc)
    n = sc[0].count
    _, _, d, outs, grads = run(sc, 2, 2, 8, per_body=8)
    batch = gpu.GpuBatch(sc, iterations=8)
    batch.step(1 / 120, 2)
    for k, (o, r) in enumerate(zip(outs, batch.bodies())):
        assert_bit_equal(o, r, f"state {k}")
    compared = 0
    for w in range(0, len(sc), 10):
        st = batch.stats(w)
        if not (32 < st["contact_count"] <= 64 and st["color_count"] > 2):
            continue
        compared += 1
        rows = slice(w * n, (w + 1) * n)
        _, _, _, one, grad = run([sc[w]], 2, 2, 8, [a[rows] for a in d], per_body=8)
        for k, (a, b) in enumerate(zip(outs, one)):
            assert_bit_equal(a[rows], b, f"world {w} state {k}")
        for name, a, b in zip(NAMES, grads, grad):
            a = a[rows]
            assert np.all(np.isfinite(a)) and np.linalg.norm(a - b) <= 5e-5 * max(np.linalg.norm(b), 1e-6), (w, name)
    assert compared >= 3


def test_adjoint_of_a_pile_against_fp64(gpu):
    """Ninety spheres overlapping by a few centimetres on a floor (contacts without
    discrete choices): several colours, more manifolds than the block has groups
    of lanes.  Gradients of two steps against the FP64 adjoint, to the 1e-3 that
    this adjoint is held to elsewhere."""
    from phys_gb300 import rollout

    rng = np.random.default_rng(8)
    k = np.arange(90)
    sc = boxes_on_floor(90, 3)
    sc.shape[1:] = 0
    sc.dims[1:] = [0.5, 0.0, 0.0]
    top = sc.pos[0, 1] + 0.5 * sc.dims[0, 1]
    at = np.stack([k % 6, k // 36, k // 6 % 6], 1) * [0.97, 0.96, 0.97] + rng.uniform(-0.02, 0.02, (90, 3))
    sc.pos[1:] = (at + [-2.4, top + 0.47, -2.4]).astype(np.float32)
    sc.linvel[:] = 0.0
    sc.linvel[1:] = rng.normal(0.0, 0.1, (90, 3)).astype(np.float32)
    roll, start, d, outs, grads = run([sc], 2, 2, 8, per_body=8)
    batch = gpu.GpuBatch([sc], iterations=8)
    batch.step(1 / 120, 2)
    st = batch.stats(0)
    assert st["contact_count"] > 128 and st["color_count"] > 4
    for i, (o, r) in enumerate(zip(outs, batch.bodies())):
        assert_bit_equal(o, r, f"state {i}")
    _, iinv, he = rollout.body_properties(sc)
    _, ref = rollout.fp64_rollout(sc.shape, sc.is_static, he, iinv, start, roll.mass, roll.friction, roll.restitution,
                                  2, 1 / 120, 8, d_final=d)
    dyn = ~sc.is_static.astype(bool)
    for name, g, r in zip(NAMES, grads, ref):
        assert np.linalg.norm(g[dyn] - r[dyn]) <= 1e-3 * max(np.linalg.norm(r[dyn]), 1e-6), name
