"""The hand-written reverse of the contact geometry and preparation (FP64, one
step) against central differences of the step itself, for every kind of contact:
sphere-sphere, sphere against a box from outside and from inside it, box faces,
box edges, and boxes without a kept vertex."""
import numpy as np
import pytest

from phys_gb300 import rollout

DT, ITERS, EPS = 1 / 120, 6, 1e-6
# Central differences at 1e-6 are off by about eps^2 times the third derivative
# (order 1e-10 here) and by the rounding of the two losses over 2 eps (1e-15 /
# 1e-6 = 1e-9 of the loss): 1e-5 of the largest gradient of its kind holds both
# with room for stiff contacts.
TOL = 1e-5


def quat(rng):
    q = rng.normal(size=4)
    return q / np.linalg.norm(q)


def pair(kind, rng):
    """shape, half extents, positions, rotations of an overlapping pair."""
    ident = np.array([0.0, 0, 0, 1])
    if kind == "spheres":
        return [0, 0], [[0.5, 0, 0], [0.4, 0, 0]], [np.zeros(3), 0.85 * unit(rng)], [quat(rng), quat(rng)]
    if kind in ("sphere_box", "box_sphere"):
        q, he = quat(rng), np.array([0.4, 0.5, 0.3])
        off = rotate(q, np.array([0.1, 0.05, he[2] + 0.25]))
        s, b = (0, [0.3, 0, 0], off, quat(rng)), (1, he, np.zeros(3), q)
    elif kind == "sphere_inside":
        q, he = quat(rng), np.array([0.4, 0.5, 0.3])
        s, b = (0, [0.2, 0, 0], rotate(q, np.array([0.1, 0.05, 0.22])), quat(rng)), (1, he, np.zeros(3), q)
    elif kind == "faces":
        q = quat(rng)
        turn = rotate_vec_quat(np.array([0.03, -0.02, 0.05]))
        s = (1, [0.3, 0.35, 0.25], rotate(q, np.array([0.1, 0.08, 0.52])), mul(q, turn))
        b = (1, [0.5, 0.6, 0.3], np.zeros(3), q)
    else:
        # two rods that cross at an angle: an edge axis, or no vertex inside
        a = rotate_vec_quat(np.array([np.pi / 4, 0, 0]))  # edge up, along x
        c = mul(rotate_vec_quat(np.array([0, 0.9, 0])), mul(rotate_vec_quat(np.array([0.0, np.pi / 2, 0.0])), a))
        # turned as a whole: along the world's axes the contact's tangents lie on
        # the boxes' own axes, where their projected radii have kinks
        q = quat(rng)
        s = (1, [1.0, 0.2, 0.2], np.zeros(3), mul(q, a))
        b = (1, [1.0, 0.2, 0.2], rotate(q, np.array([0.07, 0.53, 0.04])), mul(q, c))
    if kind == "box_sphere":
        s, b = b, s
    return [s[0], b[0]], [s[1], b[1]], [s[2], b[2]], [s[3], b[3]]


def unit(rng):
    v = rng.normal(size=3)
    return v / np.linalg.norm(v)


def mul(a, b):
    x1, y1, z1, w1 = a
    x2, y2, z2, w2 = b
    return np.array([w1 * x2 + x1 * w2 + y1 * z2 - z1 * y2, w1 * y2 - x1 * z2 + y1 * w2 + z1 * x2,
                     w1 * z2 + x1 * y2 - y1 * x2 + z1 * w2, w1 * w2 - x1 * x2 - y1 * y2 - z1 * z2])


def rotate_vec_quat(r):
    angle = np.linalg.norm(r)
    return np.append(np.sin(angle / 2) * r / angle, np.cos(angle / 2))


def rotate(q, v):
    return mul(mul(q, np.append(v, 0.0)), q * np.array([-1, -1, -1, 1.0]))[:3]


@pytest.mark.parametrize("kind", ["spheres", "sphere_box", "box_sphere", "sphere_inside", "faces", "rods"])
@pytest.mark.parametrize("seed", [1, 2, 3])
def test_reverse_of_one_contact_matches_central_differences(kind, seed):
    rng = np.random.default_rng(seed)
    shape, he, pos, rot = pair(kind, rng)
    shape = np.array(shape, np.uint8)
    he = np.array(he, np.float64)
    toward = np.array(pos[1]) - np.array(pos[0])
    toward /= np.linalg.norm(toward)
    x, q = np.array(pos, np.float64), np.array(rot, np.float64)
    v = np.array([1.6 * toward, -1.4 * toward]) + rng.normal(0, 0.1, (2, 3))  # fast enough for restitution
    w = rng.normal(0, 0.3, (2, 3))
    mass, iinv = np.array([1.3, 0.8]), rng.uniform(0.8, 2.0, (2, 3))
    mu, rest = np.array([0.4, 0.6]), np.array([0.1, 0.3])
    static = np.zeros(2, np.uint8)
    d = [rng.normal(size=s) for s in ((2, 3), (2, 4), (2, 3), (2, 3))]

    def run(args, grad=False):
        x_, q_, v_, w_, m_, f_, r_ = args
        return rollout.fp64_rollout(shape, static, he, iinv, (x_, q_, v_, w_), m_, f_, r_, 1, DT, ITERS,
                                    gravity=(0.0, 0.0, 0.0), d_final=d if grad else None)

    def loss(args):
        out, _ = run(args)
        return sum(float((a * b).sum()) for a, b in zip(d, out))

    args = [x, q, v, w, mass, mu, rest]
    free = x + v * DT
    assert np.abs(run(args)[0][0] - free).max() > 1e-4  # they touch
    _, grads = run(args, grad=True)
    for k, g in enumerate(grads):
        scale = max(np.abs(g).max(), 1e-3)
        if k == 1:
            # a rotation is perturbed by turning it: off the unit sphere a box's
            # support along its own face axis is a tie between four corners
            steps = [(b, np.eye(3)[j]) for b in range(2) for j in range(3)]
            moves = [(b, lambda a, sign, b=b, e=e: a.__setitem__(b, mul(rotate_vec_quat(sign * EPS * e), a[b])),
                      float(g[b] @ mul(np.append(e / 2, 0.0), q[b]))) for b, e in steps]
        else:
            moves = [(i, lambda a, sign, i=i: a.__setitem__(i, a[i] + sign * EPS), g[i]) for i in np.ndindex(g.shape)]
        for i, move, expected in moves:
            ends = []
            for sign in (1.0, -1.0):
                moved = [a.copy() for a in args]
                move(moved[k], sign)
                ends.append(loss(moved))
            assert abs((ends[0] - ends[1]) / (2 * EPS) - expected) <= TOL * scale, (kind, "xqvwmfr"[k], i)
