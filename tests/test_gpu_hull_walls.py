"""Container rows of hulls: vertices that lie on their bounding radius, with
orientations and container rotations of any length, and containers far from
the origin and turned against the axes."""
import numpy as np
import pytest

import oracle_lib as O
from diomedes_gb300 import abi, compute, physics as ph, scenes

pytestmark = pytest.mark.gpu

OCTAHEDRON = np.array([[1, 0, 0], [-1, 0, 0], [0, 1, 0], [0, -1, 0], [0, 0, 1], [0, 0, -1]], np.float32) * 0.5


def _hulls_at_walls(case):
    """96 octahedra of radius 0.5, each within 0.8 of one of the six walls."""
    rng = np.random.default_rng(7)
    quat = scenes.random_quats(rng, 96)
    turn, length, centre = np.array([0, 0, 0, 1.0]), np.ones(96), np.zeros(3)
    if case == "orientations":
        length = rng.uniform(0.85, 1.2, 96)
    elif case == "rotation":
        turn = np.array([0, 0, 0, 1.0]) * 1.14  # outward normals of length 1.3
    elif case == "far":
        turn, centre = np.array([0, np.sin(np.pi / 8), 0, np.cos(np.pi / 8)]), np.array([3.0e4, 0.0, -3.0e4])
    s = float(turn @ turn)
    half = 40.0
    items = []
    for k in range(96):
        axis, sign = k % 3, 1.0 if (k // 3) % 2 else -1.0
        p = rng.uniform(-20, 20, 3)
        p[axis] = sign * (half / s - rng.uniform(0.2, 0.8))
        world = centre + ph.quat_rotate(turn / np.sqrt(s), p)
        q = (quat[k] if k % 2 else np.array([0, 0, 0, 1.0])) * length[k]
        items.append(ph.hull(tuple(world), 0, OCTAHEDRON, 1.0, orientation=tuple(q),
                             velocity=tuple(rng.uniform(-1, 1, 3))))
    b, st = ph.pack_bodies(items)
    hv = np.zeros((6, 4), np.float32)
    hv[:, :3] = OCTAHEDRON
    return scenes.Scene(case, b, st, containers=[ph.container(tuple(centre), half, tuple(turn))], hull_vertices=hv,
                        options=ph.avbd_options(iterations=4))


@pytest.mark.parametrize("precision", [abi.PREC_F32, abi.PREC_SPLIT, abi.PREC_F64])
@pytest.mark.parametrize("case", ["unit", "orientations", "rotation", "far"])
def test_hulls_at_walls_match_oracle(case, precision):
    sc = _hulls_at_walls(case)
    ow = O.World(sc, precision=precision)
    cap = compute.capacity(sc.n, max_pairs=16 * sc.n, max_contacts=64 * sc.n, max_hull_vertices=6)
    rows = []
    with compute.World(cap, precision=precision) as w:
        w.upload(sc.bodies, sc.state, **sc.upload_kwargs())
        for _ in range(4):
            ow.step(sc.options, 1)
            w.step(sc.options, 1)
            for g, r in zip((*w.download(), w.contacts()), (*ow.download(), ow.contacts())):
                assert np.array_equal(np.ascontiguousarray(g).view(np.uint8), np.ascontiguousarray(r).view(np.uint8))
            rows.append(len(ow.contacts()))
    assert 0 < rows[0] < 96
