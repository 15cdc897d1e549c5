"""Pairs with a concave mesh or a compound run piece by piece in a warp: pieces with more points than a
recorder holds (faces of 32 vertices under a wide cylinder), pairs of more pieces than a warp has lanes,
compounds against compounds, hulls and meshes, against the oracle bit for bit; and the boxes of meshes
above the vertex count that a warp shares, in worlds whose last warp is partly empty."""
import numpy as np
import pytest

import orc
import pe_gb300 as pg
from pe_gb300 import scene as sc

pytestmark = pytest.mark.gpu


def _polygon_floor(n, radius):
    """A concave mesh of one n-vertex face (up) and a ring of triangles below it."""
    ang = 2 * np.pi * np.arange(n) / n
    top = np.stack([radius * np.cos(ang), np.zeros(n), -radius * np.sin(ang)], 1)
    return np.concatenate([top, [[0, -1.0, 0]]]), [list(range(n))] + [[(k + 1) % n, k, n] for k in range(n)]


def _phase_equal(scene, bits, steps=6):
    g, o = pg.GpuWorld(scene, bits), orc.OracleWorld(scene, bits)
    for _ in range(steps):
        g.step(1, pg.SERIAL_ORDER)
        o.step(1)
        a, b = g.results(), o.results()
        for k in ("res_a", "res_b", "point_size", "friction", "restitution"):
            np.testing.assert_array_equal(a[k], b[k], err_msg=k)
        for r, n in enumerate(b["point_size"]):
            np.testing.assert_array_equal(a["slots"][r, :n], b["slots"][r, :n], err_msg=f"result {r}")
        sa, sb = g.state(), o.state()
        for k in ("origin", "basis", "lin_vel", "ang_vel", "aabb_min", "aabb_max"):
            np.testing.assert_array_equal(sa[k], sb[k], err_msg=k)
    return o.results()["point_size"]


@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("n", [3, 12, 13, 32])
def test_gpu_wide_faces_overflow_recorders(bits, n):
    sb = sc.SceneBuilder(dt=1.0 / 60.0, iterations=4)
    sb.body(sb.shape(sc.CONCAVE, hull=_polygon_floor(n, 1.0)), (0, 0, 0), mass=0.0, kinematic=True)
    for k, (shape, p) in enumerate(((sc.CYLINDER, (1.6, 0.6)), (sc.BOX, (0.9, 0.5, 0.9)), (sc.SPHERE, (0.5,)))):
        sb.body(sb.shape(shape, p), (0.05 * k, 0.27 + 0.9 * k, 0.02 * k), sc._rot((0.3, 0.1, 1.0) / np.sqrt(1.1), 0.04 * (k + 1)), mass=2.0)
    assert _phase_equal(sb.build(bits), bits).sum() > 0


@pytest.mark.parametrize("bits", [32, 64])
def test_gpu_compounds_of_many_pieces(bits):
    r = np.random.default_rng(5)
    sb = sc.SceneBuilder(dt=1.0 / 60.0, iterations=4)
    hv, hf = sc.heightfield(24, 24, cell=0.3, seed=2)
    sb.body(sb.shape(sc.CONCAVE, hull=(hv, hf)), (0, 0, 0), mass=0.0, kinematic=True)
    parts = [sb.shape(sc.BOX, (0.6, 0.3, 0.4)), sb.shape(sc.SPHERE, (0.3,)), sb.shape(sc.CYLINDER, (0.25, 0.7)),
             sb.shape(sc.HULL, hull=sc.random_hull(r, 14, 0.4))]
    for k in range(5):
        kids = [(parts[int(r.integers(4))], r.uniform(-0.7, 0.7, 3), sc.random_rotations(r, 1)[0], 1.0 / 7) for _ in range(7)]
        c = sb.compound(kids)
        sb.body(c, np.array([0.7 * (k % 3) - 0.7, 0.9 + 0.8 * (k // 3), 0.5 * k - 1.0]) - sb.compound_centroid(c), mass=3.0)
    for k, s in enumerate(parts):
        sb.body(s, (0.8 * k - 1.2, 1.6, 0.4 * k - 0.6), sc.random_rotations(r, 1)[0], mass=1.0)
    assert _phase_equal(sb.build(bits), bits).sum() > 20


@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("bodies", [1, 3, 32, 35])
def test_gpu_boxes_of_large_meshes(bits, bodies):
    r = np.random.default_rng(bodies)
    sb = sc.SceneBuilder(dt=1.0 / 60.0, gravity=(0.0, 0.0, 0.0), iterations=1)
    shapes = [sb.shape(sc.HULL, hull=sc.random_hull(r, nv, 1.0)) for nv in (96, 97, 200)]
    shapes.append(sb.shape(sc.CONCAVE, hull=sc.heightfield(9, 13, seed=1)))
    for k in range(bodies):
        s = shapes[(k + bodies - 1) % 4]
        sb.body(s, r.uniform(-1, 1, 3) + (0, 0, 40.0 * k), sc.random_rotations(r, 1)[0], mass=1.0, v=r.normal(size=3), w=r.normal(size=3))
    _phase_equal(sb.build(bits), bits, steps=2)
