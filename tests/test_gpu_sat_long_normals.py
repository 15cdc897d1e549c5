"""Cylinder pairs where one cylinder's axis is perpendicular to, or along, a face normal of the other's mesh:
there the reference projects a cylinder by its radius or half height whatever the axis's length, and one
normal of the mesh is 1.9 % longer than 1.  Such a face axis may not be skipped by a bound that grows with
the length; results are the oracle's, bit for bit, separations among them."""
import numpy as np
import pytest

import orc
import pe_gb300 as pg
from pe_gb300 import scene as sc
from pe_testlib import compare_results

pytestmark = pytest.mark.gpu

# face normals of the cylinder mesh: the caps, 20 sides that rise and 20 that fall; the seventh of the
# rising ones is the long one
RING = np.deg2rad(18 * np.arange(20))
RISE = np.stack([0.98767 * np.cos(RING + np.pi / 20), np.full(20, 0.006156), -0.98767 * np.sin(RING + np.pi / 20)], 1)
FALL = np.stack([0.999981 * np.cos(RING), np.full(20, -0.006156), -0.999981 * np.sin(RING)], 1)
LONG = np.array([-0.493982, 0.006156, -0.890990])
NORMALS = np.concatenate([[[0, 1, 0], [0, -1, 0]], RISE, FALL])
NORMALS[8] = LONG


def _turned(r, y):
    """A random rotation that takes the cylinder's axis to the unit vector y."""
    x = np.cross(y, r.normal(size=3))
    x /= np.linalg.norm(x)
    return np.stack([x, y, np.cross(x, y)], 1)


def _pairs(bits, place, m, seed):
    r = np.random.default_rng(seed)
    sb = sc.SceneBuilder(dt=1.0 / 60.0, gravity=(0.0, 0.0, 0.0), iterations=2)
    for i in range(m):
        own, other = sc.random_rotations(r, 1)[0], None
        n = own @ (LONG if i % 4 else NORMALS[int(r.integers(42))])
        u = n / np.linalg.norm(n)
        across = np.cross(u, r.normal(size=3))
        across /= np.linalg.norm(across)
        other = _turned(r, across if place == "across" else u * r.choice([-1.0, 1.0]))
        size = r.uniform(0.3, 0.8, 2)
        h_own = r.uniform(0.6, 2.0)
        h_other = r.uniform(0.6, 2.0)
        reach = size[1] if place == "across" else h_other / 2
        d = u + np.cross(u, r.normal(size=3)) * r.uniform(0.0, 0.08)   # roughly along the normal
        d *= (size[0] + reach * (1.0 - r.uniform(0.0, 0.03))) / np.linalg.norm(d)
        c = np.array([10.0 * (i % 40), 0.0, 10.0 * (i // 40)])
        bodies = [(sb.shape(sc.CYLINDER, (size[0], h_own)), c, own), (sb.shape(sc.CYLINDER, (size[1], h_other)), c + d, other)]
        for shape, o, b in bodies if r.random() < 0.5 else bodies[::-1]:   # either of the two may be the first
            sb.body(shape, o, b, mass=1.0)
    return sb.build(bits)


@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("heavy", [1, 100000000])
@pytest.mark.parametrize("place", ["across", "along"])
def test_cylinders_at_a_long_face_normal(bits, heavy, place):
    m = 1200
    scene = _pairs(bits, place, m, seed=11)
    g = pg.GpuWorld(scene, bits, tuning=dict(sat_heavy_cost=heavy))
    o = orc.OracleWorld(scene, bits)
    pairs = np.array([[2 * i, 2 * i + 1] for i in range(m)], np.int32)
    for w in (g, o):
        w.integrate()
        w.broadphase()
        w.set_pairs(pairs)
        w.narrowphase()
    n = o.results()["point_size"]
    assert (n > 0).sum() > m // 20 and (n == 0).sum() > m // 20
    compare_results(g.results(), o.results(), what=place)
