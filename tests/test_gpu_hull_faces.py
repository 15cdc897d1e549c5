"""Cylinders and spheres against hulls, piece by piece: hulls with fewer and more than 32 faces, with more
reached faces than one round takes, faces of up to 24 edges, a cylinder's axis along a face's normal
(six segments instead of four), either body first.  Contacts are the oracle's, bit for bit."""
import numpy as np
import pytest

import orc
import pe_gb300 as pg
from pe_gb300 import scene as sc
from pe_testlib import compare_results

pytestmark = pytest.mark.gpu


def _prism(n, radius, half):
    """A prism with two faces of n corners and n sides of four."""
    a = 2 * np.pi * np.arange(n) / n
    ring = np.stack([radius * np.cos(a), np.zeros(n), radius * np.sin(a)], 1)
    v = np.concatenate([ring + (0, half, 0), ring - (0, half, 0)])
    faces = [list(range(n))[::-1], list(range(n, 2 * n))]
    faces += [[i, (i + 1) % n, n + (i + 1) % n, n + i] for i in range(n)]
    return v, faces


def _shape(sb, r, kind):
    if kind == "sphere":
        return sb.shape(sc.SPHERE, (r.uniform(0.3, 1.2), 0, 0))
    if kind == "cyl":
        return sb.shape(sc.CYLINDER, (r.uniform(0.2, 0.9), r.uniform(0.3, 2.0)))
    if kind.startswith("prism"):
        return sb.shape(sc.HULL, hull=_prism(int(kind[5:]), r.uniform(0.4, 0.9), r.uniform(0.2, 0.6)))
    return sb.shape(sc.HULL, hull=sc.random_hull(r, int(kind), r.uniform(0.4, 1.0)))


@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("hull", ["4", "12", "19", "64", "prism3", "prism12", "prism13", "prism24"])
@pytest.mark.parametrize("other", ["cyl", "sphere"])
def test_against_the_oracle(other, hull, bits):
    r = np.random.default_rng(len(hull) * 7 + len(other))
    sb = sc.SceneBuilder(dt=1.0 / 60.0, gravity=(0.0, 0.0, 0.0), iterations=2)
    for i in range(30):
        c = np.array([20.0 * i, 0.0, 0.0])
        d = r.normal(size=3)
        d *= (0.05, 0.5, 0.9, 1.2, 1.6)[i % 5] / np.linalg.norm(d)
        ra, rb = sc.random_rotations(r, 2)
        if i % 3 == 0:   # upright on a face
            ra = rb = np.eye(3)
            d = np.array([0.0, d[1], 0.1])
        kinds = (other, hull) if i % 2 else (hull, other)
        sb.body(_shape(sb, r, kinds[0]), c, ra, mass=1.0)
        sb.body(_shape(sb, r, kinds[1]), c + d, rb, mass=1.0)
    s = sb.build(bits)
    g, o = pg.GpuWorld(s, bits), orc.OracleWorld(s, bits)
    pairs = np.array([[2 * i, 2 * i + 1] for i in range(30)], np.int32)
    for w in (g, o):
        w.integrate()
        w.broadphase()
        w.set_pairs(pairs)
        w.narrowphase()
    compare_results(g.results(), o.results(), what=f"{other}-{hull}")
    assert o.results()["point_size"].sum() > 0
