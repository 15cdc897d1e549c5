"""The staged SAT skips axes by bounds; its results on pairs where the bounds, the queues and the lists
change shape are the oracle's, bit for bit: hulls of the fewest and the most staged vertices, boxes much
wider than what touches them, flat boxes, cylinders upright on each other and across, pairs apart, barely
touching, deep and concentric, each with a warp and with a block per pair."""
import numpy as np
import pytest

import orc
import pe_gb300 as pg
from pe_gb300 import scene as sc
from pe_testlib import compare_results

pytestmark = pytest.mark.gpu


def _hull(r, n, scale):
    """A hull whose first two vertices lie inside it, where a projection never takes them as its
    maximum: on it the reference's projection is the support function in every direction."""
    v, f = sc.random_hull(r, n, scale)
    return np.concatenate([[[0.01 * scale, 0.0, 0.02 * scale], [0.0, 0.01 * scale, 0.0]], v]), [[i + 2 for i in t] for t in f]


def _pairs(kind, bits, seed):
    r = np.random.default_rng(seed)
    sb = sc.SceneBuilder(dt=1.0 / 60.0, gravity=(0.0, 0.0, 0.0), iterations=2)

    def shape(k):
        if k == "box":
            return sb.shape(sc.BOX, r.uniform(0.3, 1.6, 3) * r.choice([1.0, 0.2, 1.0], 3))
        if k == "floor":
            return sb.shape(sc.BOX, (40.0, 1.0, 40.0))
        if k == "cyl":
            return sb.shape(sc.CYLINDER, (r.uniform(0.2, 0.8), r.uniform(0.2, 2.0)))
        return sb.shape(sc.HULL, hull=_hull(r, int(k), r.uniform(0.3, 1.0)))

    a, b = kind.split("-")
    for i in range(24):
        c = np.array([60.0 * (i % 6), 0.0, 60.0 * (i // 6)])
        d = r.normal(size=3)
        d *= (0.0, 0.02, 0.4, 0.7, 1.0, 1.3)[i % 6] / np.linalg.norm(d)
        ra, rb = sc.random_rotations(r, 2)
        if i % 4 == 1:
            ra = rb = np.eye(3)   # faces and edges parallel
        if "floor" in (a, b):     # somewhere on the floor's top
            d, ra = np.array([r.uniform(-15, 15), 0.5 + (0.0, 0.1, 0.3, 0.5, 0.7, 1.2)[i % 6], r.uniform(-15, 15)]), np.eye(3)
            if b == "floor":
                d, ra, rb = -d, rb, np.eye(3)
        sb.body(shape(a), c, ra, mass=1.0)
        sb.body(shape(b), c + d, rb, mass=1.0)
    return sb.build(bits)


KINDS = ["box-4", "box-5", "6-box", "box-33", "62-box", "floor-4", "floor-30", "17-floor", "4-4", "6-34", "35-36", "62-62", "cyl-cyl"]


@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("heavy", [1, 100000000])
@pytest.mark.parametrize("kind", KINDS)
def test_gpu_sat_matches_oracle(bits, heavy, kind):
    scene = _pairs(kind, bits, seed=KINDS.index(kind))
    g = pg.GpuWorld(scene, bits, tuning=dict(sat_heavy_cost=heavy))
    o = orc.OracleWorld(scene, bits)
    for w in (g, o):
        w.integrate()
        w.broadphase()
    pairs = np.array([[2 * i, 2 * i + 1] for i in range(24)], np.int32)   # apart or not
    g.set_pairs(pairs)
    o.set_pairs(pairs)
    g.narrowphase()
    o.narrowphase()
    compare_results(g.results(), o.results(), what=kind)
    assert o.results()["point_size"].sum() > 0
