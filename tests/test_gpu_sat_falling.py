"""Pairs whose deepest-going axis is a face axis along which the reference passes over a run of the first
shape's vertices (their projections fall one after the other, and a new minimum never becomes its
maximum): the depth it computes there is below the true one and decides the pair.  The staged SAT may not
skip such an axis; its results are the oracle's, bit for bit."""
import numpy as np
import pytest
from scipy.spatial import ConvexHull

import orc
import pe_gb300 as pg
from pe_gb300 import scene as sc
from pe_testlib import compare_results

pytestmark = pytest.mark.gpu


def _hull_interval(v, b, o, axes):
    """(min, the reference's max, the true max) of a hull along each axis."""
    p = (axes @ b) @ v.T
    low = np.minimum.accumulate(p, axis=1)
    falls = np.concatenate([np.ones((len(p), 1), bool), p[:, 1:] < low[:, :-1]], axis=1)
    off = axes @ o
    return p.min(1) + off, np.where(falls, -1e30, p).max(1) + off, p.max(1) + off


def _decided_by_a_falling_run(r):
    """A hull (the first shape) and a box that such a face axis decides, by a margin; None if these are not."""
    v, f = sc.random_hull(r, int(r.integers(6, 14)), 0.6)
    v = np.asarray(v)
    ra, rb = sc.random_rotations(r, 2)
    half = r.uniform(0.15, 0.5, 3)
    # along the box's first axis the hull's upper vertices come first, one below the other
    up = v @ ra.T @ rb[:, 0]
    run = [int(i) for i in np.argsort(-up) if up[i] > r.uniform(-0.3, 0.2)]
    order = run + [i for i in range(len(v)) if i not in run]
    v, place = v[order], np.argsort(order)
    f = [[int(place[i]) for i in q] for q in f]
    if len(v) - len(run) < 2:
        return None
    balls = half.min() - ConvexHull(v[1:]).equations[:, 3].max()   # the inner balls: deeper pairs skip nothing
    d = rb[:, 1] * r.uniform(0.4, 0.9) + rb[:, 0] * r.uniform(0, 0.1) + rb[:, 2] * r.uniform(-0.1, 0.1)
    n = [np.cross(v[q[1]] - v[q[0]], v[q[2]] - v[q[0]]) for q in f]
    faces = np.array([ra @ (a / np.linalg.norm(a)) for a in n] + [rb[:, k] for k in range(3)])
    e = {tuple(sorted((q[i], q[(i + 1) % len(q)]))) for q in f for i in range(len(q))}
    x = np.array([np.cross(ra @ (v[a] - v[b]), rb[:, k]) for a, b in e for k in range(3)])
    size = np.linalg.norm(x, axis=1)
    edges = x[size > 1e-3] / size[size > 1e-3][:, None]

    def depths(axes):
        axes = np.where((axes @ d)[:, None] < 0, -axes, axes)
        lo, hi, top = _hull_interval(v, ra, d, axes)
        he = np.abs(axes @ rb) @ half
        return np.minimum(hi + he, he - lo), np.minimum(top + he, he - lo), (hi < -he) | (he < lo)

    df, true, apart = depths(faces)
    de, _, apart_e = depths(edges)
    if true.min() > balls - 0.05 or apart.any() or apart_e.any() or df.min() > true.min() - 0.02 or de.min() < df.min() + 0.02:
        return None
    return (v, f), ra, d, half, rb


@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("heavy", [1, 100000000])
def test_face_axis_of_a_falling_run(bits, heavy):
    r = np.random.default_rng(5)
    sb = sc.SceneBuilder(dt=1.0 / 60.0, gravity=(0.0, 0.0, 0.0), iterations=2)
    n = 0
    for _ in range(1000):
        q = _decided_by_a_falling_run(r)
        if q is None:
            continue
        hull, ra, d, half, rb = q
        c = np.array([10.0 * n, 0.0, 0.0])
        sb.body(sb.shape(sc.HULL, hull=hull), c + d, ra, mass=1.0)
        sb.body(sb.shape(sc.BOX, 2 * half), c, rb, mass=1.0)
        n += 1
    assert n >= 8
    scene = sb.build(bits)
    g = pg.GpuWorld(scene, bits, tuning=dict(sat_heavy_cost=heavy))
    o = orc.OracleWorld(scene, bits)
    pairs = np.array([[2 * i, 2 * i + 1] for i in range(n)], np.int32)
    for w in (g, o):
        w.integrate()
        w.broadphase()
        w.set_pairs(pairs)
        w.narrowphase()
    compare_results(g.results(), o.results(), what="falling run")
    assert o.results()["point_size"].sum() > 0
