"""Islands from the contact graph at the sizes where the kernels change: items that fit one block and
one more, one tile of a scan and one more, small and big radix tiles, sorts whose passes need their
own offsets kernel; labels of one, two and three digits; kinematic partners, results without points,
joints.  Solved velocities against the oracle, bit for bit, and the counters against a count here."""
import numpy as np
import pytest

import orc
import pe_gb300 as pg
from pe_gb300 import scene as sc

pytestmark = pytest.mark.gpu


def _graph(n, links, seed, joints=0, empty=0.2, bits=32):
    """n bodies of one shape (body 0 kinematic) and `links` results in random order: islands of up to
    some tens of items, some results without points."""
    r = np.random.default_rng(seed)
    m = n - 1
    s = sc.Scene(dt=1.0 / 60.0, iterations=3)
    s.shape_type, s.shape_param = np.zeros(1, np.int32), np.ones((1, 3))
    s.hull_vbeg = s.hull_vcnt = s.hull_fbeg = s.hull_fcnt = np.zeros(1, np.int32)
    s.hull_verts, s.hull_face_off, s.hull_face_idx = np.zeros((0, 3)), np.zeros(1, np.int32), np.zeros(0, np.int32)
    s.body_shape, s.body_flags = np.zeros(n, np.int32), np.array([sc.KINEMATIC] + [0] * m, np.int32)
    s.mass = np.concatenate([[0.0], r.uniform(1, 4, m)])
    s.friction, s.restitution = np.full(n, 0.5), np.zeros(n)
    s.lin_damp, s.ang_damp = np.zeros(n), np.zeros(n)
    s.origin, s.basis = r.uniform(-5, 5, (n, 3)), sc.random_rotations(r, n)
    moves = np.arange(n)[:, None] > 0
    s.lin_vel, s.ang_vel = np.where(moves, r.normal(size=(n, 3)), 0.0), np.where(moves, r.normal(size=(n, 3)), 0.0)
    if joints:
        a = r.integers(1, n, joints)
        s.joint_type, s.joint_body = np.zeros(joints, np.int32), np.stack([a, np.where(a > 1, a - 1, 0)], 1).astype(np.int32)
        s.joint_flag, s.joint_real = np.zeros(joints, np.int32), np.zeros((joints, 15))
    s = s.rounded(bits) if bits == 32 else s
    group = 12                                    # links stay inside groups of bodies
    a = r.integers(1, n, links)
    b = np.minimum((a - 1) // group * group + 1 + r.integers(0, group, links), m)
    b = np.where((a == b) | (r.random(links) < 0.3), 0, b)
    np_ = np.where(r.random(links) < empty, 0, r.integers(1, 9, links)).astype(np.int32)
    nrm = r.normal(size=(links, 8, 3))
    nrm /= np.linalg.norm(nrm, axis=2, keepdims=True)
    t0 = np.cross(nrm, r.normal(size=(links, 8, 3)))
    t0 /= np.linalg.norm(t0, axis=2, keepdims=True)
    real = np.float32 if bits == 32 else np.float64
    slots = np.concatenate([r.normal(size=(links, 8, 3)), nrm, r.uniform(-.5, .5, (links, 8, 6)), -r.uniform(0, .01, (links, 8, 1)), t0,
                            np.cross(nrm, t0)], axis=2).astype(real).astype(np.float64)
    slots[np.arange(8)[None, :] >= np_[:, None]] = 0.0
    res = dict(res_a=a.astype(np.int32), res_b=b.astype(np.int32), point_size=np_, friction=np.full(links, 0.5),
               restitution=np.zeros(links), slots=slots)
    return s, res


def _islands(s, res):
    import scipy.sparse as sp
    from scipy.sparse.csgraph import connected_components
    live = res["point_size"] > 0
    a, b = res["res_a"][live], res["res_b"][live]
    ja = s.joint_body.reshape(-1, 2) if len(s.joint_type) else np.zeros((0, 2), np.int32)
    a, b = np.concatenate([a, ja[:, 0]]), np.concatenate([b, ja[:, 1]])
    kin = s.body_flags > 0
    both = ~kin[a] & ~kin[b]
    n = len(kin)
    _, lab = connected_components(sp.coo_matrix((np.ones(both.sum()), (a[both], b[both])), (n, n)), directed=False)
    dyn = np.where(kin[a], b, a)
    return int(live.sum()), len(np.unique(lab[dyn]))


@pytest.mark.parametrize("n,links,joints", [(2, 1, 0), (40, 2047, 0), (255, 1024, 5), (257, 2048, 0), (300, 2040, 8), (300, 2049, 0),
                                            (8192, 1365, 1), (8192, 1365, 2), (8193, 1365, 0), (5000, 5461, 0), (9000, 16385, 7),
                                            (70000, 66000, 0), (150000, 180000, 0)])
def test_islands_against_the_oracle(n, links, joints):
    s, res = _graph(n, links, seed=n + links, joints=joints)
    g, o = pg.GpuWorld(s, 32), orc.OracleWorld(s, 32)
    g.set_results(res)
    o.set_results(res)
    g.solve(pg.SERIAL_ORDER)
    o.solve()
    got, want, c = g.state(), o.state(), g.last_counts()
    active, islands = _islands(s, res)
    assert (c["active"], c["islands"], c["rows"]) == (active, islands, int(res["point_size"].sum()))
    for k in ("lin_vel", "ang_vel"):
        assert np.array_equal(got[k], want[k]), k
    g.close()


@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("sizes", [(2500,), (1025, 3000, 2), (70000,)])
def test_body_sort_against_the_oracle(sizes, bits):
    """Scenes too large for the one-block sort, alone and several in a world (the scene is the last key)."""
    def one(n, seed):
        r = np.random.default_rng(seed)
        s, _ = _graph(n, 1, seed, bits=bits)
        o = r.uniform(-1, 1, (n, 3)) * (n ** (1 / 3))
        return sc.dataclasses.replace(s, origin=o.astype(np.float32).astype(np.float64), gravity=(0.0, 0.0, 0.0))
    parts = [one(n, 11 + k) for k, n in enumerate(sizes)]
    whole, offs = sc.concat(parts)
    g = pg.GpuWorld(whole, bits, scenes=offs)
    g.integrate()
    g.broadphase()
    got = g.pairs()
    want = []
    for k, p in enumerate(parts):
        o = orc.OracleWorld(p, bits, stable_ties=True)
        o.integrate()
        o.broadphase()
        want.append(o.pairs().reshape(-1, 2) + int(offs[k]))
    assert np.array_equal(got, np.concatenate(want))
    g.close()
