"""The solver's islands on the GPU against the oracle, bit for bit, where the island kernels change: at
the edges of the size classes that share a warp (1, 2, 4, 8, 16, 32 items and one more), above them
(the grid-wide kernel), with bodies held by one, two and many items, with kinematic partners and with
one to eight points; and the first-fit order of coloured islands above the exact levels against a
colouring by rounds restated here."""
import numpy as np
import pytest

import orc
import pe_gb300 as pg
from pe_gb300 import scene as sc

pytestmark = pytest.mark.gpu


def _islands(sizes, bits, seed, iterations=7):
    """A world of boxes and the contact results that make one island of each size (in items)."""
    r = np.random.default_rng(seed)
    sb = sc.SceneBuilder(dt=1.0 / 60.0, iterations=iterations)
    sb.body(sb.shape(sc.BOX, (50.0, 1.0, 50.0)), (0.0, -0.5, 0.0), mass=0.0, kinematic=True)
    box = sb.shape(sc.BOX, (1.0, 0.7, 0.9))
    pairs = []
    for m in sizes:
        n = max(1, int(r.integers(m // 3 + 1, m + 2)))
        ids = [sb.body(box, r.uniform(-5, 5, 3), sc.random_rotations(r, 1)[0], mass=float(r.uniform(1, 4)), v=r.normal(size=3),
                       w=r.normal(size=3)) for _ in range(n)]
        links = [(ids[i], ids[int(r.integers(max(0, i - 3), i))]) for i in range(1, n)]   # a tree joins the island
        while len(links) < m:
            a, b = (ids[int(r.integers(n))] for _ in range(2))
            links.append((a, 0) if a == b or n == 1 else (a, b))
        links = links[:m]
        pairs += [p if r.random() < 0.5 else p[::-1] for p in (links[i] for i in r.permutation(m))]
    pairs = [pairs[i] for i in r.permutation(len(pairs))]   # islands interleaved, as pairs come
    scene = sb.build(bits)
    R = len(pairs)
    np_ = r.integers(1, 9, R).astype(np.int32)
    nrm = r.normal(size=(R, 8, 3))
    nrm /= np.linalg.norm(nrm, axis=2, keepdims=True)
    t0 = np.cross(nrm, r.normal(size=(R, 8, 3)))
    t0 /= np.linalg.norm(t0, axis=2, keepdims=True)
    slots = np.concatenate([r.normal(size=(R, 8, 3)), nrm, r.uniform(-.5, .5, (R, 8, 6)), -r.uniform(0, .01, (R, 8, 1)), t0,
                            np.cross(nrm, t0)], axis=2)
    real = np.float32 if bits == 32 else np.float64
    slots = slots.astype(real).astype(np.float64)
    for k in range(R):   # slots past the points carry their distance only
        slots[k, np_[k]:] = 0.0
    p = np.array(pairs, np.int32)
    res = dict(res_a=p[:, 0].copy(), res_b=p[:, 1].copy(), point_size=np_, friction=r.uniform(0.2, 0.8, R).astype(real).astype(np.float64),
               restitution=r.uniform(0, 0.3, R).astype(real).astype(np.float64), slots=slots)
    return scene, res


def _gpu(scene, res, bits, mode, tuning=None):
    g = pg.GpuWorld(scene, bits, tuning=tuning)
    g.set_results(res)
    g.solve(mode)
    st, n = g.state(fields=("lin_vel", "ang_vel")), g.last_counts()
    g.close()
    return st, n


def _oracle(scene, res, bits):
    o = orc.OracleWorld(scene, bits)
    o.set_results(res)
    o.solve()
    return o.state()


def _same(a, b):
    for k in ("lin_vel", "ang_vel"):
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)


EDGES = [1, 1, 1, 2, 2, 3, 4, 5, 8, 9, 16, 17, 31, 32]


@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("mode", [pg.SERIAL_ORDER, pg.COLORED])
@pytest.mark.parametrize("sizes", [EDGES, [33], EDGES * 3 + [33, 64, 65, 700], [1] * 70 + [6000]], ids=["warp", "33", "mixed", "large"])
def test_gpu_islands_match_oracle(bits, mode, sizes):
    scene, res = _islands(sizes, bits, seed=len(sizes) + bits)
    ref = _oracle(scene, res, bits)
    st, n = _gpu(scene, res, bits, mode)
    _same(st, ref)
    assert n["islands"] == len(sizes) and n["active"] == sum(sizes)


@pytest.mark.parametrize("iterations", [0, 1])
def test_gpu_islands_few_iterations(iterations):
    scene, res = _islands([1, 3, 40], 32, seed=3, iterations=iterations)
    ref = _oracle(scene, res, 32)
    for mode in (pg.SERIAL_ORDER, pg.COLORED):
        _same(_gpu(scene, res, 32, mode)[0], ref)


def _rounds(a, b, kinematic):
    """(levels, first-fit colours) of one island's items: in every round, an item that is the first of
    those left on its dynamic bodies takes the smallest colour that neither body holds yet."""
    held, level, color = {}, {}, np.zeros(len(a), int)
    depth = 0
    for j in range(len(a)):   # item order meets the rounds' winners body by body
        mine = [x for x in (a[j], b[j]) if not kinematic[x]]
        lev = max([level.get(x, 0) for x in mine], default=0) + 1
        used = set().union(*[held.setdefault(x, set()) for x in mine]) if mine else set()
        color[j] = next(c for c in range(len(a) + 1) if c not in used)
        for x in mine:
            held[x].add(color[j])
            level[x] = lev
        depth = max(depth, lev)
    return depth, color


@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("m", [9, 30, 900])
def test_gpu_first_fit_order(bits, m):
    scene, res = _islands([m], bits, seed=m)
    a, b = res["res_a"], res["res_b"]
    depth, color = _rounds(a, b, np.asarray(scene.body_flags) != 0)
    order = np.lexsort((np.arange(m), color))
    by_color = {k: v[order] for k, v in res.items()}
    tuning = dict(small_island_items=1, big_island_items=8, exact_levels_colored=depth - 1)
    st, n = _gpu(scene, res, bits, pg.COLORED, tuning)
    _same(st, _oracle(scene, by_color, bits))
    assert n["colors"] == min(int(color.max()) + 1, depth)
    st, n = _gpu(scene, res, bits, pg.COLORED, dict(tuning, exact_levels_colored=depth))   # within the exact levels
    _same(st, _oracle(scene, res, bits))
    assert n["colors"] == depth
