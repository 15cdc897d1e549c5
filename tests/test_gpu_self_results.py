"""Contact results that a caller sets with one body on both sides: the solver takes them in their place in
the order, the two sides from the same velocities, and keeps side b's.  Held against the oracle with a
second body like the first on side a."""
import copy

import numpy as np
import pytest

import orc
import pe_gb300 as pg
from test_gpu_island_flow import _gpu, _islands

pytestmark = pytest.mark.gpu

BODY = ("body_shape", "body_flags", "mass", "friction", "restitution", "lin_damp", "ang_damp", "origin", "basis", "lin_vel", "ang_vel")


def _with_self_results(sizes, bits, seed):
    """A world's results with results of a body with itself before them, on one body of every island, and the
    same with another body like it on side a."""
    scene, res = _islands(sizes, bits, seed, iterations=1)
    _, more = _islands([1] * len(sizes), bits, seed + 1)
    a, b = res["res_a"], res["res_b"]
    label = np.arange(scene.n_bodies)
    for _ in range(200):   # the smallest body of each island
        for p, q in zip(a, b):
            if p and q:
                label[p] = label[q] = min(label[p], label[q])
    on = np.unique(label[1:])[:len(sizes)].astype(np.int32)
    both = {k: np.concatenate([more[k][:len(on)], res[k]]) for k in res}
    both["res_a"][:len(on)] = both["res_b"][:len(on)] = on
    twin = dict(both, res_a=both["res_a"].copy())
    twin["res_a"][:len(on)] = scene.n_bodies + np.arange(len(on))
    wide = copy.deepcopy(scene)
    for f in BODY:
        v = getattr(wide, f)
        setattr(wide, f, np.concatenate([v, v[on]]))
    return scene, both, wide, twin


@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("mode", [pg.SERIAL_ORDER, pg.COLORED])
@pytest.mark.parametrize("sizes", [[1, 2, 3, 7, 15, 31], [32, 64, 700], [1, 5, 2100]], ids=["warp", "grid", "large"])
def test_results_of_a_body_with_itself(sizes, mode, bits):
    scene, both, wide, twin = _with_self_results(sizes, bits, seed=sum(sizes))
    o = orc.OracleWorld(wide, bits)
    o.set_results(twin)
    o.solve()
    want = o.state()
    for tuning in (None, dict(small_island_items=1, big_island_items=8)):
        got, _ = _gpu(scene, both, bits, mode, tuning)
        for k in ("lin_vel", "ang_vel"):
            np.testing.assert_array_equal(got[k], want[k][:scene.n_bodies], err_msg=k)


@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("iterations", [0, 1, 6])
def test_modes_agree_on_results_of_a_body_with_itself(iterations, bits):
    """Over several iterations, in a warp and over the grid."""
    scene, both, _, _ = _with_self_results([6, 20], bits, seed=4)
    scene.iterations = iterations
    ref, _ = _gpu(scene, both, bits, pg.SERIAL_ORDER)
    for mode in (pg.SERIAL_ORDER, pg.COLORED):
        for big in (2, 9, 4096):
            got, _ = _gpu(scene, both, bits, mode, dict(small_island_items=1, big_island_items=big))
            for k in ("lin_vel", "ang_vel"):
                np.testing.assert_array_equal(got[k], ref[k], err_msg=f"{mode} {big}: {k}")


@pytest.mark.parametrize("m", [1, 2, 40, 2500])
def test_world_of_one_body(m):
    """All results are one island there, however many: its items in order."""
    scene, both, _, _ = _with_self_results([1], 32, seed=8)
    keep = 1   # the only dynamic body
    for f in BODY:
        setattr(scene, f, getattr(scene, f)[keep:keep + 1])
    r = np.random.default_rng(m)
    at = r.integers(0, len(both["res_a"]), m)
    res = {k: v[at] for k, v in both.items()}
    res["res_a"] = res["res_b"] = np.zeros(m, np.int32)
    for mode in (pg.SERIAL_ORDER, pg.COLORED):
        got, n = _gpu(scene, res, 32, mode)
        assert (n["islands"], n["active"]) == (1, m)
        ref, _ = _gpu(scene, res, 32, pg.SERIAL_ORDER, dict(small_island_items=0, big_island_items=1))
        for k in ("lin_vel", "ang_vel"):
            np.testing.assert_array_equal(got[k], ref[k])
