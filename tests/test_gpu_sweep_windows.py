"""Pair lists of the sweep against the oracle where its windows change hands: ends at
every edge of a warp's first chunks of 32 and of its groups of four, windows past the length that
blocks sweep in chunks, several scenes in one world (a window ends with its scene), and the sweep axis
that the next step takes, computed beside the rest of the step."""
import numpy as np
import pytest

import orc
import pe_gb300 as pg
from pe_gb300 import scene as sc

pytestmark = pytest.mark.gpu


def _line(n, lengths, bits, seed, dense=False):
    """Unit boxes one apart along x, and for each length a kinematic slab that starts just left of a
    box and spans that many of them."""
    r = np.random.default_rng(seed)
    sb = sc.SceneBuilder(dt=1.0 / 60.0, iterations=2, gravity=(0.0, 0.0, 0.0))
    box = sb.shape(sc.BOX, (0.9, 0.9, 0.9))
    for i in range(n):
        z = 0.0 if dense else float(r.uniform(-3, 3))   # not every box of a window overlaps its slab
        sb.body(box, (float(i), float(r.uniform(-0.4, 0.4)), z), mass=1.0)
    for k, m in enumerate(lengths):
        start = int(r.integers(0, max(1, n - m)))
        sb.body(sb.shape(sc.BOX, (float(m), 1.0, 2.0)), (start - 0.5 + m / 2 - 0.01, 0.0, 0.0), mass=0.0, kinematic=True)
    return sb.build(bits)


@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("lengths", [(1, 31, 32, 33, 63), (64, 65, 95, 96, 97, 127, 128), (191, 192, 193, 320, 321, 449)])
def test_windows_of_a_warp(lengths, bits):
    s = _line(460, lengths, bits, seed=len(lengths) + bits)
    g, o = pg.GpuWorld(s, bits), orc.OracleWorld(s, bits, stable_ties=True)
    for _ in range(3):
        g.step(1, pg.SERIAL_ORDER)
        o.step(1)
        assert np.array_equal(g.pairs(), o.pairs())
        assert g.axis == o.axis
    g.close()


def test_windows_of_blocks():
    # 4,095 to 5,121 candidates: the last that one warp sweeps, the first in chunks, and a second chunk round
    s = _line(5400, (4095, 4096, 4097, 5119, 5121), 32, seed=3)
    g, o = pg.GpuWorld(s, 32), orc.OracleWorld(s, 32, stable_ties=True)
    for _ in range(2):
        g.step(1, pg.SERIAL_ORDER)
        o.step(1)
        assert np.array_equal(g.pairs(), o.pairs())
        assert g.axis == o.axis
    g.close()


def test_windows_end_with_their_scene():
    sizes = (40, 2, 130, 33, 1, 260)
    parts = [_line(n, (max(1, n - 3),), 32, seed=n, dense=True) for n in sizes]
    whole, offs = sc.concat(parts)
    g = pg.GpuWorld(whole, 32, scenes=offs)
    g.step(2, pg.SERIAL_ORDER)
    want = []
    for k, p in enumerate(parts):
        alone = orc.OracleWorld(p, 32, stable_ties=True)
        alone.step(2)
        want.append(alone.pairs().reshape(-1, 2) + int(offs[k]))
    assert np.array_equal(g.pairs().reshape(-1, 2), np.concatenate(want))
    g.close()


@pytest.mark.parametrize("n", [16383, 16384, 16387])
def test_windows_of_four_positions(n):
    """From 16,384 bodies on a warp counts four positions: windows that end inside and at the edges of its
    chunks, the last positions of the world, and scenes that end between a warp's positions."""
    s = _line(n - 40, [m for m in range(1, 80, 2)], 32, seed=n)
    g, o = pg.GpuWorld(s, 32), orc.OracleWorld(s, 32, stable_ties=True)
    for _ in range(2):
        g.step(1, pg.SERIAL_ORDER)
        o.step(1)
        assert np.array_equal(g.pairs(), o.pairs())
    g.close()


@pytest.mark.parametrize("bits", [32, 64])
def test_windows_of_four_positions_end_with_their_scene(bits):
    parts = [_line(int(m), (3, 5, 17, 33), bits, seed=k, dense=k % 2 == 0) for k, m in enumerate(np.resize([61, 36, 50, 127, 43], 260))]
    whole, offs = sc.concat(parts)
    assert whole.n_bodies >= 16384
    g = pg.GpuWorld(whole, bits, scenes=offs)
    g.step(1, pg.SERIAL_ORDER)
    want = []
    for k, p in enumerate(parts):
        alone = orc.OracleWorld(p, bits, stable_ties=True)
        alone.step(1)
        want.append(alone.pairs().reshape(-1, 2) + int(offs[k]))
    assert np.array_equal(g.pairs().reshape(-1, 2), np.concatenate(want))
    g.close()


def test_windows_of_blocks_in_a_large_scene():
    """A scene of 40,000 bodies: blocks take windows of more than an eighth of it, warps shared by four
    positions those of 4,097 to 5,000."""
    s = _line(39993, (4096, 4097, 4999, 5000, 5001, 6200, 39000), 32, seed=9)
    assert s.n_bodies == 40000
    g, o = pg.GpuWorld(s, 32), orc.OracleWorld(s, 32, stable_ties=True)
    for _ in range(2):
        g.step(1, pg.SERIAL_ORDER)
        o.step(1)
        assert np.array_equal(g.pairs(), o.pairs())
        assert g.axis == o.axis
    g.close()


def _swept(mn, mx, kinematic, axis):
    """The pairs of one scene's sweep in chunks of 32 from each position on; a box that is not a number has
    zero's place in the order."""
    order = np.argsort(np.nan_to_num(mn[:, axis]), kind="stable")
    mn, mx, kinematic = mn[order], mx[order], kinematic[order]
    out = []
    with np.errstate(invalid="ignore"):
        for i in range(len(mn)):
            for j0 in range(i + 1, len(mn), 32):
                j = np.arange(j0, min(j0 + 32, len(mn)))
                inside = ~(mn[j, axis] > mx[i, axis])
                hit = inside & ~((mn[i] > mx[j]) | (mn[j] > mx[i])).any(1) & ~(kinematic[i] & kinematic[j])
                out += [(order[i], order[k]) for k in j[hit]]
                if len(j) < 32 or not inside.all():
                    break
    return np.array(out, np.int32).reshape(-1, 2)


@pytest.mark.parametrize("n", [5000, 16389])   # a warp per position, and one for four
@pytest.mark.parametrize("lost", [1, 2, 3, 30])
@pytest.mark.parametrize("bits", [32, 64])
def test_windows_beside_boxes_that_are_not_numbers(bits, lost, n):
    """Windows that end shortly before such boxes, of single boxes and of slabs longer than the blocks' limit."""
    sb = sc.SceneBuilder(dt=1.0 / 60.0, iterations=2, gravity=(0.0, 0.0, 0.0))
    box = sb.shape(sc.BOX, (12.4, 0.9, 0.9))   # twelve partners each: more than are kept for the write
    for i in range(n - 4):
        sb.body(box, (float(i - n + 300), 0.0, 0.0), mass=1.0)
    for k in range(4):
        sb.body(sb.shape(sc.BOX, (4400.0, 1.0, 2.0)), (-2200.0 - 9.0 * k - 5.3, 0.0, 0.0), mass=0.0, kinematic=True)
    g = pg.GpuWorld(sb.build(bits), bits)
    st = g.state()
    at = np.random.default_rng(lost).permutation(n - 4)[:lost]
    st["origin"][at] = np.nan
    kinematic = np.arange(n) >= n - 4
    for again in range(2):
        g.axis = 0
        g.set_state({"origin": st["origin"]})
        g.integrate()
        g.broadphase()
        s = g.state(fields=("aabb_min", "aabb_max"))
        want = _swept(s["aabb_min"], s["aabb_max"], kinematic, 0)
        got = g.pairs().reshape(-1, 2)
        assert np.isnan(s["aabb_min"][at]).all() != bool(again) and len(want) > 11 * n
        assert np.array_equal(got, want)
        st["origin"][at] = 1e4 + 20.0 * np.arange(lost)[:, None]   # then no such box any more
    g.close()
