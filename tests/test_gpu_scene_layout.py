"""A world that has stepped is divided into scenes anew, with as many scenes and bodies as before: steps
replayed from captured graphs follow the new largest scene across the limits of the one-block scene sort
(2,048 bodies) and of the windows swept in chunks (4,096 candidates)."""
import numpy as np
import pytest

import orc
import pe_gb300 as pg
from pe_gb300 import scene as sc
from test_gpu_sweep_windows import _line

pytestmark = pytest.mark.gpu

SMALL, WIDE, MIDDLE = [0, 2000, 4000, 6000], [0, 100, 200, 6000], [0, 2100, 4100, 6000]


@pytest.mark.parametrize("layouts", [(SMALL, WIDE, SMALL), (WIDE, MIDDLE, WIDE), (SMALL, MIDDLE, WIDE)])
def test_steps_follow_the_scene_layout(layouts):
    s = _line(5999, (5000,), 32, seed=7)
    g, plain = pg.GpuWorld(s, 32, scenes=layouts[0]), pg.GpuWorld(s, 32, scenes=layouts[0])
    plain.set_step_graphs(False)
    for offs in layouts:
        for w in (g, plain):
            w.set_scenes(offs)
            w.step(6, pg.COLORED)   # graphs are captured from the second on
        before, axes = g.state(), g.axes(3)
        for w in (g, plain):
            w.step(1, pg.COLORED)
        assert np.array_equal(g.pairs(), plain.pairs())
        a, b = g.state(), plain.state()
        for k in a:
            assert np.array_equal(a[k], b[k]), k
        want = []
        for k in range(3):
            o = orc.OracleWorld(sc.extract(s, np.array(offs), k), 32, stable_ties=True)
            o.set_state({f: v[offs[k]:offs[k + 1]] for f, v in before.items()})
            o.axis = int(axes[k])
            o.integrate()
            o.broadphase()
            want.append(o.pairs().reshape(-1, 2) + offs[k])
        assert np.array_equal(g.pairs().reshape(-1, 2), np.concatenate(want))
    g.close()
    plain.close()
