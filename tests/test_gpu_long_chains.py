"""An island whose items wait long for one another is solved to its end: a chain of very many hinged bodies,
whose joints run one after the other (some ten microseconds each in FP64)."""
import numpy as np
import pytest

import orc
import pe_gb300 as pg
from pe_gb300 import scene as sc

pytestmark = pytest.mark.gpu


def _chain(n):
    sb = sc.SceneBuilder(dt=1.0 / 60.0, iterations=1)
    box = sb.shape(sc.BOX, (1.0, 0.7, 0.9))
    for k in range(2):
        sb.body(box, (0.0, 0.0, 0.0), mass=2.0)
    sb.joint(1, 0, 1, anchor_a=(0.6, 0.0, 0.0), anchor_b=(-0.6, 0.0, 0.0), axis_a=(0, 0, 1), axis_b=(0, 0, 1), limits=(-0.2, 0.1), motor_speed=1.0)
    s = sb.build(64)
    r = np.random.default_rng(1)
    one = np.zeros(n + 1, int)
    for f in ("body_shape", "body_flags", "mass", "friction", "restitution", "lin_damp", "ang_damp", "basis"):
        setattr(s, f, getattr(s, f)[one])
    s.origin = np.stack([1.2 * np.arange(n + 1), np.zeros(n + 1), np.zeros(n + 1)], 1)
    s.lin_vel, s.ang_vel = r.normal(size=(2, n + 1, 3))
    one = one[1:]
    s.joint_type, s.joint_flag, s.joint_real = s.joint_type[one], s.joint_flag[one], s.joint_real[one]
    s.joint_body = np.stack([np.arange(n), np.arange(1, n + 1)], 1).astype(np.int32)
    return s


def test_a_chain_of_a_second():
    s = _chain(120000)
    g, o = pg.GpuWorld(s, 64), orc.OracleWorld(s, 64)
    for w in (g, o):
        w.solve()
    assert g.last_counts()["islands"] == 1
    a, b = g.state(fields=("lin_vel", "ang_vel")), o.state()
    for k in a:
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)
