"""A request with a shape that the serving loop does not take is refused when it is submitted: the loop and
the requests before and after it go on as if it had never been there."""
import numpy as np
import pytest

import pe_gb300 as pg
from pe_gb300 import scene as sc

pytestmark = pytest.mark.gpu

FIELDS = ("origin", "basis", "lin_vel", "ang_vel")


def _scene(kinds):
    sb = sc.SceneBuilder(dt=1.0 / 60.0)
    sb.body(sb.shape(sc.BOX, (20.0, 1.0, 20.0)), (0.0, -0.5, 0.0), mass=0.0, kinematic=True)
    for k, (kind, size) in enumerate(kinds):
        sb.body(sb.shape(kind, size), (0.3 * k, 1.0 + 1.1 * k, 0.1 * k), mass=1.0 + k)
    return sb


def _fan(n, apex):
    """A cone over an n-gon: n side triangles, the n-gon itself if `apex` is None."""
    a = 2 * np.pi * np.arange(n) / n
    v = np.concatenate([np.stack([np.cos(a), np.zeros(n), -np.sin(a)], 1), [[0.0, 1.0, 0.0]]])
    return v, [[n, i, (i + 1) % n] for i in range(n)] if apex else [list(range(n))]


def _refused(what):
    sb = _scene([(sc.BOX, (0.7, 0.9, 1.1)), (sc.SPHERE, (0.45, 0.0, 0.0))])
    if what == "compound":
        box = sb.shape(sc.BOX, (0.4, 0.4, 0.4))
        sb.body(sb.compound([(box, (0.5, 0.0, 0.0), np.eye(3), 1.0), (box, (-0.5, 0.0, 0.0), np.eye(3), 1.0)]), (0.0, 5.0, 0.0))
    elif what == "faces":
        sb.body(sb.shape(sc.HULL, hull=_fan(16382, True)), (0.0, 5.0, 0.0))
    elif what == "polygon":
        sb.body(sb.shape(sc.CONCAVE, hull=_fan(33, False)), (0.0, -3.0, 0.0), mass=0.0, kinematic=True)
    s = sb.build(32)
    if what == "type":
        s.shape_type = s.shape_type.copy()
        s.shape_type[2] = 9
    return s


@pytest.mark.parametrize("what", ["compound", "faces", "polygon", "type"])
def test_refused_request_leaves_the_others_alone(what):
    first = _scene([(sc.BOX, (1.0, 1.0, 1.0)), (sc.CYLINDER, (0.5, 1.0, 0.0))]).build(32)
    later = _scene([(sc.SPHERE, (0.6, 0.0, 0.0)), (sc.BOX, (0.5, 0.8, 0.6)), (sc.CYLINDER, (0.3, 0.9, 0.0))]).build(32)
    srv = pg.Server(real_bits=32, mode=pg.COLORED)
    ids = {srv.submit(first, 20): first}
    srv.step()
    with pytest.raises(pg.PeGpuError):
        srv.submit(_refused(what), 5)
    ids[srv.submit(later, 25)] = later
    assert srv.step() == (2, 0)
    done = {}
    for _ in range(30):
        srv.step()
        for rid in [i for i in ids if i not in done]:
            st, res = srv.result(rid)
            if st == pg.DONE:
                done[rid] = res
    for rid, s in ids.items():
        alone = pg.GpuWorld(s, 32)
        alone.step(20 if s is first else 25, pg.COLORED)
        want = alone.state(fields=FIELDS)
        for f in FIELDS:
            np.testing.assert_array_equal(done[rid][f], want[f], err_msg=f)
        alone.close()
    st = srv.stats()
    assert (st["finished"], st["live"], st["queued"]) == (2, 0, 0)
    srv.close()
