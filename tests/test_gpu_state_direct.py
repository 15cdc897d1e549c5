"""Body state into and out of page-locked arrays (used in place), ordinary ones (staged) and a mix, in both
types and precisions, at array sizes around the one up to which page-locked memory is used in place, and
at an odd offset inside a page-locked block: the same values on every route."""
import numpy as np
import pytest
import torch

import pe_gb300 as pg
from pe_gb300 import scene as sc

pytestmark = pytest.mark.gpu
SHAPES = {"origin": (3,), "basis": (3, 3), "lin_vel": (3,), "ang_vel": (3,), "aabb_min": (3,), "aabb_max": (3,), "world_inv_inertia": (3, 3)}


def _world(n, bits):
    r = np.random.default_rng(n)
    sb = sc.SceneBuilder(dt=0.01)
    box = sb.shape(sc.BOX, (1.0, 0.5, 0.7))
    rot, pos, vel = sc.random_rotations(r, n), r.uniform(-50, 50, (n, 3)), r.normal(size=(n, 6))
    for i in range(n):
        sb.body(box, pos[i], rot[i], mass=1.0, v=vel[i, :3], w=vel[i, 3:])
    g = pg.GpuWorld(sb.build(bits), bits)
    g.integrate()
    return g


def _pinned(shape, dtype, skip):
    """A page-locked array `skip` values into its block."""
    t = torch.empty(int(np.prod(shape)) + skip, dtype=torch.float32 if dtype == np.float32 else torch.float64).pin_memory()
    return t.numpy()[skip:].reshape(shape)


@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n", [1, 33, 14563, 29128, 44000])
def test_every_route_gives_the_same(n, dtype, bits):
    g = _world(n, bits)
    fields = [f for f in SHAPES if f in g.state()]
    plain = {f: np.full((n,) + SHAPES[f], 7, dtype) for f in fields}
    g.state(tuple(fields), out=plain)
    for skip, mixed in ((0, False), (3, False), (1, True)):
        out = {f: _pinned((n,) + SHAPES[f], dtype, skip) if not mixed or k % 2 else np.zeros((n,) + SHAPES[f], dtype)
               for k, f in enumerate(fields)}
        g.state(tuple(fields), out=out)
        for f in fields:
            assert np.array_equal(out[f], plain[f]), (f, skip, mixed)
        # and in again: half the speeds
        out["lin_vel"] *= dtype(0.5)
        g.set_state({f: out[f] for f in ("origin", "basis", "lin_vel", "ang_vel")})
        now = {f: np.zeros((n,) + SHAPES[f], dtype) for f in fields}
        g.state(tuple(fields), out=now)
        for f in ("origin", "basis", "ang_vel"):
            assert np.array_equal(now[f], plain[f]), f
        assert np.array_equal(now["lin_vel"], out["lin_vel"])
        g.set_state({"lin_vel": plain["lin_vel"]})
    g.close()
