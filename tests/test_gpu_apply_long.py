"""Impulses of a point that many sub-tests hit, against the oracle's build with
correctly rounded math: a fan of n triangles whose apex rests within the
thickness above a fixed triangle puts n contributions on the apex (one, a
warp's worth, more than a warp's, more than the shared-memory stage holds)."""
import numpy as np
import pytest

from collision_gb300 import scenes
from oracle.ccopy import OracleSolver

pytestmark = pytest.mark.gpu


def _fan(n):
    h = 1e-3
    a = np.linspace(0.0, 2.0 * np.pi, n + 1) + 0.013
    ring = np.stack([0.05 * np.cos(a), 0.05 * np.sin(a), np.full(n + 1, 0.05)], axis=1)
    # above a sloping floor (z = 0.2 x), whose box reaches the fan's
    p = np.concatenate([[[0.011, 0.007, 0.2 * 0.011 + 0.4 * h]], ring])
    t = np.array([[0, 1 + k, 2 + k] for k in range(n)], np.int32)
    v = np.tile([0.1, 0.05, -0.3], (len(p), 1))
    floor = np.array([[-1.0, -1.1, -0.2], [1.2, -1.0, 0.24], [0.1, 1.3, 0.02]])
    return scenes.assemble(f"fan{n}", [(p, t, v, False), (floor, np.array([[0, 1, 2]], np.int32),
                                                         np.zeros((3, 3)), True)],
                           dict(dt=1e-3, thickness=h, lam=0.2))


@pytest.mark.parametrize("n", [1, 2, 31, 33, 255, 257, 600])
def test_many_contributions_at_one_point(n):
    from collision_gb300.solver import CollisionSolver3d
    sc = _fan(n)
    ora = OracleSolver(sc, record=0, crmath=True)
    x, v, hc = sc.x, sc.v, np.zeros(sc.nv, np.uint8)
    xc = scenes.candidate(sc, x, v)
    o = ora.step(x, xc, v, hc)
    assert o["rc"] == 0 and o["has_collsn"][0] == 1
    for mode in (0, 1):
        s = CollisionSolver3d(0)
        s.setMode(mode)
        s.assembleFromScene(sc)
        xg, vg, hg = s.resolveCollision(x, xc, v, hc)
        assert s.counters()["contacts"] >= n
        assert np.array_equal(xg, o["x"]) and np.array_equal(vg, o["v"]) and np.array_equal(hg, o["has_collsn"])
        s.close()
