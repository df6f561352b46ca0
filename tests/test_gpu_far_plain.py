"""The plain path far from the origin, where its filter takes positions relative
to each sub-test, against the oracle's build with correctly rounded math: a
sheet falling on a box at offsets around which the filter changes and beyond."""
import numpy as np
import pytest

from collision_gb300 import scenes
from oracle.ccopy import OracleSolver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [0.0, 30.0, 1e3, 1e6])
def test_plain_steps_far_from_the_origin(offset):
    from collision_gb300.solver import CollisionSolver3d
    sc = scenes.cloth_on_obstacle(13, "box", 0.2, 2.0, seed=11, gap=3e-3)
    sc.x[:] = sc.x + offset
    sc.domain[:] = np.asarray(sc.domain) + offset
    gpu, ora = CollisionSolver3d(0), OracleSolver(sc, record=0, crmath=True)
    gpu.assembleFromScene(sc)
    x, v, hc = sc.x, sc.v, np.zeros(sc.nv, np.uint8)
    contacts = 0
    for step in range(5):
        xc = scenes.candidate(sc, x, v)
        got = gpu.resolveCollision(x, xc, v, hc)
        r = ora.step(x, xc, v, hc)
        assert r["rc"] == 0
        assert np.array_equal(got[0], r["x"]) and np.array_equal(got[1], r["v"]), step
        assert np.array_equal(got[2], r["has_collsn"]), step
        contacts += gpu.counters()["contacts"]
        x, v, hc = got
    assert contacts > 0
    gpu.close()
