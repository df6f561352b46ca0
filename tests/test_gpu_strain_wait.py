"""The strain sweeps' waits for one another: a closed string, whose first
point's last element is its last, so that every sweep waits for the whole of
the one before while that one waits for others; and a wait that runs out,
which ends the call with an error and leaves the solver usable."""
import numpy as np
import pytest

from collision_gb300 import scenes

pytestmark = pytest.mark.gpu


def _loop(n, dt=1e-3):
    """A closed string of n bonds of length 1e-3, stretched and compressed along its length."""
    i = np.arange(n)
    r = n * 1e-3 / (2 * np.pi)
    a = 2 * np.pi * i / n
    x = np.stack([r * np.cos(a), r * np.sin(a), 0.5 + 1e-4 * np.sin(9 * a)], axis=1)
    along = np.stack([-np.sin(a), np.cos(a), np.zeros(n)], axis=1)
    v = along * (3e-3 / dt * np.sin(0.25 * i / 3.0))[:, None]
    bonds = np.stack([i, (i + 1) % n], axis=1).astype(np.int32)
    rest = np.linalg.norm(x[bonds[:, 0]] - x[bonds[:, 1]], axis=1)
    big = 2 * r + 10.0
    return scenes.Scene("loop", x, v, np.zeros(n, np.uint8), np.zeros((0, 3), np.int32), np.zeros(0, np.int32),
                        np.zeros((0, 3)), bonds, np.zeros(n, np.int32), rest, np.array([-big] * 3 + [big] * 3),
                        dict(dt=dt, thickness=1e-5, eps=1e-6, k=1000.0, m=0.01, lam=0.02, cr=0.0))


def _step(s, sc):
    return s.resolveCollision(sc.x, scenes.candidate(sc, sc.x, sc.v), sc.v, np.zeros(sc.nv, np.uint8))


# 2,000 polls are about a millisecond: a sweep of 20,000 levels takes a dozen
@pytest.mark.parametrize("n,wait", [(3, None), (100, None), (20000, None), (20000, 2000)])
def test_closed_string_equals_global_path(n, wait):
    from collision_gb300.solver import CollisionSolver3d
    sc = _loop(n)
    got = []
    for window in (True, False):
        s = CollisionSolver3d(0)
        s.assembleFromScene(sc)
        s.setStrainWindow(window)
        if wait:
            s.setTuning(s.TUNE_STRAIN_WAIT, wait)
        got.append((_step(s, sc), s.counters()["strain_averaged"]))
        s.close()
    assert got[0][1] == got[1][1] and (got[0][1] > 0 or n < 100)
    for a, b in zip(got[0][0], got[1][0]):
        assert np.array_equal(a, b)


def test_wait_that_runs_out():
    from collision_gb300.solver import CollisionSolver3d
    sc = _loop(4000)
    s, ref = CollisionSolver3d(0), CollisionSolver3d(0)
    for q in (s, ref):
        q.assembleFromScene(sc)
    limit = s.getTuning(s.TUNE_STRAIN_WAIT)
    s.setTuning(s.TUNE_STRAIN_WAIT, 0)
    with pytest.raises(Exception, match="gave up"):
        _step(s, sc)
    s.setTuning(s.TUNE_STRAIN_WAIT, limit)
    for a, b in zip(_step(s, sc), _step(ref, sc)):
        assert np.array_equal(a, b)
    s.close()
    ref.close()
