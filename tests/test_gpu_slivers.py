"""Triangles so thin for their size that the reference's point-triangle test
calls a point lengths away from them a hit: the plain and the mixed path give
the oracle's steps (its build with correctly rounded math) there too."""
import numpy as np
import pytest

from collision_gb300 import scenes
from oracle.ccopy import OracleSolver

pytestmark = pytest.mark.gpu


def _pair(rng, size):
    """A sliver of the given size and a triangle with a corner on its line, past its end, whose box meets its box."""
    def unit():
        d = rng.normal(size=3)
        return d / np.linalg.norm(d)
    d = unit()
    u = np.cross(d, unit())
    u /= np.linalg.norm(u)
    height = 4.7e-7 / size * 10 ** rng.uniform(0.0, 1.0)
    past = rng.choice([-1, 1]) * size * rng.uniform(1.2, 2.0) * d
    x = np.array([size * rng.uniform(-1, 1) * d, size * rng.uniform(-1, 1) * d + height * u, 0 * d,
                  past, 0.3 * size * u, 0.3 * size * np.cross(d, u)])
    tris = np.array([[0, 1, 2], [3, 4, 5]], np.int32)
    rest = np.array([[np.linalg.norm(x[t[j]] - x[t[(j + 1) % 3]]) for j in range(3)] for t in tris])
    big = 10 * size
    params = dict(dt=1e-3, thickness=1e-3, eps=1e-6, k=1000.0, m=0.01, lam=0.02, cr=0.0)
    return scenes.Scene("sliver", x, rng.normal(size=(6, 3)) * 1e-3, np.zeros(6, np.uint8), tris,
                        np.arange(2, dtype=np.int32), rest, np.zeros((0, 2), np.int32), np.zeros(0, np.int32),
                        np.zeros(0), np.array([-big] * 3 + [big] * 3), params)


def _steps(sc):
    ora = OracleSolver(sc, record=0, crmath=True)
    ora.set_zone_cap(20)
    return ora.step(sc.x, scenes.candidate(sc, sc.x, sc.v), sc.v, np.zeros(sc.nv, np.uint8))


@pytest.mark.parametrize("size", [10.0, 40.0])
@pytest.mark.parametrize("mode", ["plain", "mixed"])
def test_hits_of_slivers(size, mode):
    from collision_gb300.solver import CollisionSolver3d
    rng = np.random.default_rng(int(size))
    scs, want = [], []
    while len(scs) < 48:
        sc = _pair(rng, size)
        r = _steps(sc)
        if r["rc"] == 0 and r["has_collsn"].any():
            scs.append(sc)
            want.append(r)
    s = CollisionSolver3d(0)
    s.setMode(s.MIXED if mode == "mixed" else s.PLAIN_FP64)
    s.setZoneCap(20)
    s.assembleBatch(scs)
    x = np.concatenate([sc.x for sc in scs])
    v = np.concatenate([sc.v for sc in scs])
    cand = np.concatenate([scenes.candidate(sc, sc.x, sc.v) for sc in scs])
    got = s.resolveCollisionBatch(x, cand, v, np.zeros(len(x), np.uint8))
    assert np.array_equal(got[2], np.concatenate([r["has_collsn"] for r in want]))
    assert np.array_equal(got[0], np.concatenate([r["x"] for r in want]))
    assert np.array_equal(got[1], np.concatenate([r["v"] for r in want]))
    s.close()
