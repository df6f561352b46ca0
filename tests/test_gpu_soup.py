"""Triangles flying through one another: passes whose sub-tests outgrow the
first queues, and impact-zone passes that outgrow the one-CTA join (more
joining records than it sorts, more points than its table holds), give what
the pair-per-thread narrow phase and the general zone kernels give."""
import numpy as np
import pytest

from collision_gb300 import scenes

pytestmark = pytest.mark.gpu


def _soup(n, spread, speed, seed):
    """n separate triangles of size 0.2 in a cube of side `spread`, each flying its own way."""
    rng = np.random.default_rng(seed)
    x = (spread * rng.random((n, 1, 3)) + 0.2 * rng.random((n, 3, 3))).reshape(-1, 3)
    v = (speed * rng.normal(size=(n, 1, 3)) + 0.02 * speed * rng.normal(size=(n, 3, 3))).reshape(-1, 3)
    tris = np.arange(3 * n, dtype=np.int32).reshape(n, 3)
    rest = np.linalg.norm(x[tris] - x[np.roll(tris, -1, axis=1)], axis=2)
    return scenes.Scene("soup", x, v, np.zeros(3 * n, np.uint8), tris, np.arange(n, dtype=np.int32), rest,
                        np.zeros((0, 2), np.int32), np.zeros(0, np.int32), np.zeros(0),
                        np.array([-100.0] * 3 + [100.0] * 3),
                        dict(dt=1e-3, thickness=1e-3, eps=1e-6, k=1000.0, m=0.01, lam=0.02, cr=0.0))


def _step(sc, mode, knobs):
    from collision_gb300.solver import CollisionSolver3d
    s = CollisionSolver3d(0)
    s.setMode(mode)
    s.setZoneCap(12)
    for k, val in knobs.items():
        s.setTuning(getattr(s, k), val)
    s.assembleBatch([sc])
    out = s.resolveCollisionBatch(sc.x, scenes.candidate(sc, sc.x, sc.v), sc.v, np.zeros(sc.nv, np.uint8))
    c = s.counters()
    s.close()
    return out, c


@pytest.mark.parametrize("n,spread,speed", [(150, 0.4, 400.0), (1200, 1.5, 150.0), (4000, 3.0, 100.0)])
def test_soup(n, spread, speed):
    sc = _soup(n, spread, speed, seed=n)
    want, c0 = _step(sc, 0, dict(TUNE_SPLIT_NARROW=0, TUNE_SMALL_SORT=0))
    assert c0["contacts"] > 0
    for mode in (0, 1):
        for device_loop in (1, 0):
            got, c = _step(sc, mode, dict(TUNE_DEVICE_LOOP=device_loop))
            for a, b in zip(got, want):
                assert np.array_equal(a, b), (mode, device_loop)
            assert c["contacts"] == c0["contacts"]
