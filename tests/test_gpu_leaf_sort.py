"""Broad-phase builds around the sizes at which the leaf sort changes: one CTA
up to 8,192 leaves, tiles of 2,048 above, whose digit counts are scanned by one
CTA between 9 and 32 tiles. The pairs must be those of all pairs tested."""
import numpy as np
import pytest

from collision_gb300 import scenes

pytestmark = pytest.mark.gpu


def _sparse_soup(n):
    """n small triangles at about four boxes' overlap each."""
    rng = np.random.default_rng(n)
    side = 0.04 * n ** (1 / 3)
    p = (rng.uniform(0, side, (n, 1, 3)) + rng.uniform(-0.02, 0.02, (n, 3, 3))).reshape(-1, 3)
    v = rng.uniform(-0.1, 0.1, p.shape)
    t = np.arange(3 * n, dtype=np.int32).reshape(-1, 3)
    return scenes.assemble(f"soup{n}", [(p, t, v, False)], dict(dt=1e-3, thickness=1e-6))


@pytest.mark.parametrize("n", [1, 4095, 8191, 8192, 8193, 16384, 16385, 20001])
def test_pairs_equal_brute_force(n):
    from collision_gb300.solver import CollisionSolver3d
    sc = _sparse_soup(n)
    s = CollisionSolver3d(0)
    s.assembleFromScene(sc)
    s.resolveCollision(sc.x, scenes.candidate(sc, sc.x, sc.v), sc.v, np.zeros(sc.nv, np.uint8))
    for moving in (False, True):
        want = np.sort(s.candidatePairs(moving, brute_force=True), axis=1)
        got = np.sort(s.candidatePairs(moving), axis=1)
        assert np.array_equal(got[np.lexsort(got.T)], want[np.lexsort(want.T)])
    s.close()
