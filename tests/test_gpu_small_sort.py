"""Broad-phase builds at the sizes where the one-CTA leaf sort changes how many
elements a thread holds (1, 2, 4 and 8), and below a warp's worth: the pairs
must be those of all pairs tested."""
import numpy as np
import pytest

from collision_gb300 import scenes
from tests.test_gpu_leaf_sort import _sparse_soup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 31, 32, 33, 64, 1000, 1024, 1025, 2048, 2049, 4096, 4097, 6000])
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
