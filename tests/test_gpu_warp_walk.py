"""Broad-phase walks with a warp per query, and long walks handed over to a
warp, against testing all pairs: leaf counts around a warp, around the size up
to which every query gets a warp (32,768 leaves), and large boxes over many
small ones."""
import numpy as np
import pytest

from collision_gb300 import scenes
from tests.test_gpu_tree_small import _soup

pytestmark = pytest.mark.gpu


def _over_box(n):
    return scenes.cloth_on_obstacle(n, "box", 0.2, 2.0, gap=5e-4, seed=n)


@pytest.mark.parametrize("make", [lambda: _soup(2, 1), lambda: _soup(3, 2), lambda: _soup(33, 3),
                                  lambda: _soup(700, 4), lambda: _over_box(40), lambda: _over_box(128),
                                  lambda: _over_box(129), lambda: scenes.strings(nstr=8, nseg=100, seed=2)],
                         ids=["2", "3", "33", "700", "box40", "box128", "box129", "strings"])
def test_pairs_equal_brute_force(make):
    from collision_gb300.solver import CollisionSolver3d
    sc = make()
    s = CollisionSolver3d(0)
    s.assembleFromScene(sc)
    s.resolveCollision(sc.x, scenes.candidate(sc, sc.x, sc.v), sc.v, np.zeros(sc.nv, np.uint8))
    for moving in (False, True):
        want = np.sort(s.candidatePairs(moving, brute_force=True), axis=1)
        got = np.sort(s.candidatePairs(moving), axis=1)
        assert len(got) == len(want)
        assert np.array_equal(got[np.lexsort(got.T)], want[np.lexsort(want.T)])
    s.close()
