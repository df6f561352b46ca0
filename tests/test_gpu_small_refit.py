"""Refits of small hierarchies in one CTA against the level-by-level refit
(TUNE_REFIT_UP 0): hierarchies of two leaves up to and past the size it takes
(4,096), several scenes at once with scenes of one element among them, and
later passes over a part of the scenes. Outputs, counts and pairs must agree."""
import numpy as np
import pytest

from collision_gb300 import scenes
from tests.test_gpu_leaf_sort import _sparse_soup

pytestmark = pytest.mark.gpu

CASES = {"2": (lambda: [_sparse_soup(2)], 1), "33": (lambda: [_sparse_soup(33)], 1),
         "4095": (lambda: [_sparse_soup(4095)], 1), "4096": (lambda: [_sparse_soup(4096)], 1),
         "4097": (lambda: [_sparse_soup(4097)], 1),
         "scenes": (lambda: [_sparse_soup(1), _sparse_soup(300), _sparse_soup(1), _sparse_soup(2)], 1),
         "passes": (lambda: [_sparse_soup(1)] + scenes.batched(2, 16, 24, seed=3), 9)}


def _run(mix, nsteps, up):
    from collision_gb300.solver import CollisionSolver3d
    b = CollisionSolver3d(0)
    b.assembleBatch(mix)
    b.setMode(1)
    b.setZoneCap(40)
    b.setTuning(b.TUNE_REFIT_UP, up)
    x = np.concatenate([s.x for s in mix])
    v = np.concatenate([s.v for s in mix])
    hc = np.zeros(len(x), np.uint8)
    dt = np.concatenate([np.full(s.nv, s.params["dt"]) for s in mix])[:, None]
    out = []
    for _ in range(nsteps):
        x, v, hc, _ = b.resolveCollisionBatch(x, x + dt * v, v, hc)
        c = b.counters()
        out.append([x, v, hc, np.array([c[k] for k in ("passes", "candidate_pairs", "visits", "hit_pairs", "contacts")])])
    pairs = np.sort(b.candidatePairs(True), axis=1)
    out.append([pairs[np.lexsort(pairs.T)]])
    b.close()
    return out


@pytest.mark.parametrize("case", list(CASES))
def test_small_refit_equals_the_general_one(case):
    make, nsteps = CASES[case]
    mix = make()
    for a, b in zip(_run(mix, nsteps, 1), _run(mix, nsteps, 0)):
        for u, w in zip(a, b):
            assert np.array_equal(u, w)
