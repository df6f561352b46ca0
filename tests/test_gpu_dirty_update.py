"""Pruned passes that box only the elements the previous pass touched, against
the same passes with every box formed again (TUNE_PRUNED_WARP 0): scenes whose
boxes grow past the tree-rebuild bound and shrink again within a step, single
elements, several scenes, FP64 and mixed, and buffers that overflow in a pass.
Outputs, zones, leaf ranks and tree volumes must agree to the bit."""
import numpy as np
import pytest

from collision_gb300 import scenes

pytestmark = pytest.mark.gpu


def _swarm(n, seed, side, speed):
    """n triangles thrown at each other: their swept boxes set the scene's."""
    rng = np.random.default_rng(seed)
    c = rng.uniform(-side, side, (n, 1, 3))
    p = (c + rng.uniform(-0.05, 0.05, (n, 3, 3))).reshape(-1, 3)
    v = (np.repeat(-speed * c / side, 3, axis=1) + rng.uniform(-0.3, 0.3, (n, 3, 3)) * speed).reshape(-1, 3)
    t = np.arange(3 * n, dtype=np.int32).reshape(-1, 3)
    return scenes.assemble(f"swarm{n}", [(p, t, v, False)], dict(dt=1e-2, thickness=1e-3))


CASES = {"swarm": (lambda: [_swarm(60, 1, 0.2, 20.0)], 4, None), "two": (lambda: [_swarm(2, 2, 0.02, 5.0)], 3, None),
         "one": (lambda: [_swarm(1, 3, 0.1, 5.0), _swarm(40, 4, 0.15, 15.0)], 3, None),
         "batch": (lambda: scenes.batched(12, 16, 40, seed=9), 8, None),
         "overflow": (lambda: scenes.batched(6, 16, 48, seed=3), 6, 4096),
         "strings": (lambda: [scenes.strings(nstr=12, nseg=90, seed=5)], 8, None)}


def _run(mix, nsteps, warp, mode, capacity):
    from collision_gb300.solver import CollisionSolver3d
    b = CollisionSolver3d(0)
    b.assembleBatch(mix)
    b.setMode(mode)
    b.setZoneCap(40)
    b.setTuning(b.TUNE_PRUNED_WARP, warp)
    if capacity:
        b.setTuning(b.TUNE_PAIR_CAPACITY, capacity)
    x = np.concatenate([s.x for s in mix])
    v = np.concatenate([s.v for s in mix])
    hc = np.zeros(len(x), np.uint8)
    dt = np.concatenate([np.full(s.nv, s.params["dt"]) for s in mix])[:, None]
    out = []
    for _ in range(nsteps):
        x, v, hc, _ = b.resolveCollisionBatch(x, x + dt * v, v, hc)
        c = b.counters()
        out.append((x, v, hc, b.zoneRoots(), b.leafRanks(0), b.leafRanks(1),
                    np.array([b.treeVolume(i) for i in range(len(mix))]),
                    np.array([c["passes"], c["ccd_passes"], c["hit_pairs"], c["contacts"], c["pruned_queries"]])))
    b.close()
    return out


@pytest.mark.parametrize("mode", [0, 1], ids=["plain", "mixed"])
@pytest.mark.parametrize("case", list(CASES))
def test_dirty_boxes_equal_all_boxes(case, mode):
    make, nsteps, capacity = CASES[case]
    mix = make()
    a, b = _run(mix, nsteps, 1, mode, capacity), _run(mix, nsteps, 0, mode, capacity)
    print(case, [tuple(s[7]) for s in a])
    for u, w in zip(a, b):
        for x, y in zip(u, w):
            assert np.array_equal(x, y)
