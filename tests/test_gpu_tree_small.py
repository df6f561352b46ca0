"""The GPU tree build's insertion groups at small and uneven leaf counts: the
ranks and volumes of both trees against the host emulation."""
import numpy as np
import pytest

from collision_gb300 import scenes

pytestmark = pytest.mark.gpu


def _soup(n, seed):
    """n separate small triangles in a unit box."""
    rng = np.random.default_rng(seed)
    p = (rng.uniform(0, 1, (n, 1, 3)) + rng.uniform(-0.02, 0.02, (n, 3, 3))).reshape(-1, 3)
    v = rng.uniform(-1, 1, p.shape)
    t = np.arange(3 * n, dtype=np.int32).reshape(-1, 3)
    return scenes.assemble(f"soup{n}", [(p, t, v, False)], dict(dt=1e-3, thickness=1e-4))


@pytest.mark.parametrize("n", [1, 2, 3, 5, 31, 255, 256, 257, 258, 259, 513, 1500])
def test_small_trees_equal_host_emulation(n):
    from collision_gb300.solver import CollisionSolver3d
    sc = _soup(n, n)
    got = []
    for host in (0, 1):
        s = CollisionSolver3d(0)
        s.setTuning(s.TUNE_HOST_TREE, host)
        s.assembleFromScene(sc)
        s.resolveCollision(sc.x, scenes.candidate(sc, sc.x, sc.v), sc.v, np.zeros(sc.nv, np.uint8))
        got.append((s.leafRanks(0), s.leafRanks(1), s.treeVolume(0)))
        s.close()
    assert np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][1], got[1][1]) and got[0][2] == got[1][2]
