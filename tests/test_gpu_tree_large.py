"""Trees around the line between the two insertion kernels, and a batch with
trees on both sides of it: ranks and volumes of the host emulation."""
import numpy as np
import pytest

from collision_gb300 import scenes

pytestmark = pytest.mark.gpu


def _cloth(cells, seed):
    """A sheet of 2 x cells triangles in rows of at most 300 squares, waved and with noise."""
    rng = np.random.default_rng(seed)
    w = min(300, cells)
    n = -(-cells // w) + 1
    i, j = np.meshgrid(np.arange(w + 1), np.arange(n), indexing="xy")
    x = np.stack([i.ravel() / 300.0, j.ravel() / 300.0, 0.05 * np.sin(i.ravel() / 9.0) * np.cos(j.ravel() / 7.0)], 1)
    x += 1e-4 * rng.normal(size=x.shape)
    c = np.arange(cells)
    a = (c // w) * (w + 1) + c % w
    tris = np.stack([np.stack([a, a + 1, a + w + 2], 1), np.stack([a, a + w + 2, a + w + 1], 1)], 1).reshape(-1, 3)
    return scenes.assemble("cloth", [(x, tris.astype(np.int32), np.zeros_like(x) + [0, 0, -0.5], False)], dict(dt=1e-3))


@pytest.mark.parametrize("leaves", [[131072], [131074], [2, 131072, 131074, 5000]])
def test_ranks_around_the_line(leaves):
    from collision_gb300.solver import CollisionSolver3d
    scs = [_cloth(k // 2, k) for k in leaves]
    assert [sc.ne for sc in scs] == leaves
    x = np.concatenate([sc.x for sc in scs])
    v = np.concatenate([sc.v for sc in scs])
    xc = np.concatenate([scenes.candidate(sc, sc.x, sc.v) for sc in scs])
    got = []
    for host in (0, 1):
        s = CollisionSolver3d(0)
        s.setTuning(s.TUNE_HOST_TREE, host)
        s.assembleBatch(scs)
        s.resolveCollisionBatch(x, xc, v, np.zeros(len(x), np.uint8))
        got.append(([s.leafRanks(w) for w in (0, 1)], [s.treeVolume(i) for i in range(len(scs))]))
        s.close()
    for a, b in zip(got[0][0], got[1][0]):
        assert np.array_equal(a, b)
    assert got[0][1] == got[1][1]
