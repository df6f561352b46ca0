"""The GPU tree build's decisions in units of the tree's extents, against the
host emulation: flat sheets whose boxes share coordinates, identical elements
(ties), extents of very different size, coordinates far from the origin, where
the units and the pads of the boxes vanish, and elements of a wide range of
sizes. Ranks of both trees and volumes."""
import numpy as np
import pytest

from collision_gb300 import scenes

pytestmark = pytest.mark.gpu


def _mesh(kind):
    rng = np.random.default_rng(len(kind))
    if kind in ("flat", "far", "farther", "tilted"):
        p, t = scenes.grid_cloth(30, 1.0, 0.3)
        if kind == "tilted":
            p = p @ np.linalg.qr(rng.standard_normal((3, 3)))[0]
        return p + {"far": 1e4, "farther": 1e9}.get(kind, 0.0), t
    if kind == "same":
        one = rng.uniform(0, 1, (1, 3, 3))
        p = np.repeat(one, 300, axis=0).reshape(-1, 3)
    elif kind == "long":
        c = rng.uniform(-1, 1, (700, 1, 3)) * [1e3, 1.0, 1e-4]
        p = (c + rng.uniform(-1, 1, (700, 3, 3)) * [1.0, 1e-2, 1e-5]).reshape(-1, 3)
    else:  # sizes
        c = rng.uniform(-1, 1, (900, 1, 3))
        p = (c + rng.uniform(-1, 1, (900, 3, 3)) * 10.0 ** rng.uniform(-6, 0, (900, 1, 1))).reshape(-1, 3)
    return p, np.arange(len(p), dtype=np.int32).reshape(-1, 3)


@pytest.mark.parametrize("kind", ["flat", "far", "farther", "tilted", "same", "long", "sizes"])
def test_unit_decisions_equal_host_emulation(kind):
    from collision_gb300.solver import CollisionSolver3d
    p, t = _mesh(kind)
    rng = np.random.default_rng(3)
    v = rng.uniform(-1, 1, p.shape) * 1e-3
    # (identical free elements meet without a normal, where the reference exits)
    sc = scenes.assemble(kind, [(p, t, v, kind == "same")], dict(dt=1e-3, thickness=1e-9))
    got = []
    for host in (0, 1):
        s = CollisionSolver3d(0)
        s.setMode(1)
        s.setZoneCap(2)
        s.setTuning(s.TUNE_HOST_TREE, host)
        s.assembleBatch([sc])
        s.resolveCollisionBatch(sc.x, scenes.candidate(sc, sc.x, sc.v), sc.v, np.zeros(sc.nv, np.uint8))
        got.append((s.leafRanks(0), s.leafRanks(1), s.treeVolume(0)))
        s.close()
    assert np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][1], got[1][1]) and got[0][2] == got[1][2]
