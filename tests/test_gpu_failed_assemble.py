"""An assemble call that fails leaves no half of a mesh behind: the calls on it
end with an error, and the solver takes the next mesh. A call refused before
the old mesh is given up keeps it."""
import numpy as np
import pytest

from collision_gb300 import scenes

pytestmark = pytest.mark.gpu


def _bad(sc):
    sc = sc.copy()
    sc.tris[3] = sc.tris[3, [0, 0, 1]]
    return sc


@pytest.mark.parametrize("place", [0, 1, 2])
def test_steps_after_a_failed_assemble(place):
    import torch
    from collision_gb300.solver import CollisionSolver3d
    good = [scenes.cloth_on_obstacle(7, "box", 0.2, 2.0, seed=i, gap=3e-3) for i in range(3)]
    mixed = [_bad(sc) if i == place else sc for i, sc in enumerate(good)]
    s, ref = CollisionSolver3d(0), CollisionSolver3d(0)
    x = np.concatenate([sc.x for sc in good])
    v = np.concatenate([sc.v for sc in good])
    xc = np.concatenate([scenes.candidate(sc, sc.x, sc.v) for sc in good])
    hc = np.zeros(len(x), np.uint8)
    dev = torch.from_numpy(x).cuda()
    for window in (True, False):
        s.setStrainWindow(window)
        s.assembleBatch(good)
        with pytest.raises(Exception, match="repeated point"):
            s.assembleBatch(mixed)
        assert s.numScenes() == 0
        for call in (lambda: s.resolveCollisionBatch(x, xc, v, hc), lambda: s.checkCCD(dev, dev), s.autotune):
            with pytest.raises(Exception, match="last assemble call failed"):
                call()
    s.setStrainWindow(True)
    s.assembleBatch(good)
    ref.assembleBatch(good)
    with pytest.raises(Exception):
        s.assembleBatch([])  # refused at once: the mesh stays
    for a, b in zip(s.resolveCollisionBatch(x, xc, v, hc), ref.resolveCollisionBatch(x, xc, v, hc)):
        assert np.array_equal(a, b)
    s.close()
    ref.close()
