"""Parameters given before the mesh is assembled, as the reference's static
setters are, count as those given after it: time steps other than the default,
one mesh and a batch."""
import numpy as np
import pytest

from collision_gb300 import scenes

pytestmark = pytest.mark.gpu


def _mesh(sc):
    return dict(n_points=sc.nv, tris=sc.tris, tri_surface=sc.tri_surf, tri_rest=sc.tri_rest, bonds=sc.bonds,
                bond_rest=sc.bond_rest, fixed=sc.fixed)


@pytest.mark.parametrize("batch", [False, True])
@pytest.mark.parametrize("dt", [1e-3, 7e-4])
def test_order_of_parameters_and_mesh(dt, batch):
    from collision_gb300.solver import CollisionSolver3d
    sc = scenes.cloth_on_obstacle(17, "sphere", 0.2, 2.0, dt=dt, seed=3, gap=2e-3)
    got = []
    for first in (True, False):
        s = CollisionSolver3d(0)
        if first:
            s.setParams(sc.params)
        s.assembleBatch([_mesh(sc)]) if batch else s.assembleFromMesh(**_mesh(sc))
        if not first:
            s.setParams(sc.params)
        s.setDomainBoundary(sc.domain[:3], sc.domain[3:])
        x, v, hc = sc.x, sc.v, np.zeros(sc.nv, np.uint8)
        for _ in range(4):
            x, v, hc = s.resolveCollision(x, scenes.candidate(sc, x, v), v, hc)
        got.append((x, v, hc))
        s.close()
    assert got[0][2].any()
    for a, b in zip(*got):
        assert np.array_equal(a, b)
