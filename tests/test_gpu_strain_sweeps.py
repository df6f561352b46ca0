"""The pipelined strain sweeps against the kernel that walks the edge schedule
in global memory (setStrainWindow(False)): sheets of a few edges, odd and long
ones, separate strings, several scenes at once, and a sheet whose levels are
too wide for the shared-memory ring of records. Both make the same
Gauss-Seidel steps in the same order, so the bits must be equal."""
import numpy as np
import pytest

from collision_gb300 import scenes

pytestmark = pytest.mark.gpu


def _waves(x, spacing, dt):
    """In-plane waves whose strain reaches a quarter, three spacings high."""
    k = 0.25 / (3.0 * spacing)
    a = 3.0 * spacing / dt
    return np.stack([a * np.sin(k * x[:, 0] + 0.3), a * np.sin(k * x[:, 1] + 0.7), np.zeros(len(x))], axis=1)


def _sheet(n, dt=1e-3):
    """A wavy sheet in free space, stretched and compressed by its velocities."""
    p, t = scenes.grid_cloth(n, 1.0, 0.5)
    p[:, 2] += 0.02 * np.sin(5.0 * p[:, 0]) * np.cos(4.0 * p[:, 1])
    spacing = 1.0 / (n - 1)
    return scenes.assemble(f"waves{n}", [(p, t, _waves(p, spacing, dt), False)],
                           dict(dt=dt, thickness=0.01 * spacing))


def _strings(n, nseg, dt=1e-3):
    """n parallel strings, stretched along their length."""
    x = np.stack([np.tile(np.arange(nseg + 1) / nseg, n), np.repeat(np.arange(n) * 0.1, nseg + 1),
                  np.full(n * (nseg + 1), 0.5)], axis=1)
    x[:, 2] += 0.02 * np.sin(5.0 * x[:, 0])
    i = np.arange(nseg)
    bonds = np.concatenate([np.stack([i, i + 1], axis=1) + s * (nseg + 1) for s in range(n)]) + 8
    bp, bt = scenes.box_mesh((-0.2, -0.2, -1.1), (0.2, 0.2, -1.0))
    return scenes.assemble(f"lines{n}", [(bp, bt, np.zeros_like(bp), True),
                                         (x, None, _waves(x, 1.0 / nseg, dt), False)],
                           dict(dt=dt, thickness=0.01 / nseg), bonds=bonds,
                           bond_curve=np.repeat(np.arange(n, dtype=np.int32), nseg))


CASES = {"sheet2": lambda: [_sheet(2)], "sheet3": lambda: [_sheet(3)], "sheet17": lambda: [_sheet(17)],
         "sheet32": lambda: [_sheet(32)], "sheet130": lambda: [_sheet(130)], "sheet420": lambda: [_sheet(420)],
         "line1": lambda: [_strings(1, 1)], "lines3": lambda: [_strings(3, 700)],
         "several": lambda: [_sheet(2), _sheet(41), _strings(2, 33), _sheet(5), _sheet(64)]}


@pytest.mark.parametrize("case", list(CASES))
def test_sweeps_equal_global_path(case):
    from collision_gb300.solver import CollisionSolver3d
    scs = CASES[case]()
    x = np.concatenate([sc.x for sc in scs])
    v = np.concatenate([sc.v for sc in scs])
    xc = np.concatenate([scenes.candidate(sc, sc.x, sc.v) for sc in scs])
    got = []
    for window in (True, False):
        s = CollisionSolver3d(0)
        s.assembleBatch(scs)
        s.setStrainWindow(window)
        r = s.resolveCollisionBatch(x, xc, v, np.zeros(len(x), np.uint8))
        got.append((r[:3], s.counters()["strain_averaged"]))
        s.close()
    assert got[0][1] == got[1][1]
    assert got[0][1] > 0 or len(x) < 200
    for a, b in zip(got[0][0], got[1][0]):
        assert np.array_equal(a, b)
