"""The plain path's staged moving passes (the coplanarity cubic's bound, then
the full sub-tests) against the oracle's build with correctly rounded math:
near-contact element pairs of every kind, in batches whose pair counts leave
the filter's groups of sixteen threads and its blocks uneven, bit for bit."""
import numpy as np
import pytest

from oracle.ccopy import OracleSolver
from tests.test_gpu_mixed_fuzz import _cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 129, 400])
def test_plain_passes_equal_oracle(n):
    from collision_gb300.solver import CollisionSolver3d
    mix = _cases(n, 100 + n, 2)
    off = np.concatenate([[0], np.cumsum([s.nv for s in mix])])
    x = np.concatenate([s.x for s in mix])
    v = np.concatenate([s.v for s in mix])
    dt = np.concatenate([np.full((s.nv, 1), s.params["dt"]) for s in mix])
    gpu = CollisionSolver3d(0)
    gpu.assembleBatch(mix)
    ora = [OracleSolver(s, record=0, crmath=True) for s in mix]
    hc = np.zeros(len(x), np.uint8)
    for step in range(2):
        xg, vg, hg, _ = gpu.resolveCollisionBatch(x, x + dt * v, v, hc)
        for i, o in enumerate(ora):
            s = slice(off[i], off[i + 1])
            r = o.step(x[s], x[s] + dt[s] * v[s], v[s], hc[s])
            assert r["rc"] == 0
            assert np.array_equal(xg[s], r["x"]) and np.array_equal(vg[s], r["v"]), (step, i, mix[i].name)
            assert np.array_equal(hg[s], r["has_collsn"]), (step, i, mix[i].name)
        x, v, hc = xg, vg, hg
    if n >= 129:
        assert gpu.counters()["contacts"] > 0
    gpu.close()
