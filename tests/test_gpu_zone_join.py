"""A pass's impact zones joined in one CTA against the general kernels (which
run alone with TUNE_SMALL_SORT 0), with the detection loop on the device and on
the host: passes of a few records, of hundreds, of more than the CTA takes, and
movable bodies, whose pairs are not joined. Zones, their roots and every output
bit must agree."""
import numpy as np
import pytest

from collision_gb300 import scenes

pytestmark = pytest.mark.gpu

CASES = {"few": (lambda: scenes.batched(6, 16, 48, seed=3), 9), "many": (lambda: scenes.batched(48, 16, 64, seed=5), 8),
         "dense": (lambda: [scenes.folded_cloth(n=65, dt=5e-4, h=2e-3, seed=1, vscale=60.0)] * 3, 6),
         "bodies": (lambda: [scenes.deck("ball_plane", advance=0.9)], 3)}


def _run(mix, nsteps, small, device_loop):
    from collision_gb300.solver import CollisionSolver3d
    b = CollisionSolver3d(0)
    b.assembleBatch(mix)
    b.setMode(1)
    b.setZoneCap(60)
    b.setTuning(b.TUNE_SMALL_SORT, small)
    b.setTuning(b.TUNE_DEVICE_LOOP, device_loop)
    x = np.concatenate([s.x for s in mix])
    v = np.concatenate([s.v for s in mix])
    hc = np.zeros(len(x), np.uint8)
    dt = np.concatenate([np.full(s.nv, s.params["dt"]) for s in mix])[:, None]
    out = []
    for _ in range(nsteps):
        x, v, hc, _ = b.resolveCollisionBatch(x, x + dt * v, v, hc)
        c = b.counters()
        out.append((x, v, hc, b.zoneRoots(), (c["passes"], c["zone_passes"], c["zone_unions"])))
    b.close()
    return out


@pytest.mark.parametrize("case", list(CASES))
def test_join_equals_general_kernels(case):
    make, nsteps = CASES[case]
    mix = make()
    want = _run(mix, nsteps, 0, 1)
    print(case, [s[4] for s in want])
    assert case == "bodies" or any(s[4][2] > 0 for s in want)
    for small, device_loop in ((1, 1), (1, 0)):
        got = _run(mix, nsteps, small, device_loop)
        for a, b in zip(got, want):
            for u, w in zip(a[:4], b[:4]):
                assert np.array_equal(u, w)
            assert a[4][:2] == b[4][:2]
