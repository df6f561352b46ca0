"""A program's very first step builds a scene's two reference trees side by
side, as its later scenes do: in a fresh process the first solver's builds
take about as long as a second one's (twice as long if one waits for the
other)."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = """
import numpy as np
from collision_gb300 import scenes
from collision_gb300.solver import CollisionSolver3d
sc = scenes.cloth_on_obstacle(129, "box", 0.2, 2.0, seed=3, gap=3e-3)
for _ in range(2):
    s = CollisionSolver3d(0)
    s.assembleFromScene(sc)
    s.resolveCollision(sc.x, scenes.candidate(sc, sc.x, sc.v), sc.v, np.zeros(sc.nv, np.uint8))
    print(s.counters()["tree_builds"], s.counters()["tree_build_us"])
    s.close()
"""


def test_first_trees_side_by_side():
    out = subprocess.run([sys.executable, "-c", PROGRAM], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr
    (n0, us0), (n1, us1) = [tuple(map(int, line.split())) for line in out.stdout.splitlines()[-2:]]
    assert n0 == n1 == 2
    assert us0 < 1.5 * us1
