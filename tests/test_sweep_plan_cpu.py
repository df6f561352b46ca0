"""The schedule of the pipelined strain sweeps, on the CPU: a host model that
takes the sweeps' steps in random orders their waits allow must give the
sequential sweeps' values (tests/sweep_plan_shim.cpp)."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

from collision_gb300 import scenes

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA_INC = "/usr/local/cuda/include"


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    gxx = shutil.which("g++")
    if not gxx or not os.path.isdir(CUDA_INC):
        pytest.skip("needs g++ and the CUDA headers")
    so = str(tmp_path_factory.mktemp("sweep_plan") / "libsweep_plan.so")
    src = os.path.join(ROOT, "collision_gb300", "csrc")
    subprocess.run([gxx, "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-I", src, "-I", CUDA_INC,
                    os.path.join(ROOT, "tests", "sweep_plan_shim.cpp"), os.path.join(src, "cc_sweep_plan.cpp"),
                    "-o", so], check=True)
    lib = C.CDLL(so)
    ip = C.POINTER(C.c_int)
    lib.sweep_plan_check.argtypes = [ip, C.c_int, ip, C.c_int, C.c_int, C.c_int, ip]

    def run(tris, bonds, nv, seed):
        t = np.ascontiguousarray(tris, np.int32).reshape(-1, 3)
        b = np.ascontiguousarray(bonds, np.int32).reshape(-1, 2)
        info = np.zeros(6, np.int32)
        ptr = lambda a: a.ctypes.data_as(ip)  # noqa: E731
        return lib.sweep_plan_check(ptr(t), len(t), ptr(b), len(b), nv, seed, ptr(info)), info
    return run


def _cloth(n):
    p, t = scenes.grid_cloth(n)
    return t, np.zeros((0, 2)), len(p)


def _shuffled(n, seed):
    t, b, nv = _cloth(n)
    rng = np.random.default_rng(seed)
    return rng.permutation(nv)[t][rng.permutation(len(t))], b, nv


def _strings():
    s = scenes.strings(nstr=5, nseg=40, seed=4)
    return np.zeros((0, 3)), s.bonds, s.nv


def _mixed():
    t, _, nv = _cloth(9)
    chain = np.stack([np.arange(30), np.arange(1, 31)], axis=1) + nv
    return t, np.concatenate([chain, [[0, nv], [0, 5]]]), nv + 31


@pytest.mark.parametrize("make", [lambda: _cloth(2), lambda: _cloth(3), lambda: _cloth(17), lambda: _cloth(130),
                                  lambda: _shuffled(23, 1), lambda: _shuffled(70, 2), _strings, _mixed],
                         ids=["cloth2", "cloth3", "cloth17", "cloth130", "shuffled23", "shuffled70", "strings", "mixed"])
def test_pipelined_sweeps_equal_the_sequential_ones(check, make):
    tris, bonds, nv = make()
    for seed in range(3):
        rc, info = check(tris, bonds, nv, seed)
        assert rc == 0, (rc, info)

