"""Division by a rounded reciprocal with two remainder corrections against the
division itself, bit for bit: time steps in use, random pairs, mantissas near
one and near two, the ends of the range it takes, zeros and values that are
not finite."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA_INC = "/usr/local/cuda/include"


@pytest.fixture(scope="module")
def divide(tmp_path_factory):
    gxx = shutil.which("g++")
    if not gxx or not os.path.isdir(CUDA_INC):
        pytest.skip("needs g++ and the CUDA headers")
    so = str(tmp_path_factory.mktemp("quotient") / "libquotient.so")
    subprocess.run([gxx, "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC",
                    "-I", os.path.join(ROOT, "collision_gb300", "csrc"), "-I", CUDA_INC,
                    os.path.join(ROOT, "tests", "quotient_shim.cpp"), "-o", so], check=True)
    lib = C.CDLL(so)

    def run(a, b):
        a, b = np.ascontiguousarray(a, float), np.ascontiguousarray(b, float)
        out = np.zeros_like(a)
        lib.quotient_host(a.ctypes.data_as(C.c_void_p), b.ctypes.data_as(C.c_void_p), out.ctypes.data_as(C.c_void_p),
                          len(a))
        return out
    return run


def _ulps(rng, n):
    """Mantissas within a few units of 1 or 2."""
    return np.where(rng.random(n) < 0.5, 1.0, 2.0) + rng.integers(-40, 40, n) * 2.0 ** -52


@pytest.mark.parametrize("case", ["steps", "random", "ulps", "wide", "special"])
def test_quotient_is_the_division(divide, case):
    rng = np.random.default_rng(len(case))
    n = 200000
    a = rng.standard_normal(n)
    b = rng.uniform(0.5, 2.0, n)
    if case == "steps":
        b = rng.choice([1e-3, 5e-4, 1e-2, 0.1, 1.0 / 3.0, 1e-4, 0.25], n)
        a *= 10.0 ** rng.integers(-12, 2, n)
    elif case == "ulps":
        a, b = _ulps(rng, n), _ulps(rng, n)
    elif case == "wide":
        a, b = a * 2.0 ** rng.integers(-420, 420, n), b * 2.0 ** rng.integers(-420, 420, n)
    elif case == "special":
        v = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, 1e308, 1.0, -3.0, 2.0 ** -400, 2.0 ** 400])
        a, b = rng.choice(v, n), rng.choice(v, n)
    with np.errstate(all="ignore"):
        want = a / b
    got = divide(a, b)
    nan = np.isnan(want)
    assert np.array_equal(np.isnan(got), nan)
    assert got[~nan].tobytes() == want[~nan].tobytes()
