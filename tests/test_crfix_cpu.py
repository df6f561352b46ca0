"""The fixed-point forms of cos, sin, acos and the cube root against their
double-double forms (host build): where a fixed-point result counts it is the
same double, and it counts for nearly every argument in the range used; the
estimates that acos and the cube root start from may be a few ulp off."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("needs g++")
    so = str(tmp_path_factory.mktemp("crfix") / "libcrfix.so")
    subprocess.run([gxx, "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC",
                    os.path.join(HERE, "crfix_host.cpp"), "-o", so], check=True)
    return C.CDLL(so)


def _args(case, rng, n):
    u = rng.random(n)
    sign = rng.choice([-1.0, 1.0], n)
    return {"cos_wide": (0, sign * 7.99 * u), "cos_small": (0, sign * 10 ** (-7 * u)),
            "cos_quarters": (0, np.pi / 4 * rng.integers(1, 10, n) + sign * 10 ** (-8 * u)),
            "sin_wide": (1, sign * 7.99 * u), "sin_small": (1, sign * 10 ** (-17 * u)),
            "sin_quarters": (1, np.pi / 4 * rng.integers(1, 10, n) + sign * 10 ** (-8 * u)),
            "acos": (2, sign * u * (1 - 2.0 ** -53)), "acos_ends": (2, sign * (1 - 10 ** (-15.5 * u))),
            "acos_zero": (2, sign * 10 ** (-17 * u)),
            "root": (3, 10 ** (60 * u - 30)), "root_wide": (3, 10 ** (580 * u - 290))}[case]


@pytest.mark.parametrize("case", ["cos_wide", "cos_small", "cos_quarters", "sin_wide", "sin_small", "sin_quarters",
                                  "acos", "acos_ends", "acos_zero", "root", "root_wide"])
def test_fixed_point_is_the_double_double_value(lib, case):
    n = 40000
    rng = np.random.default_rng(sum(map(ord, case)))
    fn, a = _args(case, rng, n)
    a = np.ascontiguousarray(a)
    est = rng.integers(-3, 4, n).astype(np.int32)
    out, ref, ok = np.zeros(n), np.zeros(n), np.zeros(n, np.uint8)
    lib.crfix_eval(fn, a.ctypes.data_as(C.c_void_p), est.ctypes.data_as(C.c_void_p), out.ctypes.data_as(C.c_void_p),
                   ok.ctypes.data_as(C.c_void_p), ref.ctypes.data_as(C.c_void_p), n)
    ok = ok.astype(bool)
    assert ok.mean() > 0.99, case
    assert np.array_equal(out[ok], ref[ok]), case
