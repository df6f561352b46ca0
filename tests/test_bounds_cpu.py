"""The FP32 bounds that end a sub-test before its FP64 form, against that
form (host build of both): no sub-test they rule out hits, or meets a
degenerate normal, where the bounds are tightest - points and edges at the
reach, triangles of any thinness and size, far from the origin, at rest and
moving - and a cubic's roots are those of the reference's formulas with
nothing in front of them."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "collision_gb300", "csrc")
CUDA_INC = "/usr/local/cuda/include"
MACH_EPS = np.finfo(float).eps


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    gxx = shutil.which("g++")
    if not gxx or not os.path.isdir(CUDA_INC):
        pytest.skip("needs g++ and the CUDA headers")
    so = str(tmp_path_factory.mktemp("bounds") / "libbounds.so")
    subprocess.run([gxx, "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-I", CSRC, "-I", CUDA_INC,
                    os.path.join(HERE, "bounds_shim.cpp"), "-o", so], check=True)
    return C.CDLL(so)


def _ptr(a):
    return a.ctypes.data_as(C.c_void_p)


def _unit(rng, n):
    d = rng.normal(size=(n, 3))
    return d / np.linalg.norm(d, axis=1)[:, None]


def _across(rng, d):
    return (lambda u: u / np.linalg.norm(u, axis=1)[:, None])(np.cross(d, _unit(rng, len(d))))


def _slivers(rng, n, size):
    """Three points almost on a line and a fourth on it, near it, or past its ends; heights around the
    determinant's cut and above."""
    d = _unit(rng, n)
    h = 4.7e-7 / size * 10 ** rng.uniform(-0.5, 3.5, n)
    x = np.zeros((n, 4, 3))
    x[:, 0] = size * rng.uniform(-1, 1, (n, 1)) * d
    x[:, 1] = size * rng.uniform(-1, 1, (n, 1)) * d + h[:, None] * _across(rng, d)
    off = size * 10 ** rng.uniform(-9, 0, n) * rng.integers(0, 2, n)
    x[:, 3] = size * rng.uniform(-3, 3, (n, 1)) * d + off[:, None] * _across(rng, d)
    return x


def _at_reach(rng, n, size, h, ee):
    """Triangles (as flat as 1e-6) with a point, or pairs of edges, h apart to within 1e-3 of h."""
    d = _unit(rng, n)
    u = _across(rng, d)
    nrm = np.cross(d, u)
    flat = 10 ** rng.uniform(-6, 0, (n, 1))
    x = np.zeros((n, 4, 3))
    gap = (h * (1 + 10 ** rng.uniform(-9, -3, n) * rng.choice([-1, 1], n)))[:, None] * nrm
    if ee:
        x[:, 0], x[:, 1] = -size * rng.random((n, 1)) * d, size * rng.random((n, 1)) * d
        x[:, 2], x[:, 3] = -flat * size * u - size * rng.random((n, 1)) * d + gap, flat * size * u + gap
    else:
        x[:, 0], x[:, 1] = size * d, flat * size * u
        w = rng.random((n, 2)) * 1.02 - 0.01
        x[:, 3] = w[:, :1] * x[:, 0] + w[:, 1:] * x[:, 1] + gap
    return x


def _hittable(kind, size):
    """The point-triangle test returns false below det = 1000 MACH_EPS, whatever the point."""
    return kind != "point" or size ** 4 > 1000 * MACH_EPS


CASES = [("sliver", s) for s in (0.1, 0.35, 1.0, 4.0, 10.0, 100.0)] + \
        [("point", s) for s in (1e-4, 0.01, 1.0, 30.0)] + [("edges", s) for s in (1e-4, 0.01, 1.0, 30.0)]


@pytest.mark.parametrize("kind,size", CASES)
@pytest.mark.parametrize("far", [0.0, 1.0, 1e4])
def test_static_bound_rules_out_no_hit(lib, kind, size, far):
    n = 60000
    rng = np.random.default_rng([len(kind), int(size * 1e5), int(far)])
    h = 1e-3 if kind == "sliver" else 0.1 * size
    x = _slivers(rng, n, size) if kind == "sliver" else _at_reach(rng, n, size, h, kind == "edges")
    x = np.ascontiguousarray(x + far * _unit(rng, n)[:, None, :])
    ee = np.full(n, kind == "edges", np.uint8)
    out = np.zeros(n, np.uint8)
    lib.static_bounds(_ptr(x), _ptr(ee), C.c_double(h), C.c_double(1e-6), _ptr(out), n)
    hit = (out & 2) != 0
    assert not (hit & ((out & 1) != 0)).any()
    if _hittable(kind, size):
        assert hit.sum() > 20, "too few hits to tell anything"


@pytest.mark.parametrize("kind,size", CASES)
@pytest.mark.parametrize("far", [0.0, 1e4])
def test_moving_bounds_rule_out_no_hit(lib, kind, size, far):
    n = 60000
    rng = np.random.default_rng([len(kind), int(size * 1e5), int(far), 1])
    dt, eps = 1e-3, 1e-6 if kind == "sliver" else 1e-3 * size
    xt = _slivers(rng, n, size) if kind == "sliver" else _at_reach(rng, n, size, eps, kind == "edges")
    xt = xt + far * _unit(rng, n)[:, None, :]
    t = dt * rng.random(n)
    v = rng.normal(size=(n, 1, 3)) * 3 + rng.normal(size=(n, 4, 3)) * size * 10 ** rng.uniform(-6, 3, (n, 1, 1))
    x = np.ascontiguousarray(xt - t[:, None, None] * v)
    v = np.ascontiguousarray(v)
    ee = np.full(n, kind == "edges", np.uint8)
    out = np.zeros(n, np.uint8)
    lib.moving_bounds(_ptr(x), _ptr(v), _ptr(t), _ptr(ee), C.c_double(dt), C.c_double(eps), _ptr(out), n)
    hit = (out & 4) != 0
    assert not (hit & ((out & 1) != 0)).any(), "the moving filter"
    assert not (hit & ((out & 2) != 0)).any(), "misses_at"
    if far == 0.0 and _hittable(kind, size):
        assert hit.sum() > 20, "too few hits to tell anything"


@pytest.mark.parametrize("kind", ["ends", "near_double", "complex", "scaled", "low_degree"])
def test_roots_are_the_references(lib, kind):
    """Roots at 0, dt and dt + 2 MACH_EPS among others, almost double and complex pairs."""
    n, dt = 200000, 1e-3
    rng = np.random.default_rng(sum(map(ord, kind)))
    ends = rng.choice([0.0, MACH_EPS, 2 * MACH_EPS, dt, dt + MACH_EPS, dt + 2 * MACH_EPS, 0.5 * dt], n)
    r0 = ends + dt * 10 ** rng.uniform(-17, 0, n) * rng.choice([-1, 0, 1], n)
    r1 = dt * rng.normal(size=n) * 10 ** rng.uniform(-1, 3, n)
    r2 = dt * rng.normal(size=n) * 10 ** rng.uniform(-1, 3, n)
    if kind == "near_double":
        r1, r2 = r0, r0 + dt * 10 ** rng.uniform(-12, -1, n) * rng.choice([-1, 1], n)
    lead = 10 ** rng.uniform(-12 if kind == "scaled" else -3, 3, n) * rng.choice([-1, 1], n)
    if kind == "complex":
        im2 = (dt * 10 ** rng.uniform(-9, 2, n)) ** 2
        b1, b0 = -2 * r1, r1 * r1 + im2
    else:
        b1, b0 = -(r1 + r2), r1 * r2
    coef = np.stack([lead, lead * (b1 - r0), lead * (b0 - r0 * b1), -lead * r0 * b0], 1)
    if kind == "low_degree":
        coef[:, 0] = MACH_EPS * rng.choice([0.0, 0.9, -1.0], n)
        coef[:, 1] *= rng.choice([0.0, 1.0], n)
        coef[:, 3] = -coef[:, 2] * r0
    coef = np.ascontiguousarray(coef)
    got, want = np.zeros((n, 3)), np.zeros((n, 3))
    ga, wa = np.zeros(n, np.uint8), np.zeros(n, np.uint8)
    lib.cubic_roots(_ptr(coef), C.c_double(dt), _ptr(got), _ptr(ga), _ptr(want), _ptr(wa), n)
    assert np.array_equal(ga, wa)
    on = wa != 0
    assert on.sum() > 1000
    assert np.array_equal(got[on], want[on])
