// The FP32 bounds in front of the FP64 tests beside those tests, on the host
// (tests/test_bounds_cpu.py): the device text with host forms of what it
// calls.
#include "cc_common.cuh"

#include <algorithm>
#include <vector>

namespace ccg {
inline int atomicOr(int* p, int v) {
    const int old = *p;
    *p |= v;
    return old;
}
inline int aggregated_add(int* p, int n) {
    const int old = *p;
    *p += n;
    return old;
}
// sums of two floats and their products, rounded up or down (the double sum
// or product is exact, or off by far less than its distance to a float)
inline float rounded_up(double x) { return cut32_up(x); }
inline float rounded_down(double x) { return cut32_down(x); }
inline float __fadd_ru(float a, float b) { return rounded_up((double)a + b); }
inline float __fsub_ru(float a, float b) { return rounded_up((double)a - b); }
inline float __fsub_rd(float a, float b) { return rounded_down((double)a - b); }
inline float __fmul_ru(float a, float b) { return rounded_up((double)a * b); }
}  // namespace ccg

#include "cc_narrow.cuh"

using namespace ccg;

namespace {

struct Host {
    double4_32a xo[4], av[4];
    uint8_t fixed[4] = {0, 0, 0, 0};
    PassCounters ctr;
    NarrowCtx c;
    CallState st;
    Host(const double* x, const double* v, const Params& p) : ctr(), c(), st() {
        for (int q = 0; q < 4; ++q) {
            xo[q] = make_double4_32a(x[3 * q], x[3 * q + 1], x[3 * q + 2], 0.0);
            av[q] = make_double4_32a(v[3 * q], v[3 * q + 1], v[3 * q + 2], 0.0);
        }
        c.xo = xo;
        c.av = av;
        c.fixed = fixed;
        c.ctr = &ctr;
        c.check = 1;
        c.p = p;
    }
    // the FP64 test at the given positions: a hit, or the reference's exit
    bool hits(bool ee, const double (*X)[3], double h) {
        const int pts[4] = {0, 1, 2, 3};
        ctr.err = 0;
        const bool hit = ee ? edge_to_edge(c, st, pts, X, h) : point_to_tri(c, st, pts, X, h);
        return hit || (ctr.err & kErrNan);
    }
    void at(double t, double (*X)[3]) const {
        for (int q = 0; q < 4; ++q) {
            const double x[3] = {xo[q].x, xo[q].y, xo[q].z}, v[3] = {av[q].x, av[q].y, av[q].z};
            for (int k = 0; k < 3; ++k) X[q][k] = x[k] + t * v[k];
        }
    }
};

}  // namespace

extern "C" {

// Bit 0: the static filter rules the test out, bit 1: the FP64 test hits.
void static_bounds(const double* x, const uint8_t* ee, double thickness, double eps, uint8_t* out, int n) {
    const double zero[12] = {0};
    const int pts[4] = {0, 1, 2, 3};
    Params p{};
    p.dt = 1e-3, p.thickness = thickness, p.eps = eps;
    for (int i = 0; i < n; ++i) {
        Host h(x + 12 * i, zero, p);
        double X[4][3];
        h.at(0.0, X);
        out[i] = (plain_may_hit<false>(h.xo, h.av, pts, ee[i], p) ? 0 : 1) | (h.hits(ee[i], X, thickness) ? 2 : 0);
    }
}

// At time t of each: bit 0 the moving filter rules the sub-test out, bit 1
// misses_at does, bit 2 the FP64 test at t hits.
void moving_bounds(const double* x, const double* v, const double* t, const uint8_t* ee, double dt, double eps,
                   uint8_t* out, int n) {
    const int pts[4] = {0, 1, 2, 3};
    Params p{};
    p.dt = dt, p.eps = eps;
    for (int i = 0; i < n; ++i) {
        Host h(x + 12 * i, v + 12 * i, p);
        double X[4][3];
        h.at(t[i], X);
        // as moving_test calls it
        F3 x32[4], v32[4];
        float most = 0.f;
        double dx[3], dv[3];
        for (int q = 1; q < 4; ++q) {
            for (int k = 0; k < 3; ++k) dx[k] = x[12 * i + 3 * q + k] - x[12 * i + k], dv[k] = v[12 * i + 3 * q + k] - v[12 * i + k];
            x32[q] = cut_f3(dx);
            v32[q] = cut_f3(dv);
            most = fmaxf(most, fmaxabs(x32[q]) + (float)dt * fmaxabs(v32[q]));
        }
        most += fmaxabs(cut_f3(x + 12 * i)) + (float)dt * fmaxabs(cut_f3(v + 12 * i));
        const float t32 = cut32(t[i]), slack = most * 0x1p-44f, h32 = (float)eps * 1.001f, e32 = (float)eps;
        const bool miss = ee[i] ? misses_at<true>(x32, v32, t32, slack, h32, e32)
                                : misses_at<false>(x32, v32, t32, slack, h32, e32);
        out[i] = (plain_may_hit<true>(h.xo, h.av, pts, ee[i], p) ? 0 : 1) | (miss ? 2 : 0) |
                 (h.hits(ee[i], X, eps) ? 4 : 0);
    }
}

// isCoplanar (dcollid3d.cpp:371-482) on the coefficients of a t^3 + b t^2 +
// c t + d: is_coplanar's roots and return value, and those of the reference's
// formulas with no test in front of them.
void cubic_roots(const double* coef, double dt, double* got, uint8_t* got_any, double* want, uint8_t* want_any, int n) {
    for (int i = 0; i < n; ++i) {
        const double* q = coef + 4 * i;
        double r[4] = {-1, -1, -1, dt};
        int ncr = 0;
        got_any[i] = is_coplanar(Cubic{q[0], q[1], q[2], q[3]}, dt, r, &ncr);
        for (int k = 0; k < 3; ++k) got[3 * i + k] = r[k];
        double a = q[0], b = q[1], c = q[2], d = q[3];
        double w[3] = {-1, -1, -1};
        if (std::fabs(a) > kMachEps) {
            b /= a; c /= a; d /= a;
            a = b; b = c; c = d;
            const double Q = (a * a - 3 * b) / 9, R = (2 * a * a * a - 9 * a * b + 27 * c) / 54;
            const double Q3 = Q * Q * Q, R2 = R * R;
            if (R2 < Q3) {
                const double s = std::sqrt(Q), theta = cr::acos(R / std::sqrt(Q3));
                w[0] = -2 * s * cr::cos(theta / 3) - a / 3;
                w[1] = -2 * s * cr::cos((theta + 2 * kPi) / 3) - a / 3;
                w[2] = -2 * s * cr::cos((theta - 2 * kPi) / 3) - a / 3;
            } else {
                const double A = -(R > 0 ? 1.0 : -1.0) * cr::pow(std::fabs(R) + std::sqrt(R2 - Q3), 1.0 / 3.0);
                const double B = std::fabs(A) < kRoundEps ? 0.0 : Q / A;
                w[0] = (A + B) - a / 3.0;
                if (std::fabs(A - B) < kRoundEps) w[1] = w[2] = -0.5 * (A + B) - a / 3.0;
            }
        } else {
            a = b; b = c; c = d;
            const double delta = b * b - 4.0 * a * c;
            if (std::fabs(a) > kRoundEps && delta > 0) {
                w[0] = (-b + std::sqrt(delta)) / (2.0 * a);
                w[1] = (-b - std::sqrt(delta)) / (2.0 * a);
            } else if (std::fabs(a) < kRoundEps && std::fabs(b) > kRoundEps) {
                w[0] = -c / b;
            }
        }
        bool any = false;
        for (int k = 0; k < 3; ++k) {
            w[k] -= kMachEps;
            if (w[k] < 0 || w[k] > dt) w[k] = -1;
            any |= w[k] > kMachEps;
        }
        std::sort(w, w + 3);
        for (int k = 0; k < 3; ++k) want[3 * i + k] = w[k];
        want_any[i] = any;
    }
}
}
