// The fixed-point forms of the correctly rounded functions beside their
// double-double forms, on the host (tests/test_crfix_cpu.py).
#include "../collision_gb300/csrc/cc_crmath.cuh"

extern "C" {
// out: the fixed-point result, ok: whether it counts, ref: the double-double one; est: ulps the estimate is moved by
void crfix_eval(int fn, const double* a, const int* est, double* out, unsigned char* ok, double* ref, int n) {
    using namespace ccg::cr;
    for (int i = 0; i < n; ++i) {
        const double x = a[i];
        auto moved = [&](double y) {
            for (int k = 0; k < est[i]; ++k) y = std::nextafter(y, 1e308);
            for (int k = 0; k > est[i]; --k) y = std::nextafter(y, -1e308);
            return y;
        };
        switch (fn) {
            case 0: ok[i] = fx::sin_or_cos(x, true, &out[i]), ref[i] = cos_slow(x); break;
            case 1: ok[i] = fx::sin_or_cos(x, false, &out[i]), ref[i] = sin_slow(x); break;
            case 2:
                ok[i] = fx::acos_from(x, moved(::acos(std::fabs(x) > 0.5 ? std::fabs(x) : x)), &out[i]);
                ref[i] = acos_slow(x);
                break;
            default: ok[i] = fx::cube_root_from(x, moved(::cbrt(x)), &out[i]), ref[i] = pow_slow(x, 1.0 / 3.0); break;
        }
    }
}
}
