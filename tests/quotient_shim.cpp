// The division by a reciprocal, on the host (tests/test_quotient_cpu.py).
#include "cc_common.cuh"

extern "C" void quotient_host(const double* a, const double* b, double* out, int n) {
    for (int i = 0; i < n; ++i) out[i] = ccg::quotient(a[i], b[i], 1.0 / b[i]);
}
