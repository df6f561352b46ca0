// The filters' FP32 data of one point.
#pragma once

#include "cc_launch.h"

namespace ccg {

// FP32 box of every point over the pass's time window, rounded outward:
// [x_old] for proximity, [x_old, x_old + dt*avgVel] for CCD.
template <bool MOVING>
__device__ __forceinline__ void point_box(const double4_32a* __restrict__ xo, const double4_32a* __restrict__ av,
                                          const int* __restrict__ vscene, const SceneDev* __restrict__ scenes, int p,
                                          float4* lo, float4* hi, float4* p32, float4* v32) {
    const double4_32a x = xo[p];
    const double xs[3] = {x.x, x.y, x.z};
    double a[3], b[3];
    for (int d = 0; d < 3; ++d) a[d] = b[d] = xs[d];
    if (MOVING) {
        const double dt = scenes[vscene[p]].p.dt;
        const double4_32a v = av[p];
        const double vs[3] = {v.x, v.y, v.z};
        for (int d = 0; d < 3; ++d) {
            const long long o = order_of(xs[d]), e = order_of(xs[d] + vs[d] * dt);
            a[d] = of_order(o < e ? o : e);
            b[d] = of_order(o > e ? o : e);
        }
        v32[p] = make_float4((float)v.x, (float)v.y, (float)v.z, 0.f);
    }
    lo[p] = make_float4(cut32_down(a[0]), cut32_down(a[1]), cut32_down(a[2]), 0.f);
    hi[p] = make_float4(cut32_up(b[0]), cut32_up(b[1]), cut32_up(b[2]), 0.f);
    p32[p] = make_float4((float)x.x, (float)x.y, (float)x.z, 0.f);
}

}  // namespace ccg
