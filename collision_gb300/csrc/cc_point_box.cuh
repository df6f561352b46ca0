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
    double dt = MOVING ? scenes[vscene[p]].p.dt : 0.0;
    double4_32a x = xo[p];
    double a[3] = {x.x, x.y, x.z}, b[3] = {x.x, x.y, x.z};
    if (MOVING) {
        double4_32a v = av[p];
        double e[3] = {x.x + v.x * dt, x.y + v.y * dt, x.z + v.z * dt};
        for (int d = 0; d < 3; ++d) {
            a[d] = fmin(a[d], e[d]);
            b[d] = fmax(b[d], e[d]);
        }
    }
    lo[p] = make_float4(__double2float_rd(a[0]), __double2float_rd(a[1]), __double2float_rd(a[2]), 0.f);
    hi[p] = make_float4(__double2float_ru(b[0]), __double2float_ru(b[1]), __double2float_ru(b[2]), 0.f);
    p32[p] = make_float4((float)x.x, (float)x.y, (float)x.z, 0.f);
    if (MOVING) {
        double4_32a v = av[p];
        v32[p] = make_float4((float)v.x, (float)v.y, (float)v.z, 0.f);
    }
}

}  // namespace ccg
