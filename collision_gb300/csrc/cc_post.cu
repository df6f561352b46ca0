// Per-point stages around the detection passes: average velocity, applying
// a pass's impulses, impact-zone rigid motion, the domain clamp, final
// positions and final velocities (dcollid.cpp:116-220, 290-310, 562-624,
// 677-751; dcollid3d.cpp:70-200).
#include "cc_launch.h"
#include "cc_narrow.cuh"

namespace ccg {

namespace {

inline int nblk(int n, int t) { return (n + t - 1) / t; }

// computeAverageVelocity, dcollid.cpp:160-220: avgVel = (x_cand - x_old)/dt.
// Its FP64 instructions bound it: 768,000 points 87 -> 35 us with quotients
// by the scene's 1 / dt.
__global__ void k_step_init(const double* __restrict__ x_old, const double* __restrict__ x_cand, int nv,
                            const uint8_t* __restrict__ in_elem, const int* __restrict__ vscene,
                            const SceneDev* __restrict__ scenes, double4_32a* xo, double4_32a* av,
                            PassCounters* ctr) {
    int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= nv) return;
    double o[3] = {x_old[3 * p], x_old[3 * p + 1], x_old[3 * p + 2]};
    xo[p] = make_double4_32a(o[0], o[1], o[2], 0.0);
    if (!in_elem[p]) return;
    const SceneDev& sd = scenes[vscene[p]];
    const double dt = sd.p.dt, inv = sd.inv_dt;
    const bool moves = dt > kRoundEps;
    double v[3];
    bool bad = false;
    for (int j = 0; j < 3; ++j) {
        v[j] = moves ? quotient(x_cand[3 * p + j] - o[j], dt, inv) : 0.0;
        if (((unsigned)__double2hiint(v[j]) & 0x7ff00000u) == 0x7ff00000u) bad = true;  // not finite
    }
    if (bad) atomicOr(&ctr->err, kErrNan);
    av[p] = make_double4_32a(v[0], v[1], v[2], 0.0);
}

// Contributions by point: counted, with the points that have any listed ...
__global__ void k_contrib_count(const Contrib* __restrict__ c, PassCounters* ctr, int cap, int* cnt, int* touched) {
    if (ctr->err & kErrRetry) return;
    int n = ctr->ncontrib < cap ? ctr->ncontrib : cap;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int v = c[i].vertex;
        if (atomicAdd(&cnt[v], 1) == 0) touched[aggregated_add(&ctr->ntouch, 1)] = v;
    }
}

// ... given a segment each (in any order) ...
__global__ void k_contrib_segments(PassCounters* ctr, const int* __restrict__ cnt, const int* __restrict__ touched,
                                   int* off) {
    if (ctr->err & kErrRetry) return;
    const int n = ctr->ntouch;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
        const int v = touched[t];
        off[v] = aggregated_add(&ctr->nseg_used, cnt[v]);
    }
}

// ... and listed there.
__global__ void k_contrib_scatter(const Contrib* __restrict__ c, const PassCounters* ctr, int cap,
                                  const int* __restrict__ off, int* cur, int* idx) {
    if (ctr->err & kErrRetry) return;
    int n = ctr->ncontrib < cap ? ctr->ncontrib : cap;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        int v = c[i].vertex;
        idx[off[v] + atomicAdd(&cur[v], 1)] = i;
    }
}

// updateAverageVelocity, dcollid.cpp:677-751, one warp per point with
// contributions: they are put in visiting order and summed one by one from
// zero, as the reference accumulates collsnImpulse and friction. Slots nv..
// are the movable bodies: their spread impulses are added one by one onto the
// body's running collsnImpulse_RG, which the reference never clears, and
// their count is the pass's collsn_num_RG.
//
// The order: each lane ranks its contributions' keys against all of the
// point's, in shared memory for up to kApplyStage (one thread's insertion
// sort loaded two dependent values per comparison: 1.7 ms for a folding
// sheet's proximity pass, whose points meet up to hundreds of sub-tests).
// The sums: lanes 0..2 add the impulse's components and lanes 3..5 the
// friction's, in order. The point's counters are left zero for the next pass.
constexpr int kApplyWarps = 4;
constexpr int kApplyStage = 256;
__global__ void __launch_bounds__(kApplyWarps * 32) k_apply(
    const Contrib* __restrict__ c, PassCounters* ctr, int* cnt, int* cur, const int* __restrict__ off,
    const int* __restrict__ touched, const int* __restrict__ idx, int* ord, int nv, double4_32a* av,
    uint8_t* has_collsn, double4_32a* dump, double4_32a* body_acc, int* body_num, PassStamp ps) {
    __shared__ unsigned long long s_key[kApplyWarps][kApplyStage];
    __shared__ int s_ord[kApplyWarps][kApplyStage];
    if (ctr->err & kErrRetry) return;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int m = ctr->ntouch;
    for (int t = blockIdx.x * kApplyWarps + w; t < m; t += gridDim.x * kApplyWarps) {
        const int p = touched[t], n = cnt[p], o = off[p];
        const bool staged = n <= kApplyStage;
        unsigned long long* key = s_key[w];
        int* order = staged ? s_ord[w] : ord + o;
        __syncwarp();
        if (lane == 0) cnt[p] = cur[p] = 0;
        if (n == 1) {
            if (lane == 0) order[0] = idx[o];
        } else {
            if (staged)
                for (int i = lane; i < n; i += 32) key[i] = c[idx[o + i]].key;
            __syncwarp();
            for (int i = lane; i < n; i += 32) {
                const int x = idx[o + i];
                const unsigned long long kx = staged ? key[i] : c[x].key;
                int r = 0;
                for (int j = 0; j < n; ++j) {
                    const unsigned long long kj = staged ? key[j] : c[idx[o + j]].key;
                    r += kj < kx || (kj == kx && j < i);
                }
                order[r] = x;
            }
        }
        __syncwarp();
        const bool body = p >= nv;
        double acc = 0.0;
        if (body && lane < 3) {
            const double4_32a a = body_acc[p - nv];
            acc = lane == 0 ? a.x : lane == 1 ? a.y : a.z;
        }
        if (lane < (body ? 3 : 6)) {
#pragma unroll 4
            for (int i = 0; i < n; ++i) {
                const Contrib& q = c[order[i]];
                const double x = lane < 3 ? q.imp[lane] : q.fric[lane - 3];
                if (lane < 3 || (q.flags & 1)) acc += x;
            }
        }
        double imp[3], fric[3];
        for (int k = 0; k < 3; ++k) {
            imp[k] = __shfl_sync(0xffffffffu, acc, k);
            fric[k] = __shfl_sync(0xffffffffu, acc, 3 + k);
        }
        if (lane == 0 && body) {
            body_acc[p - nv] = make_double4_32a(imp[0], imp[1], imp[2], 0.0);
            body_num[p - nv] = n;
        } else if (lane == 0) {
            double4_32a a = av[p];
            double v[3] = {a.x, a.y, a.z};
            bool bad = false;
            for (int k = 0; k < 3; ++k) {
                v[k] += (imp[k] + fric[k]) / n;
                if (!isfinite(v[k])) bad = true;
            }
            if (bad) atomicOr(&ctr->err, kErrNan);
            av[p] = make_double4_32a(v[0], v[1], v[2], 0.0);
            has_collsn[p] = 1;
            stamp_point(ps, p);
            if (dump) dump[p] = make_double4_32a(imp[0], imp[1], imp[2], (double)n);  // collsnImpulse, collsn_num
        }
    }
}

// The spread part of updateAverageVelocity (dcollid.cpp:726-733), after
// each point's own impulses: avgVel += collsnImpulse_RG / collsn_num_RG for
// every member of a body that received spread impulses this pass.
__global__ void k_apply_rg(const int* __restrict__ members, const int* __restrict__ member_body, int nmembers,
                           const PassCounters* ctr, const double4_32a* __restrict__ body_acc,
                           const int* __restrict__ body_num, const uint8_t* __restrict__ fixed, double4_32a* av,
                           uint8_t* has_collsn, PassStamp ps) {
    if (ctr->err & kErrRetry) return;
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nmembers) return;
    const int b = member_body[i], n = body_num[b];
    const int p = members[i];
    if (n == 0 || (fixed[p] & 1)) return;
    const double4_32a a = body_acc[b];
    double4_32a v = av[p];
    v.x += a.x / n;
    v.y += a.y / n;
    v.z += a.z / n;
    av[p] = v;
    has_collsn[p] = 1;
    stamp_point(ps, p);
}

__device__ __forceinline__ double det3(const double (*a)[3]) {
    return a[0][0] * (a[1][1] * a[2][2] - a[2][1] * a[1][2]) - a[0][1] * (a[1][0] * a[2][2] - a[2][0] * a[1][2]) +
           a[0][2] * (a[1][0] * a[2][1] - a[2][0] * a[1][1]);
}

// What every member's motion divides by: w . w and dt, and their inverses.
struct ZoneInverses {
    double ww, of_ww, of_dt;
};
__device__ __forceinline__ ZoneInverses zone_inverses(const double* w, double inv_dt) {
    const double ww = dot3(w, w);
    return ZoneInverses{ww, 1.0 / ww, inv_dt};
}

// The last loop of updateImpactListVelocity (dcollid3d.cpp:160-199) for one
// member p of a zone: its new average velocity from the zone's rigid motion
// (centre x_cm moving at v_cm, angular velocity w of magnitude mag_w, and
// sw = sin(dt mag_w) / mag_w, cw = cos(dt mag_w), which the reference forms
// again for every member with the same result). Static points keep theirs.
// True when a velocity is NaN.
__device__ __forceinline__ bool zone_member_motion(int p, const uint8_t* __restrict__ fixed,
                                                   const double4_32a* __restrict__ xo, double4_32a* av,
                                                   const double* x_cm, const double* v_cm, const double* w,
                                                   double mag_w, double sw, double cw, double dt,
                                                   const ZoneInverses& inv, const PassStamp& ps) {
    if (fixed[p] & 1) return false;
    stamp_point(ps, p);
    double xs[3], dx[3], xF[3], xR[3], wxR[3], tmpV[3], x_new[3], nv_[3];
    load3(xo, p, xs);
    for (int d = 0; d < 3; ++d) dx[d] = xs[d] - x_cm[d];
    if (mag_w < kRoundEps) {
        for (int d = 0; d < 3; ++d) { xF[d] = dx[d]; wxR[d] = 0.0; }
        for (int d = 0; d < 3; ++d) xR[d] = dx[d] - xF[d];
    } else {
        double sc = quotient(dot3(dx, w), inv.ww, inv.of_ww);
        for (int d = 0; d < 3; ++d) xF[d] = sc * w[d];
        for (int d = 0; d < 3; ++d) xR[d] = dx[d] - xF[d];
        for (int d = 0; d < 3; ++d) tmpV[d] = sw * w[d];
        cross3(tmpV, xR, wxR);
    }
    bool bad = false;
    for (int d = 0; d < 3; ++d) {
        x_new[d] = x_cm[d] + dt * v_cm[d] + xF[d] + cw * xR[d] + wxR[d];
        nv_[d] = quotient(x_new[d] - xs[d], dt, inv.of_dt);
        if (isnan(nv_[d])) bad = true;
    }
    av[p] = make_double4_32a(nv_[0], nv_[1], nv_[2], 0.0);
    return bad;
}

// Angular velocity of a zone from its angular momentum L and inertia I
// (Cramer's rule, dcollid3d.cpp:143-153).
__device__ __forceinline__ void zone_omega(const double (*I)[3], const double* L, double* w) {
    double tmp[3][3];
    const double det = det3(I), inv = 1.0 / det;
    for (int r = 0; r < 3; ++r) {
        for (int a = 0; a < 3; ++a)
            for (int b = 0; b < 3; ++b) tmp[a][b] = I[a][b];
        for (int s = 0; s < 3; ++s) tmp[s][r] = L[s];
        w[r] = det < kRoundEps ? 0.0 : quotient(det3(tmp), det, inv);
    }
}

// updateImpactListVelocity, dcollid3d.cpp:70-200, of one zone by one thread,
// over its members in the order of the reference's member list (which fixes
// the rounding of every sum); sin and cos correctly rounded, as the
// reference's libm gives them.
__device__ void zone_motion(const int* __restrict__ members, int i, int end, const uint8_t* __restrict__ fixed,
                            const double4_32a* __restrict__ xo, double4_32a* av, const int* __restrict__ vscene,
                            const SceneDev* __restrict__ scenes, PassCounters* ctr, const PassStamp& ps) {
    const SceneDev& sd = scenes[vscene[members[i]]];
    const double m = sd.p.m, dt = sd.p.dt;
    double x_cm[3] = {0.0, 0.0, 0.0}, v_cm[3] = {0.0, 0.0, 0.0};
    double L[3] = {0.0, 0.0, 0.0}, I[3][3] = {{0.0, 0.0, 0.0}, {0.0, 0.0, 0.0}, {0.0, 0.0, 0.0}}, tmp[3][3];
    int num_pts = end - i;
    for (int q = i; q < end; ++q) {
        int p = members[q];
        double xs[3], vs[3];
        load3(xo, p, xs);
        load3(av, p, vs);
        for (int d = 0; d < 3; ++d) { x_cm[d] += xs[d]; v_cm[d] += vs[d]; }
    }
    for (int d = 0; d < 3; ++d) { x_cm[d] /= num_pts; v_cm[d] /= num_pts; }
    for (int q = i; q < end; ++q) {
        int p = members[q];
        double xs[3], vs[3], dx[3], dv[3], Li[3];
        load3(xo, p, xs);
        load3(av, p, vs);
        for (int d = 0; d < 3; ++d) { dx[d] = xs[d] - x_cm[d]; dv[d] = vs[d] - v_cm[d]; }
        cross3(dx, dv, Li);
        for (int d = 0; d < 3; ++d) Li[d] = m * Li[d];
        for (int d = 0; d < 3; ++d) L[d] = Li[d] + L[d];
    }
    for (int q = i; q < end; ++q) {
        int p = members[q];
        double xs[3], dx[3];
        load3(xo, p, xs);
        for (int d = 0; d < 3; ++d) dx[d] = xs[d] - x_cm[d];
        double mag_dx = mag3(dx);
        for (int r = 0; r < 3; ++r)
            for (int s = 0; s < 3; ++s) {
                tmp[r][s] = -dx[r] * dx[s];
                if (r == s) tmp[r][s] += mag_dx * mag_dx;
                I[r][s] += tmp[r][s] * m;
            }
    }
    double w[3];
    zone_omega(I, L, w);
    double mag_w = mag3(w);
    double sn, cs;
    cr::sincos(dt * mag_w, &sn, &cs);
    const double sw = mag_w < kRoundEps ? 0.0 : sn / mag_w;
    const double cw = cs;
    const ZoneInverses inv = zone_inverses(w, sd.inv_dt);
    bool bad = false;
    for (int q = i; q < end; ++q)
        bad |= zone_member_motion(members[q], fixed, xo, av, x_cm, v_cm, w, mag_w, sw, cw, dt, inv, ps);
    if (bad) atomicOr(&ctr->err, kErrNan);
}

// Zones of at least this many members are solved one warp per zone where the
// zone list is built on the device; in a pass with at most `few` zones (a
// knob), every zone of two or more members is: one thread per zone keeps the
// FP64 pipe busiest when zones are many, one warp per zone gives the shortest
// chain when they are few. Zone solves of a step of 48 sheets in contact: no
// zone small enough for that 1.90 ms, up to 64 or 1,024 in a pass 1.75; zones
// of 16 / 32 / 64 / 128 members and more by a CTA 1.67 / 1.67 / 1.75 / 2.09,
// none 2.71 (256 sheets: 8.59 / 8.63 / 8.67 / 9.01, none 15.0).
constexpr int kZoneWarpMin = 16;
__device__ __forceinline__ int zone_warp_min(int nzones, int few) { return nzones <= few ? 2 : kZoneWarpMin; }
constexpr int kZoneSums = 9;  // summed components: L, then the six of I that differ
constexpr int kZoneWarps = 8, kZoneThreads = kZoneWarps * 32;
constexpr int kZoneCtas = 152;  // blocks of each role: with both, two per SM

// A member's terms of the sums after the centre of mass: m (dx x dv), and the
// upper triangle of m (|dx|^2 delta - dx dx) - the lower one is the same
// products with their factors swapped, so its sums are the same.
__device__ __forceinline__ void zone_terms(const double* xs, const double* vs, const double* x_cm, const double* v_cm,
                                           double m, double* t) {
    double dx[3], dv[3], Li[3];
    for (int d = 0; d < 3; ++d) { dx[d] = xs[d] - x_cm[d]; dv[d] = vs[d] - v_cm[d]; }
    cross3(dx, dv, Li);
    for (int d = 0; d < 3; ++d) t[d] = m * Li[d];
    const double mag_dx = mag3(dx);
    const double mag2 = mag_dx * mag_dx;
    int k = 3;
    for (int r = 0; r < 3; ++r)
        for (int q = r; q < 3; ++q) {
            double v = -dx[r] * dx[q];
            if (r == q) v += mag2;
            t[k++] = v * m;
        }
}
__device__ __forceinline__ void zone_inertia(const double* u, double (*I)[3]) {
    I[0][0] = u[0], I[0][1] = I[1][0] = u[1], I[0][2] = I[2][0] = u[2];
    I[1][1] = u[3], I[1][2] = I[2][1] = u[4], I[2][2] = u[5];
}

struct ZoneArgs {
    const int* members;
    const uint8_t* fixed;
    const double4_32a* xo;
    double4_32a* av;
    const int* vscene;
    const SceneDev* scenes;
    PassCounters* ctr;
    PassStamp ps;
};

// A zone of at least kZoneWarpMin members (or any, in a pass of few zones) by
// a warp. The sums of updateImpactListVelocity (centre of mass and velocity,
// angular momentum, inertia) must be formed member by member in list order to
// round as the reference's do, and GB300's FP64 pipe makes such a chain slow
// on one thread: here the lanes load 32 members at a time and form every
// per-member term in parallel, and a lane per component adds the staged terms
// in order - the same additions on the same operands as the one-thread form.
// The final per-member motion is spread over the lanes.
__device__ bool zone_by_warp(const ZoneArgs& z, int i, int end, double (*st)[kZoneSums]) {
    const int lane = threadIdx.x & 31;
    const SceneDev& sd = z.scenes[z.vscene[z.members[i]]];
    const double m = sd.p.m, dt = sd.p.dt;
    const int num_pts = end - i;
    double x_cm[3], v_cm[3], L[3], u[6], I[3][3];
    double acc = 0.0;  // this lane's component of the current sum
    for (int c = i; c < end; c += 32) {
        const int q = c + lane;
        if (q < end) {
            const int p = z.members[q];
            double xs[3], vs[3];
            load3(z.xo, p, xs);
            load3(z.av, p, vs);
            for (int d = 0; d < 3; ++d) st[lane][d] = xs[d], st[lane][3 + d] = vs[d];
        }
        __syncwarp();
        if (lane < 6) {  // lane d sums component d over the members in list order
            const int k1 = end - c < 32 ? end - c : 32;
            for (int k = 0; k < k1; ++k) acc += st[k][lane];
        }
        __syncwarp();
    }
    acc = acc / num_pts;
    for (int d = 0; d < 3; ++d) {
        x_cm[d] = __shfl_sync(0xffffffffu, acc, d);
        v_cm[d] = __shfl_sync(0xffffffffu, acc, 3 + d);
    }
    acc = 0.0;
    for (int c = i; c < end; c += 32) {
        const int q = c + lane;
        if (q < end) {
            const int p = z.members[q];
            double xs[3], vs[3];
            load3(z.xo, p, xs);
            load3(z.av, p, vs);
            zone_terms(xs, vs, x_cm, v_cm, m, st[lane]);
        }
        __syncwarp();
        if (lane < kZoneSums) {
            const int k1 = end - c < 32 ? end - c : 32;
            for (int k = 0; k < k1; ++k) acc = st[k][lane] + acc;
        }
        __syncwarp();
    }
    for (int d = 0; d < 3; ++d) L[d] = __shfl_sync(0xffffffffu, acc, d);
    for (int k = 0; k < 6; ++k) u[k] = __shfl_sync(0xffffffffu, acc, 3 + k);
    zone_inertia(u, I);
    // every lane forms the same rotation (sin and cos on two lanes)
    double w[3];
    zone_omega(I, L, w);
    const double mag_w = mag3(w);
    double sn, cs;
    cr::sincos_warp(dt * mag_w, &sn, &cs);
    const double sw = mag_w < kRoundEps ? 0.0 : sn / mag_w;
    const double cw = cs;
    const ZoneInverses inv = zone_inverses(w, sd.inv_dt);
    bool bad = false;
    for (int q = i + lane; q < end; q += 32)
        bad |= zone_member_motion(z.members[q], z.fixed, z.xo, z.av, x_cm, v_cm, w, mag_w, sw, cw, dt, inv, z.ps);
    __syncwarp();
    return bad;
}

// A large zone by a CTA: the same sums in the same order, a lane of warp 0 per
// component, but every member's terms and its final motion by all the CTA's
// threads. What bounds it is the 2 n additions in order (~64 cycles each on
// this FP64 pipe: 41 us of 640 members). A movable body of 642 points on one
// thread took 3 ms of every pass.
__device__ bool zone_by_cta(const ZoneArgs& z, int i, int end, double (*st)[kZoneSums]) {
    __shared__ double s_sum[kZoneSums];
    __shared__ double s_rot[6];  // w, mag_w, sw, cw
    const int tid = threadIdx.x;
    const SceneDev& sd = z.scenes[z.vscene[z.members[i]]];
    const double m = sd.p.m, dt = sd.p.dt;
    const int num_pts = end - i;
    double acc = 0.0;  // this thread's component of the current sum
    for (int c = i; c < end; c += kZoneThreads) {
        const int q = c + tid;
        if (q < end) {
            const int p = z.members[q];
            double xs[3], vs[3];
            load3(z.xo, p, xs);
            load3(z.av, p, vs);
            for (int d = 0; d < 3; ++d) st[tid][d] = xs[d], st[tid][3 + d] = vs[d];
        }
        __syncthreads();
        if (tid < 6) {
            const int k1 = end - c < kZoneThreads ? end - c : kZoneThreads;
            for (int k = 0; k < k1; ++k) acc += st[k][tid];
        }
        __syncthreads();
    }
    if (tid < 6) s_sum[tid] = acc / num_pts;
    __syncthreads();
    double x_cm[3], v_cm[3];
    for (int d = 0; d < 3; ++d) x_cm[d] = s_sum[d], v_cm[d] = s_sum[3 + d];
    acc = 0.0;
    for (int c = i; c < end; c += kZoneThreads) {
        const int q = c + tid;
        if (q < end) {
            const int p = z.members[q];
            double xs[3], vs[3];
            load3(z.xo, p, xs);
            load3(z.av, p, vs);
            zone_terms(xs, vs, x_cm, v_cm, m, st[tid]);
        }
        __syncthreads();
        if (tid < kZoneSums) {
            const int k1 = end - c < kZoneThreads ? end - c : kZoneThreads;
            for (int k = 0; k < k1; ++k) acc = st[k][tid] + acc;
        }
        __syncthreads();
    }
    if (tid < kZoneSums) s_sum[tid] = acc;
    __syncthreads();
    if (tid < 32) {  // warp 0: the same rotation in every lane, sin and cos on two lanes
        double L[3], u[6], I[3][3], w[3];
        for (int d = 0; d < 3; ++d) L[d] = s_sum[d];
        for (int k = 0; k < 6; ++k) u[k] = s_sum[3 + k];
        zone_inertia(u, I);
        zone_omega(I, L, w);
        const double mag_w = mag3(w);
        double sn, cs;
        cr::sincos_warp(dt * mag_w, &sn, &cs);
        if (tid == 0) {
            for (int d = 0; d < 3; ++d) s_rot[d] = w[d];
            s_rot[3] = mag_w;
            s_rot[4] = mag_w < kRoundEps ? 0.0 : sn / mag_w;
            s_rot[5] = cs;
        }
    }
    __syncthreads();
    const double w[3] = {s_rot[0], s_rot[1], s_rot[2]};
    const ZoneInverses inv = zone_inverses(w, sd.inv_dt);
    bool bad = false;
    for (int q = i + tid; q < end; q += kZoneThreads)
        bad |= zone_member_motion(z.members[q], z.fixed, z.xo, z.av, x_cm, v_cm, w, s_rot[3], s_rot[4], s_rot[5], dt,
                                  inv, z.ps);
    __syncthreads();  // the next zone reuses the shared arrays
    return bad;
}

// Every zone of a pass in one launch (zone z's members: zone_rng[z], their
// count *dnz, at most nzones): the first kZoneCtas blocks take the zones of at
// least cta_min members, the others the rest, a warp or a thread each.
__global__ void __launch_bounds__(kZoneThreads, 2) k_zone_solve(ZoneArgs z, ZoneMembers mem,
                                                                const int2* __restrict__ zone_rng, int nzones,
                                                                const int* __restrict__ dnz, int cta_min, int few) {
    __shared__ double st[kZoneThreads][kZoneSums];
    if (z.ctr->err & kErrRetry) return;
    z.members = mem.list();
    if (*dnz < nzones) nzones = *dnz;
    bool bad = false;
    if (blockIdx.x < kZoneCtas) {
        for (int k = blockIdx.x; k < nzones; k += kZoneCtas) {
            const int2 r = zone_rng[k];
            if (r.y - r.x >= cta_min) bad |= zone_by_cta(z, r.x, r.y, st);
        }
    } else {
        const int b = blockIdx.x - kZoneCtas, nb = gridDim.x - kZoneCtas;
        const int warp_min = zone_warp_min(nzones, few);
        const int wib = threadIdx.x >> 5;
        for (int k = b + nb * wib; k < nzones; k += nb * kZoneWarps) {
            const int2 r = zone_rng[k];
            if (r.y - r.x >= warp_min && r.y - r.x < cta_min) bad |= zone_by_warp(z, r.x, r.y, st + 32 * wib);
        }
        if (warp_min > 2)
            for (int k = b + nb * (int)threadIdx.x; k < nzones; k += nb * kZoneThreads) {
                const int2 r = zone_rng[k];
                if (r.y - r.x < warp_min)
                    zone_motion(z.members, r.x, r.y, z.fixed, z.xo, z.av, z.vscene, z.scenes, z.ctr, z.ps);
            }
    }
    if (bad) atomicOr(&z.ctr->err, kErrNan);
}

// The movable bodies (updateImpactZoneVelocityForRG, dcollid.cpp:267-288,
// called from updateAverageVelocity when dt > 0), zone_off their members: only
// those of scenes in a pass (run), and of more than one point, move.
__global__ void __launch_bounds__(kZoneThreads, 2) k_body_solve(ZoneArgs z, const int* __restrict__ zone_off,
                                                                int nzones, const SceneRun* __restrict__ run) {
    __shared__ double st[kZoneThreads][kZoneSums];
    if (z.ctr->err & kErrRetry) return;
    bool bad = false;
    for (int k = blockIdx.x; k < nzones; k += gridDim.x) {
        const int i = zone_off[k], end = zone_off[k + 1];
        if (end - i < 2) continue;
        if (run) {
            const int zs = z.vscene[z.members[i]];
            if (run[zs].mode == kSceneIdle || !(z.scenes[zs].p.dt > 0.0)) continue;
        }
        bad |= zone_by_cta(z, i, end, st);
    }
    if (bad) atomicOr(&z.ctr->err, kErrNan);
}

// detectDomainBoundaryCollision (dcollid.cpp:116-158) then
// updateFinalPosition (dcollid.cpp:562-584) for one point. The reference
// revisits points shared by several elements; the clamp is idempotent, so
// once per point gives the same result.
__global__ void k_finalize(const uint8_t* __restrict__ in_elem, const double4_32a* __restrict__ xo, double4_32a* av,
                           uint8_t* has_collsn, const double* __restrict__ x_cand, double* x_out, int nv,
                           const int* __restrict__ vscene, const SceneDev* __restrict__ scenes,
                           const uint8_t* __restrict__ fixed, const uint8_t* __restrict__ mask) {
    int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= nv) return;
    if (mask && !mask[vscene[p]]) return;  // another scene set's end of step
    if (!in_elem[p]) {
        for (int j = 0; j < 3; ++j) x_out[3 * p + j] = x_cand[3 * p + j];
        return;
    }
    const SceneDev& sd = scenes[vscene[p]];
    if (!sd.enabled) {
        for (int j = 0; j < 3; ++j) x_out[3 * p + j] = x_cand[3 * p + j];
        return;
    }
    const Params prm = sd.p;
    double L[3] = {sd.lo[0], sd.lo[1], sd.lo[2]}, U[3] = {sd.hi[0], sd.hi[1], sd.hi[2]};
    double xs[3], v[3];
    load3(xo, p, xs);
    load3(av, p, v);
    double dt = prm.dt, mu = prm.lambda, dv = 0;
    if (fixed[p] & 2) {  // movable points skip the clamp (dcollid.cpp:123)
        for (int j = 0; j < 3; ++j) x_out[3 * p + j] = xs[j] + v[j] * dt;
        return;
    }
    double cand[3];
    bool clamped = false;
    for (int j = 0; j < 3; ++j) {
        cand[j] = xs[j] + dt * v[j];
        if (cand[j] <= L[j] || cand[j] >= U[j]) {
            has_collsn[p] = 1;
            clamped = true;
            dv = fabs(v[j]);
            v[j] = 0.0;
        }
    }
    if (!clamped && (((unsigned)__double2hiint(mu) >> 20) & 0x7ffu) != 0x7ffu) {
        // dv = 0: the friction factor is 1, the position the candidate
        for (int j = 0; j < 3; ++j) x_out[3 * p + j] = cand[j];
        return;
    }
    double preVt = mag3(v);
    if (preVt > kMachEps)
        for (int j = 0; j < 3; ++j) v[j] *= smax(1.0 - mu * dv / preVt, 0.0);
    av[p] = make_double4_32a(v[0], v[1], v[2], 0.0);
    for (int j = 0; j < 3; ++j) x_out[3 * p + j] = xs[j] + v[j] * dt;
}

__global__ void k_final_velocity(const uint8_t* __restrict__ in_elem, const uint8_t* __restrict__ has_collsn,
                                 const double4_32a* __restrict__ av, const int* __restrict__ vscene,
                                 const SceneDev* __restrict__ scenes, double* vel, int nv,
                                 const uint8_t* __restrict__ mask) {
    int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= nv || !in_elem[p] || !has_collsn[p] || !scenes[vscene[p]].enabled) return;
    if (mask && !mask[vscene[p]]) return;
    double4_32a a = av[p];
    vel[3 * p] = a.x;
    vel[3 * p + 1] = a.y;
    vel[3 * p + 2] = a.z;
}

__global__ void k_math_selftest(int fn, const double* a, const double* b, double* out, int n) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double r;
    switch (fn) {
        case 0: r = cr::cos(a[i]); break;
        case 1: r = cr::sin(a[i]); break;
        case 2: r = cr::acos(a[i]); break;
        default: r = cr::pow(a[i], b[i]); break;
    }
    out[i] = r;
}

// updateFinalForRG, dcollid.cpp:626-675: the first point of each body, in
// element order, that has has_collsn (its index, -1 for none) and its final
// average velocity.
__global__ void k_final_rg(const int* __restrict__ visit, const int* __restrict__ visit_off, int nbodies,
                           const uint8_t* __restrict__ has_collsn, const double4_32a* __restrict__ av,
                           double4_32a* out) {
    int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= nbodies) return;
    double4_32a r = make_double4_32a(0.0, 0.0, 0.0, -1.0);
    for (int i = visit_off[b]; i < visit_off[b + 1]; ++i) {
        const int p = visit[i];
        if (has_collsn[p]) {
            const double4_32a a = av[p];
            r = make_double4_32a(a.x, a.y, a.z, (double)p);
            break;
        }
    }
    out[b] = r;
}

}  // namespace

void math_selftest(int fn, const double* a, const double* b, double* out, int n, cudaStream_t s) {
    if (n > 0) count_launch(), k_math_selftest<<<nblk(n, 128), 128, 0, s>>>(fn, a, b, out, n);
}

void step_init(const double* x_old, const double* x_cand, int nv, const uint8_t* in_elem, const int* vscene,
               const SceneDev* scenes, double4_32a* xo, double4_32a* av, PassCounters* ctr, cudaStream_t s) {
    if (nv > 0)
        count_launch(), k_step_init<<<nblk(nv, 256), 256, 0, s>>>(x_old, x_cand, nv, in_elem, vscene, scenes, xo, av,
                                                                  ctr);
}

void apply_contribs(const Contrib* contrib, const PassCounters* ctr, int contrib_cap, int nv, double4_32a* av,
                    uint8_t* has_collsn, ApplyBufs& b, cudaStream_t s, double4_32a* dump, const BodyBufs* bodies) {
    if (dump && nv > 0) cudaMemsetAsync(dump, 0, sizeof(double4_32a) * (size_t)nv, s);
    if (nv <= 0) return;
    const int nb = bodies ? bodies->n : 0, nslot = nv + nb;
    if (nb > 0) cudaMemsetAsync(bodies->num, 0, sizeof(int) * (size_t)nb, s);
    int blocks = nblk(contrib_cap, 256);
    if (blocks > 152 * 8) blocks = 152 * 8;
    PassCounters* c = const_cast<PassCounters*>(ctr);
    count_launch(), k_contrib_count<<<blocks, 256, 0, s>>>(contrib, c, contrib_cap, b.cnt, b.touched);
    const int sblocks = nblk(nslot, 256) < 152 * 8 ? nblk(nslot, 256) : 152 * 8;
    count_launch(), k_contrib_segments<<<sblocks, 256, 0, s>>>(c, b.cnt, b.touched, b.off);
    count_launch(), k_contrib_scatter<<<blocks, 256, 0, s>>>(contrib, ctr, contrib_cap, b.off, b.cur, b.idx);
    const int ablocks = nblk(nslot, kApplyWarps) < 152 * 8 ? nblk(nslot, kApplyWarps) : 152 * 8;
    count_launch(), k_apply<<<ablocks, kApplyWarps * 32, 0, s>>>(contrib, c, b.cnt, b.cur, b.off, b.touched, b.idx,
                                                                 b.ord, nv, av, has_collsn, dump,
                                                                 nb ? bodies->acc : nullptr, nb ? bodies->num : nullptr,
                                                                 b.ps);
    if (nb > 0)
        count_launch(), k_apply_rg<<<nblk(bodies->nmembers, 128), 128, 0, s>>>(
            bodies->members, bodies->member_body, bodies->nmembers, ctr, bodies->acc, bodies->num, bodies->fixed, av,
            has_collsn, b.ps);
}

void zone_solve(const int* members, const int* zone_off, int nzones, const uint8_t* fixed, const double4_32a* xo,
                double4_32a* av, const int* vscene, const SceneDev* scenes, PassCounters* ctr, cudaStream_t s,
                const SceneRun* run, PassStamp ps) {
    // (a body of one point does not move)
    if (nzones > 0)
        count_launch(), k_body_solve<<<nzones < 152 * 8 ? nzones : 152 * 8, kZoneThreads, 0, s>>>(
            ZoneArgs{members, fixed, xo, av, vscene, scenes, ctr, ps}, zone_off, nzones, run);
}

void zone_solve_dev(const ZoneMembers& members, const int2* zone_rng, const int* dnz, int zone_cap, const uint8_t* fixed,
                    const double4_32a* xo, double4_32a* av, const int* vscene, const SceneDev* scenes,
                    PassCounters* ctr, cudaStream_t s, PassStamp ps, int cta_min, int few) {
    if (cta_min < kZoneWarpMin) cta_min = kZoneWarpMin;
    if (zone_cap > 0)
        count_launch(), k_zone_solve<<<2 * kZoneCtas, kZoneThreads, 0, s>>>(
            ZoneArgs{nullptr, fixed, xo, av, vscene, scenes, ctr, ps}, members, zone_rng, zone_cap, dnz, cta_min, few);
}

void final_rigid(const BodyBufs& b, const uint8_t* has_collsn, const double4_32a* av, cudaStream_t s) {
    if (b.n > 0)
        count_launch(), k_final_rg<<<nblk(b.n, 128), 128, 0, s>>>(b.visit, b.visit_off, b.n, has_collsn, av, b.out);
}

void finalize_positions(const uint8_t* in_elem, const double4_32a* xo, double4_32a* av, uint8_t* has_collsn,
                        const double* x_cand, double* x_out, int nv, const int* vscene, const SceneDev* scenes,
                        const uint8_t* fixed, const uint8_t* mask, cudaStream_t s) {
    if (nv > 0)
        count_launch(), k_finalize<<<nblk(nv, 256), 256, 0, s>>>(in_elem, xo, av, has_collsn, x_cand, x_out, nv,
                                                                 vscene, scenes, fixed, mask);
}

void final_velocity(const uint8_t* in_elem, const uint8_t* has_collsn, const double4_32a* av, const int* vscene,
                    const SceneDev* scenes, double* vel, int nv, const uint8_t* mask, cudaStream_t s) {
    if (nv > 0)
        count_launch(), k_final_velocity<<<nblk(nv, 256), 256, 0, s>>>(in_elem, has_collsn, av, vscene, scenes, vel,
                                                                       nv, mask);
}

}  // namespace ccg
