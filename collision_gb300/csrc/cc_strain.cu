// Strain limiting: reduceSuperelast, up to 10 Gauss-Seidel passes over a
// scene's edges (dcollid.cpp:486-560, 586-596), and the records they read.
//
// The reference sweeps the edges one after the other. Here an element's
// edges are taken by one thread in their order, and elements that share no
// point run side by side: an element's level is one more than the level of
// the last earlier element at any of its points, so a level sees exactly
// the values the sequential sweep gives it. The sweeps themselves are
// pipelined: sweep k + 1 follows sweep k through the mesh, a few levels
// behind (k_strain_sweeps).
#include "cc_launch.h"
#include "cc_narrow.cuh"

namespace ccg {

namespace {

inline int nblk(int n, int t) { return (n + t - 1) / t; }

// Squared-length bounds that decide |(sqrt(s) - L)/L| > 0.1 without the
// square root and the division: outside [lo_no, hi_no] the answer is "over",
// inside [lo_def, hi_def] ... see strain_quick. The bounds sit 1e-9 (relative)
// inside and outside the exact thresholds L*(1 -+ 0.1); the reference's own
// rounding of sqrt, subtraction and division is below 1e-15, so a decision
// taken here equals the reference's.
struct StrainBounds {
    double hi_def, hi_no, lo_no, lo_def;
};
__device__ __forceinline__ StrainBounds strain_bounds(double L) {
    StrainBounds b;
    double a = L * (1.1 * (1.0 + 1e-9)), c = L * (1.1 * (1.0 - 1e-9));
    double d = L * (0.9 * (1.0 + 1e-9)), e = L * (0.9 * (1.0 - 1e-9));
    b.hi_def = a * a;  // s above: over-stretched for sure
    b.hi_no = c * c;   // s below (and above lo_no): not over-stretched
    b.lo_no = d * d;
    b.lo_def = e * e;  // s below: over-compressed for sure
    return b;
}
// The same bounds from the squared length L2 = L*L, without the square root:
// each differs from the one above by a few ulps, far inside the 1e-9 margin.
__device__ __forceinline__ StrainBounds strain_bounds_sq(double L2) {
    const double ka = (1.1 * (1.0 + 1e-9)) * (1.1 * (1.0 + 1e-9)), kc = (1.1 * (1.0 - 1e-9)) * (1.1 * (1.0 - 1e-9));
    const double kd = (0.9 * (1.0 + 1e-9)) * (0.9 * (1.0 + 1e-9)), ke = (0.9 * (1.0 - 1e-9)) * (0.9 * (1.0 - 1e-9));
    StrainBounds b;
    b.hi_def = L2 * ka;
    b.hi_no = L2 * kc;
    b.lo_no = L2 * kd;
    b.lo_def = L2 * ke;
    return b;
}
// 1: over the limit, 0: within it, -1: too close to tell without the exact test.
__device__ __forceinline__ int strain_quick(double s, const StrainBounds& b) {
    if (s > b.hi_def || s < b.lo_def) return 1;
    if (s < b.hi_no && s > b.lo_no) return 0;
    return -1;
}

struct __align__(16) StrainEdgeStep {
    int p0, p1;
    double len0;
    StrainBounds rest;  // from the rest length
    StrainBounds prev;  // from the start-of-step length (strain rate)
    double x0[3], x1[3];  // x_old of both points (constant through the sweep)
    int exact_only;       // degenerate lengths: always take the exact test
    int pad[3];
};

// An edge's full record for the step, from its endpoints' x_old.
__device__ __forceinline__ StrainEdgeStep strain_step(int p0, int p1, double len0,
                                                      const double4_32a* __restrict__ xo) {
    double x0[3], x1[3];
    load3(xo, p0, x0);
    load3(xo, p1, x1);
    double so = 0.0;
    for (int k = 0; k < 3; ++k) so += sqr(x0[k] - x1[k]);
    StrainEdgeStep r;
    r.p0 = p0;
    r.p1 = p1;
    r.len0 = len0;
    r.rest = strain_bounds(len0);
    r.prev = strain_bounds_sq(so);
    for (int k = 0; k < 3; ++k) {
        r.x0[k] = x0[k];
        r.x1[k] = x1[k];
    }
    // tiny or non-positive lengths: leave every decision to the exact test
    r.exact_only = !(so > 1e-12 && len0 > 1e-6);
    return r;
}

// Per step: every edge's record of k_strain.
__global__ void k_edge_setup(const StrainEdge* __restrict__ edges, int m, const double4_32a* __restrict__ xo,
                             StrainEdgeStep* out) {
    int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e < m) out[e] = strain_step(edges[e].p0, edges[e].p1, edges[e].len0, xo);
}

// The strain decision for given end velocities v0, v1 (bounds first, the
// exact test of dcollid.cpp:525-530 only inside the bounds' margin).
__device__ __forceinline__ bool strain_flag_vals(const StrainEdgeStep& ed, const double* v0, const double* v1,
                                                 double dt, int* n_exact) {
    double c0[3], c1[3];
    for (int k = 0; k < 3; ++k) {
        c0[k] = ed.x0[k] + dt * v0[k];
        c1[k] = ed.x1[k] + dt * v1[k];
    }
    double sn = 0.0;
    for (int k = 0; k < 3; ++k) sn += sqr(c0[k] - c1[k]);
    if (!ed.exact_only && sn > 1e-18) {
        int q0 = strain_quick(sn, ed.rest), q1 = strain_quick(sn, ed.prev);
        if (q0 == 1 || q1 == 1) return true;
        if (q0 == 0 && q1 == 0) return false;
    }
    ++*n_exact;
    double so = 0.0;
    for (int k = 0; k < 3; ++k) so += sqr(ed.x0[k] - ed.x1[k]);
    double len_new = sqrt(sn), len_old = sqrt(so);
    if (len_old > kRoundEps && len_new > kRoundEps) {
        double strain_rate = (len_new - len_old) / len_old;
        double strain = (len_new - ed.len0) / ed.len0;
        return fabs(strain) > kStrainTol || fabs(strain_rate) > kStrainTol;
    }
    return true;
}

// 0.5 * x, the averaging of the strain sweep: one less in the exponent field
// (in the high 32 bits) when that field is 2..2046, where the halving is
// exact; x itself for +-0; the FP64 multiply otherwise. GB300 issues a
// warp's FP64 multiply in ~64 cycles whatever its active lanes, and the
// averaging lies on the sweep's per-level critical path; these are a few
// 32-bit integer instructions with the same result.
__device__ __forceinline__ double half_of(double x) {
    const int hi = __double2hiint(x), lo = __double2loint(x);
    const unsigned e = ((unsigned)hi >> 20) & 0x7ffu;
    if (e - 2u < 0x7fdu) return __hiloint2double(hi - 0x00100000, lo);
    if ((((unsigned)hi << 1) | (unsigned)lo) == 0u) return x;
    return 0.5 * x;
}

// Per scene and step, flags[2s] ("some edge would average": set by
// k_sweep_check) and flags[2s+1] (the strain loop is over); passes_out[3s ..]
// the sweeps run, edges averaged, exact tests. k_strain runs one pass per
// launch: a scene whose check found nothing to average is done - its sweep
// would change nothing, which is how the reference's loop ends
// (dcollid.cpp:588-595) - and counts that sweep; otherwise it sweeps once.
__device__ __forceinline__ bool sweep_gate(int pass, int s, int* flags, int* passes_out_all) {
    __shared__ int s_go;
    if (threadIdx.x == 0) {
        int go = 0;
        if (!flags[2 * s + 1]) {
            if (!flags[2 * s]) {
                flags[2 * s + 1] = 1;
                passes_out_all[3 * s] = pass + 1;
            } else {
                flags[2 * s] = 0;
                go = 1;
            }
        }
        s_go = go;
    }
    __syncthreads();
    return s_go != 0;
}

__device__ __forceinline__ void sweep_done(int pass, int s, int n_avg, int n_exact, int* flags, int* passes_out_all) {
    __shared__ int s_avg, s_exact;
    if (threadIdx.x == 0) s_avg = s_exact = 0;
    __syncthreads();
    atomicAdd(&s_avg, n_avg);
    atomicAdd(&s_exact, n_exact);
    __syncthreads();
    if (threadIdx.x == 0) {
        passes_out_all[3 * s] = pass + 1;
        passes_out_all[3 * s + 1] += s_avg;
        passes_out_all[3 * s + 2] += s_exact;
        if (pass + 1 >= kStrainMaxIter) flags[2 * s + 1] = 1;
    }
}

// The sweep on global memory, one CTA per scene and pass, every decision in
// FP64, the edges sorted by their own dependency levels (cc_strain_plan.h).
__global__ void __launch_bounds__(256) k_strain(const StrainEdgeStep* __restrict__ edges,
                                                const int4* __restrict__ hdr_all,
                                                const SceneDev* __restrict__ scenes, int window,
                                                double4_32a* av, int pass, int* flags, int* passes_out_all,
                                                const int* __restrict__ order) {
    const int sc = order[blockIdx.x];
    const SceneDev& sd = scenes[sc];
    if ((window && sd.sw_fits) || !sd.enabled) return;  // k_strain_sweeps', or left out
    if (!sweep_gate(pass, sc, flags, passes_out_all)) return;
    const int4* hdr = hdr_all + 2 * sd.strain_hdr0;
    const int nlevels = sd.strain_levels;
    const double dt = sd.p.dt;
    int n_avg = 0, n_exact = 0;
    // the records of the next level are loaded before the barrier that ends
    // the current one: they do not depend on the velocities
    int e = 0, e1 = 0;
    if (nlevels > 0) {
        int4 h = hdr[0];
        e = h.x + threadIdx.x;
        e1 = h.y;
    }
    StrainEdgeStep cur;
    bool have = e < e1;
    if (have) cur = edges[e];
    for (int l = 0; l < nlevels; ++l) {
        int ne = 0, ne1 = 0;
        if (l + 1 < nlevels) {
            int4 h = hdr[2 * (l + 1)];
            ne = h.x + threadIdx.x;
            ne1 = h.y;
        }
        bool nhave = ne < ne1;
        StrainEdgeStep nxt;
        if (nhave) nxt = edges[ne];
        while (have) {
            double4_32a a0 = av[cur.p0], a1 = av[cur.p1];
            double v0[3] = {a0.x, a0.y, a0.z}, v1[3] = {a1.x, a1.y, a1.z};
            if (strain_flag_vals(cur, v0, v1, dt, &n_exact)) {
                ++n_avg;
                double t0 = a0.x + a1.x, t1 = a0.y + a1.y, t2 = a0.z + a1.z;
                t0 = half_of(t0); t1 = half_of(t1); t2 = half_of(t2);
                double4_32a nv4 = make_double4_32a(t0, t1, t2, 0.0);
                av[cur.p0] = nv4;
                av[cur.p1] = nv4;
            }
            e += blockDim.x;
            have = e < e1;
            if (have) cur = edges[e];
        }
        __syncthreads();
        e = ne;
        e1 = ne1;
        have = nhave;
        cur = nxt;
    }
    sweep_done(pass, sc, n_avg, n_exact, flags, passes_out_all);
}

// ------------------------------------------------ sweeps in shared memory

// An element's record for the step: per edge x_old(pi) - x_old(pj) and the
// sum of that vector's magnitudes, the squared lengths above which (x) and
// below which (y) the edge is over the strain limit, all in FP32, and its
// points' slots. A degenerate edge has NaN bounds: every decision on it is
// the exact test's. 80 bytes: the loads of a warp's eight elements (four
// lanes each) meet no bank conflict.
struct __align__(16) SweepRec {
    float4 dx[3];
    float2 limit[3];
    unsigned s01, s2n;
};
static_assert(sizeof(SweepRec) == kSweepRecBytes, "record size");

// A point's slot: its FP64 velocity, and the same in FP32 with the sum of
// the magnitudes. Lane c of an element's four reads d[c] and f[c].
struct __align__(16) SweepSlot {
    double d[4];
    float f[4];
};
static_assert(sizeof(SweepSlot) == kSweepSlotBytes, "slot size");

__device__ __forceinline__ float4 cut32x3(double x, double y, double z) {
    const float fx = cut32(x), fy = cut32(y), fz = cut32(z);
    return make_float4(fx, fy, fz, fabsf(fx) + fabsf(fy) + fabsf(fz));
}

// The strain decision of one edge in FP32: 1 over the limit, 0 within it, -1
// too close to tell. With u = 2^-24 and b the sum over the components of
// |dx| + dt (|v0| + |v1|), the inputs' roundings (velocities and dx 2u, dt
// 2u) and the operations' put each component of dx + dt (v0 - v1) within
// 8 u b_k and s within 21 u b^2 of its exact value; the margin is 40 u b^2,
// whose remaining 19 u b^2 > 15 u s covers the rounding of the margin and of
// its sum with s (2 u), and the bounds' own: 10 u (lengths cut 2u, squared,
// summed and scaled), and the 1e-9 beyond the exact threshold that a decision
// has to keep (the exact test rounds by less than 1e-15).
constexpr float kSweepMargin = 40.0f * 5.9604645e-8f;
__device__ __forceinline__ int sweep_decide(float s, float b, float2 limit) {
    const float err = b * b * kSweepMargin;
    const float s0 = s - err, s1 = s + err;
    if (s0 > limit.x || s1 < limit.y) return 1;
    if (s1 < limit.x && s0 > limit.y) return 0;
    return -1;
}
// On whole vectors, one thread.
__device__ __forceinline__ int sweep_decide(const SweepRec& r, int j, float4 f0, float4 f1, float dt32) {
    const float4 d = r.dx[j];
    const float ux = fmaf(dt32, f0.x - f1.x, d.x), uy = fmaf(dt32, f0.y - f1.y, d.y),
                uz = fmaf(dt32, f0.z - f1.z, d.z);
    return sweep_decide((ux * ux + uy * uy) + uz * uz, fmaf(dt32, f0.w + f1.w, d.w), r.limit[j]);
}
// On four lanes (sign: -1, -1, -1, 1): lane c < 3 forms component c of
// dx + dt (v0 - v1), lane 3 the sum b. The same result in all four.
__device__ __forceinline__ int sweep_decide4(float d, float f0, float f1, float sign, float2 limit, float dt32) {
    const float u = fmaf(dt32, fmaf(sign, f1, f0), d);
    float q = sign < 0.f ? u * u : 0.f;
    q += __shfl_xor_sync(0xffffffffu, q, 1);
    q += __shfl_xor_sync(0xffffffffu, q, 2);
    return sweep_decide(q, __shfl_sync(0xffffffffu, u, 3, 4), limit);
}

// The FP64 decision where FP32 cannot tell (rare: out of line).
__device__ __noinline__ bool sweep_exact(int p0, int p1, double len0, const double4_32a* __restrict__ xo, double ax,
                                         double ay, double az, double bx, double by, double bz, double dt) {
    const double v0[3] = {ax, ay, az}, v1[3] = {bx, by, bz};
    int n = 0;
    return strain_flag_vals(strain_step(p0, p1, len0, xo), v0, v1, dt, &n);
}

// Per step: every element's record. Only the differences are formed in FP64:
// 1,420,000 elements 162 -> 41 us.
__global__ void k_sweep_setup(const SweepElem* __restrict__ elems, int m, const double4_32a* __restrict__ xo,
                              SweepRec* __restrict__ out) {
    int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= m) return;
    const SweepElem el = elems[e];
    double x[3][3];
    for (int k = 0; k < 3; ++k) load3(xo, el.p[k], x[k]);
    SweepRec r;
    r.s01 = el.s01;
    r.s2n = el.s2n;
    for (int j = 0; j < 3; ++j) {
        const double *a = x[j], *b = x[(j + 1) % 3];
        const float dx = cut32(a[0] - b[0]), dy = cut32(a[1] - b[1]), dz = cut32(a[2] - b[2]);
        r.dx[j] = make_float4(dx, dy, dz, fabsf(dx) + fabsf(dy) + fabsf(dz));
        // over the limit above 1.1 times the shorter, below 0.9 times the
        // longer of the rest and the start-of-step length
        const float so = dx * dx + dy * dy + dz * dz, L = cut32(el.len0[j]), l2 = L * L;
        const bool degenerate = !(so > 1e-12f && L > 1e-6f);
        r.limit[j].x = degenerate ? __int_as_float(0x7fffffff) : 1.21f * fminf(l2, so);
        r.limit[j].y = degenerate ? __int_as_float(0x7fffffff) : 0.81f * fmaxf(l2, so);
    }
    out[e] = r;
}

// Would any edge average on the current velocities? (A block per chunk of at
// most 256 elements of one scene, the grid striding over the chunks; chunks
// of finished scenes, of scenes swept the other way than `which`, or of
// scenes where an averaging edge is already found, are skipped.) If none of
// a scene's edges would, its sweep changes nothing: before the first edge
// that averages every edge sees the start-of-pass velocities.
// which: 0 every scene, 1 only those that k_strain sweeps.
__global__ void __launch_bounds__(256) k_sweep_check(const SweepElem* __restrict__ elems,
                                                     const SweepRec* __restrict__ recs,
                                                     const double4_32a* __restrict__ xo,
                                                     const int2* __restrict__ chunks, int nchunks,
                                                     const SceneDev* __restrict__ scenes,
                                                     const double4_32a* __restrict__ av, int window, int which,
                                                     int* flags) {
    for (int c = blockIdx.x; c < nchunks; c += gridDim.x) {
        const int2 ch = chunks[c];  // (scene, first element)
        const SceneDev& sd = scenes[ch.x];
        if (!sd.enabled || flags[2 * ch.x + 1] || *(volatile int*)&flags[2 * ch.x]) continue;
        if (which == 1 && window && sd.sw_fits) continue;
        const int e = ch.y + threadIdx.x;
        if (e >= sd.sw_e0 + sd.sw_ne) continue;
        const SweepRec r = recs[e];
        const SweepElem el = elems[e];
        const double dt = sd.p.dt;
        const float dt32 = (float)dt;
        double v[3][3];
        float4 f[3];
        for (int k = 0; k < 3; ++k) {
            load3(av, el.p[k], v[k]);
            f[k] = cut32x3(v[k][0], v[k][1], v[k][2]);
        }
        const int ne = (int)(r.s2n >> 16);
        bool over = false;
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            if (j >= ne || over) continue;
            const int b = (j + 1) % 3;
            const int q = sweep_decide(r, j, f[j], f[b], dt32);
            over = q > 0 || (q < 0 && sweep_exact(el.p[j], el.p[b], el.len0[j], xo, v[j][0], v[j][1], v[j][2],
                                                  v[b][0], v[b][1], v[b][2], dt));
        }
        if (over && !flags[2 * ch.x]) atomicOr(&flags[2 * ch.x], 1);
    }
}

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
    unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}
// Named barriers of n threads (whole warps; bar takes a converged warp).
__device__ __forceinline__ void bar_sync(int id, int n) {
    __syncwarp();
    asm volatile("bar.sync %0, %1;\n" ::"r"(id), "r"(n) : "memory");
}
__device__ __forceinline__ int ld_acquire(const int* p) {
    int v;
    asm volatile("ld.acquire.gpu.global.b32 %0, [%1];\n" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_relaxed(int* p, int v) {
    asm volatile("st.relaxed.gpu.global.b32 [%0], %1;\n" ::"l"(p), "r"(v) : "memory");
}
// Flags between the warps of a block, in shared memory.
__device__ __forceinline__ int flag_load(const int* p) {
    int v;
    asm volatile("ld.acquire.cta.shared.b32 %0, [%1];\n"
                 : "=r"(v)
                 : "r"((unsigned)__cvta_generic_to_shared(p))
                 : "memory");
    return v;
}
__device__ __forceinline__ void flag_store(int* p, int v) {
    asm volatile("st.release.cta.shared.b32 [%0], %1;\n" ::"r"((unsigned)__cvta_generic_to_shared(p)), "r"(v)
                 : "memory");
}
__device__ __forceinline__ void flag_add(int* p, int v) {
    asm volatile("red.release.cta.shared.add.s32 [%0], %1;\n" ::"r"((unsigned)__cvta_generic_to_shared(p)), "r"(v)
                 : "memory");
}

// An element's record as one of its four lanes holds it.
struct SweepLane {
    float d[3];
    float2 limit[3];
    unsigned s01, s2n;
};

// One element per four lanes (lane c of them: component c; the last: the
// sums), the whole warp in step: its edges' decisions in FP32 side by side;
// only if one may be over the limit, the edges in turn on the FP64
// velocities, each averaging before the next is decided. An FP64 sum takes
// a warp ~64 cycles on this GPU however many lanes it serves, so a lane per
// component makes an average one instruction instead of three; a warp's
// eight elements share it. Lanes without an element (have false) hold
// slots of element 0 of the level and change nothing.
__device__ __forceinline__ void sweep_element(const SweepLane& r, bool have, const SweepElem* __restrict__ el,
                                              const double4_32a* __restrict__ xo, SweepSlot* win, int c, float sign,
                                              float dt32, double dt, int* n_avg, int* n_exact) {
    SweepSlot* w[3] = {&win[r.s01 & 0xffffu], &win[r.s01 >> 16], &win[r.s2n & 0xffffu]};
    const int ne = have ? (int)(r.s2n >> 16) : 0;
    float f[3] = {w[0]->f[c], w[1]->f[c], w[2]->f[c]};
    int q[3];
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        q[j] = sweep_decide4(r.d[j], f[j], f[(j + 1) % 3], sign, r.limit[j], dt32);
        if (j >= ne) q[j] = 0;
    }
    if (!__any_sync(0xffffffffu, q[0] | q[1] | q[2])) return;
    double v[3] = {w[0]->d[c], w[1]->d[c], w[2]->d[c]};
    unsigned changed = 0;
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        const int b = (j + 1) % 3;
        int d = q[j];
        if (j > 0) {  // (every lane takes part in the shuffles)
            d = sweep_decide4(r.d[j], f[j], f[b], sign, r.limit[j], dt32);
            if (j >= ne) d = 0;
        }
        if (__any_sync(0xffffffffu, d < 0)) {
            double a3[3], b3[3];
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                a3[k] = __shfl_sync(0xffffffffu, v[j], k, 4);
                b3[k] = __shfl_sync(0xffffffffu, v[b], k, 4);
            }
            if (d < 0) {
                *n_exact += c == 0;
                d = sweep_exact(el->p[j], el->p[b], el->len0[j], xo, a3[0], a3[1], a3[2], b3[0], b3[1], b3[2], dt);
            }
            __syncwarp();
        }
        if (__any_sync(0xffffffffu, d > 0)) {
            // half_of and cut32 of the sum, without a branch where it is in
            // the ordinary range (FP32's normal range after the halving lies
            // inside half_of's) or zero
            const double sum = v[j] + v[b];
            const unsigned hi = (unsigned)__double2hiint(sum), lo = (unsigned)__double2loint(sum);
            const bool zero = ((hi << 1) | lo) == 0u;
            const unsigned h = zero ? hi : hi - 0x00100000u;
            const unsigned m = (h & 0x7fffffffu) - 0x38000000u;
            double avg = __hiloint2double((int)h, (int)lo);
            float g = __uint_as_float(zero ? hi : (h & 0x80000000u) | __funnelshift_l(lo, m, 3));
            if (!zero && m - 0x00100000u >= 0x0fe00000u) {
                avg = half_of(sum);
                g = cut32(avg);
            }
            __syncwarp();
            float mag = sign < 0.f ? fabsf(g) : 0.f;
            mag += __shfl_xor_sync(0xffffffffu, mag, 1);
            mag += __shfl_xor_sync(0xffffffffu, mag, 2);
            if (sign > 0.f) g = mag;
            if (d > 0) {
                v[j] = v[b] = avg;
                f[j] = f[b] = g;
                changed |= (1u << j) | (1u << b);
                *n_avg += c == 0;
            }
        }
    }
#pragma unroll
    for (int j = 0; j < 3; ++j)
        if (changed >> j & 1u) {
            w[j]->d[c] = v[j];
            w[j]->f[c] = f[j];
        }
}

// mbarriers of the record ring, in shared memory
__device__ __forceinline__ void mbar_init(unsigned long long* b, int n) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"((unsigned)__cvta_generic_to_shared(b)), "r"(n)
                 : "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned long long* b) {
    asm volatile("mbarrier.arrive.release.cta.shared::cta.b64 _, [%0];\n" ::"r"((unsigned)__cvta_generic_to_shared(b))
                 : "memory");
}
__device__ __forceinline__ bool mbar_try(unsigned long long* b, int parity) {
    unsigned ok;
    asm volatile(
        "{\n.reg .pred p;\n"
        "mbarrier.try_wait.parity.acquire.cta.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"((unsigned)__cvta_generic_to_shared(b)), "r"(parity)
        : "memory");
    return ok != 0;
}
// bytes (a multiple of 16) from global to shared memory, both 16-byte
// aligned, counted on an mbarrier whose one arrival this is
__device__ __forceinline__ void bulk_load(void* dst, const void* src, int bytes, unsigned long long* b) {
    const unsigned bar = (unsigned)__cvta_generic_to_shared(b);
    asm volatile("mbarrier.arrive.expect_tx.release.cta.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes)
                 : "memory");
    asm volatile("cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
                     (unsigned)__cvta_generic_to_shared(dst)),
                 "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}

constexpr int kSweepWorkers = 16;                // most warps taking a level's elements, eight each
constexpr int kSweepHelpers = 4;                 // warps for copy-ins and write-backs
constexpr int kSweepService = kSweepHelpers + 3; // with the record, the publishing and the polling warp
constexpr int kSweepStop = 1 << 30;  // progress of a sweep after which nothing changes (or that failed)
// Tries (about 50 ns each) before a level's records are given up; and tries
// (100 ns and more) of the warp that brings them while neither the workers
// nor any earlier sweep move, several times what the polls take to notice.
constexpr int kSweepTries = 1 << 16;
constexpr int kSweepRecordTries = 1 << 26;

struct SweepArgs {
    const SweepElem* elems;
    const SweepRec* recs;
    const int* lev;
    const int4* epoch;
    const int* need;
    const int2 *load, *wb;
    const SceneDev* scenes;
    const int* order;
    const double4_32a* xo;
    double4_32a* av;
    const int* flags;
    int* ticket;
    int* progress;  // per scene and sweep: epochs written back
    int* stat;      // per scene and sweep: averaged edges, exact tests
    int* failed;    // per scene
    int workers;    // worker warps of the block
    int polls;      // polls without progress before a sweep gives up on the ones before (kSweepPolls)
};

// One CTA per scene and sweep. The sweeps of a scene are a pipeline through
// the mesh: a point's last element in sweep k lies only a few levels behind
// its first (6 levels on a grid sheet of any size), so sweep k + 1 may take
// it as soon as sweep k has written it back, and the ten sweeps of a scene
// of L levels take about L + 10 * 20 levels' time instead of 10 L. A sweep
// that starts although an earlier one found nothing to average changes
// nothing either; it is told to stop when that is known.
//
// CTAs take (scene, sweep) pairs from a ticket counter, a scene's sweeps in
// order, so a CTA waits only for one that has already started. The wait is
// bounded: a sweep gives up when none of those before it has moved for
// kSweepPolls polls (on a closed string the sweeps follow one another whole,
// so the one before may itself be waiting). A sweep that gives up, or finds a
// level's records missing, ends at the end of its step in all its warps
// together, and the scene is reported as failed.
//
// What bounds a level is its chain: barrier, slot loads, three FP32
// decisions, and where an edge averages its FP64 sums (~64 cycles each on
// this GPU). So the level loop holds nothing else: the worker warps take the
// elements, whose records one warp brings in by bulk copies up to
// kSweepRing levels ahead, and once per epoch (sw_k levels) they meet the kSweepHelpers warps that
// issue the copy-ins of the epoch after the next, form the FP32 values of
// those that have landed and write back the points last used in the epoch
// before, everything they read from global memory loaded a step ahead. A
// fence or a poll takes longer than an epoch's levels, so neither is on that
// path: one warp publishes what has been written back, one follows the sweep
// before, both at their own pace through flags in shared memory.
//
// Slots are for a point's live time only (cc_sweep_plan.h): a 129 x 129
// sheet takes 903 slots and 96 KB with its record ring.
//
// Measured (strain loop of one step, ten sweeps; before: one CTA per scene,
// sweep after sweep, edges on levels of their own): folded 129 x 129 sheet
// (510 levels, 73% of the edges averaging) 11.6 -> 0.89 ms, 257 x 257 sheet
// (1,022 levels) 17.6 -> 1.30 ms, 64 strings of 512 bonds 5.4 -> 0.53 ms,
// 256 scenes of 16..128 per side (70 of them averaging) 9.1 -> 2.6 ms. A
// level takes 1,000 to 2,900 cycles, about a third of it waiting for the
// next level's record and the barrier.
__global__ void __launch_bounds__((kSweepWorkers + kSweepService) * 32) k_strain_sweeps(const SweepArgs A) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int s_ticket, s_avg, s_exact, s_fail;
    __shared__ int s_stop[2];             // step t's in s_stop[t & 1]: everyone ends after it
    __shared__ int s_seen, s_wrote, s_quit;  // epochs the sweep before has published; helper warps' write-back steps
    __shared__ int s_moves;                  // times an earlier sweep was seen to move while the one before did not
    __shared__ unsigned long long s_full[kSweepRing], s_empty[kSweepRing];  // the record ring's levels
    __shared__ int2 s_level[kSweepRing];  // their first elements and counts
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) {
        s_ticket = atomicAdd(A.ticket, 1);
        s_avg = s_exact = s_fail = s_stop[0] = s_stop[1] = s_wrote = s_quit = s_moves = 0;
        // the first sweep waits for nothing
        s_seen = s_ticket % kStrainMaxIter == 0 ? kSweepStop - 1 : 0;
        for (int i = 0; i < kSweepRing; ++i) {
            mbar_init(&s_full[i], 1);
            mbar_init(&s_empty[i], 1);
        }
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    __syncthreads();
    const int sc = A.order[s_ticket / kStrainMaxIter], k = s_ticket % kStrainMaxIter;
    const SceneDev& sd = A.scenes[sc];
    if (!sd.sw_fits || !sd.enabled || !A.flags[2 * sc] || A.flags[2 * sc + 1]) return;
    const int K = sd.sw_k, L = sd.sw_levels, E = sd.sw_epochs, width = sd.sw_width;
    const int* lev = A.lev + sd.sw_lev0;
    const int4* epoch = A.epoch + sd.sw_ep0;
    SweepSlot* win = reinterpret_cast<SweepSlot*>(smem);
    const int W = min((width + 7) / 8, A.workers);
    if (warp >= W && warp < A.workers) return;
    const int stepped = (W + kSweepHelpers) * 32;  // threads meeting at the end of a step (barrier 2)
    const int all = (W + kSweepService) * 32;      // and at the end of the sweep (barrier 3)
    int* mine = A.progress + sc * kStrainMaxIter + k;
    SweepRec* ring = sd.sw_ring ? reinterpret_cast<SweepRec*>(win + sd.sw_slots) : nullptr;

    if (warp < W) {  // ---- workers: barrier 1 between the levels
        const int WT = W * 32, WQ = W * 8;  // threads, elements side by side
        const int c = tid & 3, quad = tid >> 2;
        const float sign = c < 3 ? -1.f : 1.f;
        const double dt = sd.p.dt;
        const float dt32 = (float)dt;
        int n_avg = 0, n_exact = 0;
        // the level's first element and count; none for a warp that waits in
        // vain: its lanes decide as one, and it goes on meeting the barriers
        // until the sweep ends (the vote goes while the level is loaded)
        auto level = [&](int l) {
            bool got = false;
            for (int tries = 0; !got && tries < kSweepTries; ++tries)
                got = mbar_try(&s_full[l % kSweepRing], (l / kSweepRing) & 1);
            const int2 lv = s_level[l % kSweepRing];
            const bool ok = __all_sync(0xffffffffu, got);
            if (!ok) flag_store(&s_fail, 1);
            return make_int2(ok ? lv.x : 0, ok ? lv.y : 0);
        };
        auto record = [&](int l, int2 lv, int i, SweepLane& r) {
            const int k = i < lv.y ? i : 0;  // lanes without an element read the level's first
            auto take = [&](const SweepRec& p) {
#pragma unroll
                for (int j = 0; j < 3; ++j) {
                    r.d[j] = reinterpret_cast<const float*>(&p.dx[j])[c];
                    r.limit[j] = p.limit[j];
                }
                r.s01 = p.s01;
                r.s2n = p.s2n;
            };
            if (ring)
                take(ring[(l % kSweepRing) * width + k]);
            else
                take(A.recs[lv.x + k]);
        };
        // a level's first record per thread is loaded before the barrier that
        // starts the level
        int l = 0;
        int2 lv = level(0);
        SweepLane r;
        record(0, lv, quad, r);
        for (int t = -2; t <= E; ++t) {
            if (t >= 0)
                for (int j = 0; j < K && l < L; ++j) {
                    if (j > 0) {
                        if (W > 1)
                            bar_sync(1, WT);
                        else
                            __syncwarp();
                        if (tid == 0) mbar_arrive(&s_empty[(l - 1) % kSweepRing]);
                    }
                    for (int i = quad;;) {
                        // (whole warps: the first of a warp's elements decides)
                        if ((i & ~7) >= lv.y) break;
                        sweep_element(r, i < lv.y, A.elems + lv.x + i, A.xo, win, c, sign, dt32, dt, &n_avg, &n_exact);
                        i += WQ;
                        if ((i & ~7) < lv.y) record(l, lv, i, r);
                    }
                    if (++l < L) {
                        lv = level(l);
                        record(l, lv, quad, r);
                    }
                }
            bar_sync(2, stepped);
            if (tid == 0 && t >= 0 && t < E) mbar_arrive(&s_empty[(l - 1) % kSweepRing]);
            if (s_stop[t & 1]) break;
        }
        n_avg = __reduce_add_sync(0xffffffffu, n_avg);
        n_exact = __reduce_add_sync(0xffffffffu, n_exact);
        if (lane == 0 && n_avg) atomicAdd(&s_avg, n_avg);
        if (lane == 0 && n_exact) atomicAdd(&s_exact, n_exact);
        bar_sync(3, all);
        return;
    }

    const int role = warp - A.workers;
    if (role < kSweepHelpers) {  // ---- copy-ins and write-backs
        const int h = tid - A.workers * 32;
        constexpr int HT = kSweepHelpers * 32;
        const int4 none = make_int4(0, 0, 0, 0);
        // the ranges of epochs t + 3 .. t - 1, what epoch t + 2 has to wait
        // for, and this thread's first copy-in of epoch t + 2 and write-back
        // of epoch t - 1, all loaded a step ahead
        const int* need_of = A.need + sd.sw_ep0;
        int4 in_next = E > 1 ? epoch[1] : none, in = epoch[0], in1 = none, cur = none, out = none;
        int need = need_of[0], need_next = E > 1 ? need_of[1] : 0;
        int2 ld = make_int2(-1, -1), ld1 = make_int2(-1, -1), wb = make_int2(-1, -1);
        if (in.x + h < in.y) ld = A.load[in.x + h];
        for (int t = -2; t <= E; ++t) {
            // loads for the next step
            int2 ld_n = make_int2(-1, -1), wb_n = make_int2(-1, -1);
            int4 in_n = none;
            int need_n = 0;
            if (in_next.x + h < in_next.y) ld_n = A.load[in_next.x + h];
            if (cur.z + h < cur.w) wb_n = A.wb[cur.z + h];
            if (t + 4 < E) {
                in_n = epoch[t + 4];
                need_n = need_of[t + 4];
            }
            // write-backs of epoch t - 1 (before the wait: the next sweep waits for them)
            if (t >= 1) {
                for (int i = out.z + h; i < out.w; i += HT) {
                    const int2 ps = i == out.z + h ? wb : A.wb[i];
                    const double* d = win[ps.y].d;
                    A.av[ps.x] = make_double4_32a(d[0], d[1], d[2], 0.0);
                }
                __syncwarp();
                if (lane == 0) flag_add(&s_wrote, 1);
            }
            // copy-ins of epoch t + 2
            int seen;
            while ((seen = flag_load(&s_seen)) < need) __nanosleep(20);
            for (int i = in.x + h; i < in.y; i += HT) {
                const int2 ps = i == in.x + h ? ld : A.load[i];
                cp_async16(&win[ps.y].d[0], &A.av[ps.x]);
                cp_async16(&win[ps.y].d[2], reinterpret_cast<const char*>(&A.av[ps.x]) + 16);
            }
            cp_commit();
            // FP32 values of epoch t + 1, whose copies were issued a step ago
            cp_wait<1>();
            for (int i = in1.x + h; i < in1.y; i += HT) {
                const int2 ps = i == in1.x + h ? ld1 : A.load[i];
                SweepSlot& w = win[ps.y];
                *reinterpret_cast<float4*>(w.f) = cut32x3(w.d[0], w.d[1], w.d[2]);
            }
            if (h == 0) s_stop[t & 1] = seen >= kSweepStop || flag_load(&s_fail) ? 1 : 0;
            bar_sync(2, stepped);
            if (s_stop[t & 1]) break;
            out = cur;
            wb = wb_n;
            cur = in1;
            in1 = in;
            ld1 = ld;
            in = in_next;
            ld = ld_n;
            need = need_next;
            in_next = in_n;
            need_next = need_n;
        }
        cp_wait<0>();
        if (h == 0) flag_store(&s_quit, 1);
        bar_sync(3, all);
        return;
    }
    if (role == kSweepHelpers) {  // ---- publishes the epochs written back
        if (lane == 0)
            for (int done = 0; done < E - 1 && !flag_load(&s_quit);) {
                const int n = flag_load(&s_wrote) / kSweepHelpers;  // steps 1 .. n: epochs 0 .. n - 1
                if (n > done && n < E) {
                    __threadfence();
                    st_relaxed(mine, n);
                    done = n;
                } else {
                    __nanosleep(20);
                }
            }
        bar_sync(3, all);
        if (lane == 0) {
            A.stat[2 * (sc * kStrainMaxIter + k)] = s_avg;
            A.stat[2 * (sc * kStrainMaxIter + k) + 1] = s_exact;
            if (s_fail) A.failed[sc] = 1;
            __threadfence();
            st_relaxed(mine, s_avg == 0 || s_fail ? kSweepStop : E);
        }
        return;
    }
    if (role == kSweepHelpers + 1) {  // ---- brings the records of the levels, kSweepRing ahead
        int issued = 0;
        int off = lane <= L ? lev[lane] : 0, off_next = 0;  // offsets of 32 levels, and of the next
        for (int l = 0; l < L; ++l) {
            if (l % 32 == 0) {
                if (l > 0) off = off_next;
                off_next = l + 32 + lane <= L ? lev[l + 32 + lane] : 0;
            }
            const int o0 = __shfl_sync(0xffffffffu, off, l % 32);
            const int oa = __shfl_sync(0xffffffffu, off, (l + 1) % 32);
            const int ob = __shfl_sync(0xffffffffu, off_next, 0);
            const int n = (l % 32 == 31 ? ob : oa) - o0;
            const int slot = l % kSweepRing;
            bool go = true;
            if (l >= kSweepRing)
                for (int tries = 0, last = 0; !mbar_try(&s_empty[slot], (l / kSweepRing - 1) & 1);) {
                    // (the workers may wait for another sweep, and that one for others)
                    const int moved = flag_load(&s_seen) + flag_load(&s_moves);
                    if (moved != last) tries = 0;
                    last = moved;
                    if (flag_load(&s_quit) || ++tries > kSweepRecordTries) {
                        go = false;
                        break;
                    }
                    __nanosleep(100);
                }
            if (!__all_sync(0xffffffffu, go)) break;
            if (lane == 0) {
                s_level[slot] = make_int2(o0, n);
                if (ring)
                    bulk_load(ring + (size_t)slot * width, A.recs + o0, n * kSweepRecBytes, &s_full[slot]);
                else
                    mbar_arrive(&s_full[slot]);
            }
            issued = l + 1;
        }
        // nothing may be in flight into this block's memory when it ends
        for (int l = max(0, issued - kSweepRing); l < issued; ++l)
            for (int tries = 0; tries < kSweepTries && !mbar_try(&s_full[l % kSweepRing], (l / kSweepRing) & 1);)
                ++tries;
        bar_sync(3, all);
        return;
    }
    // ---- follows the sweep before
    if (lane == 0 && k > 0) {
        unsigned others = 0;  // epochs of the sweeps before that one
        for (int seen = 0, polls = 0; seen < E && !flag_load(&s_quit);) {
            const int now = ld_acquire(mine - 1);
            if (now > seen) {
                flag_store(&s_seen, now);
                seen = now;
                polls = 0;
            } else if (++polls > A.polls) {
                unsigned sum = 0;  // (an ended sweep's kSweepStop cut so that nine fit)
                for (int j = 2; j <= k; ++j) sum += (unsigned)min(ld_acquire(mine - j), kSweepStop >> 2);
                if (sum == others) {
                    flag_store(&s_fail, 1);
                    flag_store(&s_seen, kSweepStop);
                    break;
                }
                others = sum;
                polls = 0;
                flag_add(&s_moves, 1);
            } else {
                __nanosleep(40);
            }
        }
    }
    bar_sync(3, all);
}

// The sweeps' outcome per scene: the passes the reference's loop takes (its
// last is the first to average nothing, or the tenth), and the totals.
__global__ void k_sweep_count(const SceneDev* __restrict__ scenes, int nscenes, const int* __restrict__ flags,
                              const int* __restrict__ stat, const int* __restrict__ failed, int* passes_out) {
    const int sc = blockIdx.x * blockDim.x + threadIdx.x;
    if (sc >= nscenes || !scenes[sc].sw_fits || !scenes[sc].enabled || flags[2 * sc + 1]) return;
    int passes = 1, avg = 0, exact = 0;
    if (flags[2 * sc])
        for (int k = 0; k < kStrainMaxIter; ++k) {
            const int* s = stat + 2 * (sc * kStrainMaxIter + k);
            avg += s[0];
            exact += s[1];
            passes = k + 1;
            if (s[0] == 0) break;
        }
    passes_out[3 * sc] = failed[sc] ? -1 : passes;
    passes_out[3 * sc + 1] = avg;
    passes_out[3 * sc + 2] = exact;
}

// Start of a strain loop for the scenes in mask (all: mask null): their
// flags, counters and pipeline state cleared; the others marked finished, so
// that every kernel of this loop leaves them and their counters alone.
__global__ void k_strain_init(const uint8_t* __restrict__ mask, int nscenes, int* flags, int* passes_out, int* ticket,
                              int* progress, int* stat, int* failed) {
    int sc = blockIdx.x * blockDim.x + threadIdx.x;
    if (sc >= nscenes) return;
    if (sc == 0) *ticket = 0;
    if (mask && !mask[sc]) {
        flags[2 * sc + 1] = 1;
        return;
    }
    flags[2 * sc] = flags[2 * sc + 1] = 0;
    passes_out[3 * sc] = passes_out[3 * sc + 1] = passes_out[3 * sc + 2] = 0;
    failed[sc] = 0;
    for (int k = 0; k < kStrainMaxIter; ++k) {
        progress[sc * kStrainMaxIter + k] = 0;
        stat[2 * (sc * kStrainMaxIter + k)] = stat[2 * (sc * kStrainMaxIter + k) + 1] = 0;
    }
}

}  // namespace

size_t strain_edge_step_bytes(int nedges) { return sizeof(StrainEdgeStep) * (size_t)(nedges > 0 ? nedges : 1); }
int strain_state_ints(int nscenes) { return 1 + nscenes * (1 + 3 * kStrainMaxIter); }

void strain_configure() {
    cudaFuncSetAttribute(k_strain_sweeps, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSweepMaxBytes);
}

void strain_setup(const StrainBufs& b, const StrainPlan& plan, const double4_32a* xo, cudaStream_t s) {
    if (b.nelems > 0)
        count_launch(), k_sweep_setup<<<nblk(b.nelems, 256), 256, 0, s>>>(b.elems, b.nelems, xo, (SweepRec*)b.recs);
    if (plan.any_global && b.nedges > 0)
        count_launch(), k_edge_setup<<<nblk(b.nedges, 256), 256, 0, s>>>(b.edges, b.nedges, xo,
                                                                         (StrainEdgeStep*)b.edge_steps);
}

void strain_limit(const StrainBufs& b, const SceneDev* scenes, int nscenes, const StrainPlan& plan,
                  const double4_32a* xo, double4_32a* av, const uint8_t* mask, cudaStream_t s) {
    if (nscenes <= 0) return;
    int* ticket = b.state;
    int* failed = ticket + 1;
    int* progress = failed + nscenes;
    int* stat = progress + nscenes * kStrainMaxIter;
    count_launch(), k_strain_init<<<nblk(nscenes, 128), 128, 0, s>>>(mask, nscenes, b.flags, b.passes_out, ticket,
                                                                     progress, stat, failed);
    const SweepRec* recs = (const SweepRec*)b.recs;
    const int window = plan.window ? 1 : 0;
    auto check = [&](int which) {
        if (b.nchunks > 0)
            count_launch(), k_sweep_check<<<b.nchunks < 152 * 8 ? b.nchunks : 152 * 8, 256, 0, s>>>(
                b.elems, recs, xo, b.chunks, b.nchunks, scenes, av, window, which, b.flags);
    };
    check(0);
    if (plan.window) {
        SweepArgs a{b.elems, recs, b.lev, b.epoch, b.need, b.load, b.wb, scenes, b.order, xo, av, b.flags,
                    ticket, progress, stat, failed, plan.workers, plan.polls};
        count_launch(), k_strain_sweeps<<<nscenes * kStrainMaxIter, (plan.workers + kSweepService) * 32, plan.smem,
                                          s>>>(a);
        count_launch(), k_sweep_count<<<nblk(nscenes, 128), 128, 0, s>>>(scenes, nscenes, b.flags, stat, failed,
                                                                         b.passes_out);
    }
    if (plan.any_global)
        for (int pass = 0; pass < kStrainMaxIter; ++pass) {
            if (pass > 0) check(1);
            count_launch(), k_strain<<<nscenes, 256, 0, s>>>((const StrainEdgeStep*)b.edge_steps, b.hdr, scenes,
                                                             window, av, pass, b.flags, b.passes_out, b.order);
        }
}

}  // namespace ccg
