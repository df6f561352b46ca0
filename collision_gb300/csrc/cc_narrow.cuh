// Narrow phase on the GPU: proximity (t = 0) and continuous (CCD) tests of
// one element pair, and the repulsion / inelastic / friction impulses of each
// hit, emitted as keyed per-point contributions instead of the reference's
// in-place accumulation (dcollid3d.cpp:925-1300).
//
// One thread handles one element pair; positions stay in registers (the
// reference writes them into the shared POINT coordinates, dcollid3d.cpp:333-339).
#pragma once

#include "cc_common.cuh"
#include "cc_crmath.cuh"

namespace ccg {

struct NarrowCtx {
    const double4_32a* xo;       // x_old per point
    const double4_32a* av;       // average velocity per point
    const uint8_t* fixed;    // per point: bit 0 is_fixed, bit 1 is_movableRG
    const int* ev;           // 3 point ids per element (bonds: third is -1)
    const int* esurf;        // surface id per element (-1 for bonds)
    const uint8_t* erigid;   // element has a fixed or movable point (isRigidBody(hse))
    const int* vbody;        // movable body of each point, -1 for none
    const double* body_mass; // total_mass of each body
    int body_slot0;          // contribution slot of body 0 (after every point's)
    const int* rank;         // leaf rank of each element in its scene's reference tree
    int pass;                // the scene's pass index
    int zone;                // impact-zone mode (s_detImpZone) of the scene
    Params p;                // the scene's parameters
    Contrib* contrib;
    int contrib_cap;
    PassCounters* ctr;
    UnionRec* urec;          // createImpZone calls of impact-zone passes
    int urec_cap;
    VisitRec* rec;
    int rec_cap;
    // mixed precision: per-point FP32 boxes over the pass's time window
    // (rounded outward), used to reject sub-tests that cannot hit
    const float4* pbox_lo;
    const float4* pbox_hi;
    const float4* p32;    // x_old rounded to FP32
    const float4* v32;    // avgVel rounded to FP32 (moving passes)
    float hpad;   // h of the sub-tests, padded (filter_reach)
    float epad;   // eps (barycentric tolerance), rounded up
    int check;    // decide hits only: no impulses, contacts or zones
    float dt32;   // dt rounded up to FP32
};

struct CallState {
    unsigned long long keybase;
    int plist[6];
    int np;
    int dcount[6];
    int sub;
    int nsub;   // sub-tests evaluated in FP64
    int ncr;    // cubics with a root in the time window
    int ncontacts;
};

__device__ __forceinline__ bool is_static(const NarrowCtx& c, int p) { return (c.fixed[p] & 1) != 0; }
__device__ __forceinline__ bool is_movable(const NarrowCtx& c, int p) { return (c.fixed[p] & 2) != 0; }
__device__ __forceinline__ bool is_rigid(const NarrowCtx& c, int p) { return c.fixed[p] != 0; }

__device__ __forceinline__ void emit(const NarrowCtx& c, CallState& st, int vertex, const double* imp,
                                     const double* fric, int has_fric) {
    for (int i = 0; i < st.np; ++i)
        if (st.plist[i] == vertex) { st.dcount[i]++; break; }
    int slot = aggregated_add(&c.ctr->ncontrib, 1);
    if (slot >= c.contrib_cap) {
        atomicOr(&c.ctr->err, kErrContribOverflow);
        return;
    }
    Contrib& o = c.contrib[slot];
    o.key = st.keybase | (unsigned long long)st.sub;
    o.vertex = vertex;
    o.flags = has_fric;
    for (int j = 0; j < 3; ++j) { o.imp[j] = imp[j]; o.fric[j] = fric[j]; }
}

// SpreadImpactZoneImpulse (dcollid.cpp:1101-1115) adds impulse*nor to the
// collsnImpulse_RG of every member of p's zone - a movable body's zone is the
// body - and counts one. Every member gets the same additions in the same
// order, so the sum is kept once per body, in a contribution slot of its own.
__device__ __forceinline__ void emit_body(const NarrowCtx& c, CallState& st, int p, double impulse,
                                          const double* nor) {
    int slot = aggregated_add(&c.ctr->ncontrib, 1);
    if (slot >= c.contrib_cap) {
        atomicOr(&c.ctr->err, kErrContribOverflow);
        return;
    }
    Contrib& o = c.contrib[slot];
    o.key = st.keybase | (unsigned long long)st.sub;
    o.vertex = c.body_slot0 + c.vbody[p];
    o.flags = 0;
    for (int j = 0; j < 3; ++j) { o.imp[j] = impulse * nor[j]; o.fric[j] = 0.0; }
}

// ---------------------------------------------------------------- unions
// createImpZone(pts, 4), dcollid.cpp:473-484: the four points join one zone.
// The call is recorded with its visiting-order key; the unions themselves
// are replayed in that order after the pass.
__device__ __forceinline__ void create_imp_zone(const NarrowCtx& c, const CallState& st, const int* pts) {
    int slot = aggregated_add(&c.ctr->nunion, 1);
    if (slot >= c.urec_cap) {
        atomicOr(&c.ctr->err, kErrUnionOverflow);
        return;
    }
    UnionRec r;
    r.key = st.keybase | (unsigned long long)st.sub;
    for (int i = 0; i < 4; ++i) r.p[i] = pts[i];
    c.urec[slot] = r;
}

// -------------------------------------------------------------- impulses
// PointToTriImpulse, dcollid3d.cpp:925-1107.
static __device__ void point_to_tri_impulse(const NarrowCtx& c, CallState& st, const int* pts, const double* nor,
                                     double* w, double dist) {
    double v_rel[3] = {0.0, 0.0, 0.0}, vn, vt;
    double impulse = 0.0, m_impulse, sum_w = 0.0;
    double rigid_impulse[2] = {0.0, 0.0};
    const double k = c.p.k, m = c.p.m, dt = c.p.dt, lambda = c.p.lambda, h = c.p.thickness, cr = c.p.cr;
    double av[4][3];
    for (int q = 0; q < 4; ++q) load3(c.av, pts[q], av[q]);
    bool st0 = is_static(c, pts[0]), st1 = is_static(c, pts[1]), st2 = is_static(c, pts[2]),
         st3 = is_static(c, pts[3]);
    bool mv[4] = {is_movable(c, pts[0]), is_movable(c, pts[1]), is_movable(c, pts[2]), is_movable(c, pts[3])};
    dist = h - dist;
    for (int i = 0; i < 3; ++i) {
        v_rel[i] += av[3][i];
        for (int j = 0; j < 3; ++j) v_rel[i] -= w[j] * av[j][i];
    }
    vn = dot3(v_rel, nor);
    if (dot3(v_rel, v_rel) > sqr(vn))
        vt = sqrt(dot3(v_rel, v_rel) - sqr(vn));
    else
        vt = 0.0;
    bool tri_static[3] = {st0, st1, st2};
    if (vn < 0) {
        if (st3 || (st0 && st1 && st2)) {
            impulse = vn;
            rigid_impulse[0] = vn;
            rigid_impulse[1] = vn;
        } else if (mv[0] && mv[1] && mv[2] && mv[3]) {
            double m1 = c.body_mass[c.vbody[pts[0]]], m2 = c.body_mass[c.vbody[pts[3]]];
            rigid_impulse[0] = vn * m2 / (m1 + m2);
            rigid_impulse[1] = vn * m1 / (m1 + m2);
        } else if (mv[0] && mv[1] && mv[2]) {
            rigid_impulse[0] = 0.5 * vn;
            impulse = 0.5 * vn;
        } else if (mv[3]) {
            impulse = 0.5 * vn;
            rigid_impulse[1] = 0.5 * vn;
        } else {
            impulse = vn * 0.5;
        }
        for (int i = 0; i < 3; ++i) {
            if (tri_static[i]) w[i] = 0.0;
            sum_w += w[i];
        }
        if (fabs(sum_w) > kMachEps) {
            double inv = 1.0 / sum_w;
            for (int i = 0; i < 3; ++i) w[i] = inv * w[i];
        }
    }
    bool all_rigid = is_rigid(c, pts[0]) && is_rigid(c, pts[1]) && is_rigid(c, pts[2]) && is_rigid(c, pts[3]);
    if (vn * dt < 0.1 * dist) {
        if (all_rigid) {
            rigid_impulse[0] *= 1.0 + cr;
            rigid_impulse[1] *= 1.0 + cr;
        } else {
            double tmp = -smin(dt * k * dist / m, (0.1 * dist / dt - vn));
            impulse += tmp;
            rigid_impulse[0] += tmp;
            rigid_impulse[1] += tmp;
        }
    }
    if (fabs(sum_w) < kMachEps)
        m_impulse = impulse;
    else
        m_impulse = 2.0 * impulse / (1.0 + dot3(w, w));
    if (all_rigid) {
        if (mv[0]) emit_body(c, st, pts[0], rigid_impulse[0], nor);
        if (mv[3]) emit_body(c, st, pts[3], -1.0 * rigid_impulse[1], nor);
        return;
    }
    int has_fric = fabs(vt) > kRoundEps;
    const double inv_vt = 1.0 / vt;
    double imp[3], fric[3], slide[3];
    for (int j = 0; j < 3; ++j) slide[j] = v_rel[j] - vn * nor[j];
    for (int i = 0; i < 3; ++i) {
        if (tri_static[i]) continue;
        double t_impulse = mv[i] ? rigid_impulse[0] : m_impulse;
        const double share = w[i] * t_impulse;
        const double f = has_fric ? smax(-fabs(quotient(lambda * w[i] * t_impulse, vt, inv_vt)), -1.0) : 0.0;
        for (int j = 0; j < 3; ++j) {
            imp[j] = share * nor[j];
            fric[j] = has_fric ? f * slide[j] : 0.0;
        }
        emit(c, st, pts[i], imp, fric, has_fric);
    }
    if (!st3) {
        double t_impulse = mv[3] ? rigid_impulse[1] : m_impulse;
        const double f = has_fric ? smax(-fabs(quotient(lambda * t_impulse, vt, inv_vt)), -1.0) : 0.0;
        for (int j = 0; j < 3; ++j) {
            imp[j] = -(t_impulse * nor[j]);
            fric[j] = has_fric ? f * slide[j] : 0.0;
        }
        emit(c, st, pts[3], imp, fric, has_fric);
    }
}

// EdgeToEdgeImpulse, dcollid3d.cpp:1109-1300.
static __device__ void edge_to_edge_impulse(const NarrowCtx& c, CallState& st, const int* pts, const double* nor,
                                     double a, double b, double dist) {
    double v_rel[3], vn, vt;
    double impulse = 0.0, m_impulse;
    double rigid_impulse[2] = {0.0, 0.0};
    const double k = c.p.k, m = c.p.m, dt = c.p.dt, lambda = c.p.lambda, h = c.p.thickness, cr = c.p.cr;
    double wa[2] = {1.0 - a, a}, wb[2] = {1.0 - b, b};
    double av[4][3];
    for (int q = 0; q < 4; ++q) load3(c.av, pts[q], av[q]);
    bool sq[4] = {is_static(c, pts[0]), is_static(c, pts[1]), is_static(c, pts[2]), is_static(c, pts[3])};
    bool mv[4] = {is_movable(c, pts[0]), is_movable(c, pts[1]), is_movable(c, pts[2]), is_movable(c, pts[3])};
    dist = h - dist;
    for (int j = 0; j < 3; ++j) {
        v_rel[j] = (1.0 - b) * av[2][j] + b * av[3][j];
        v_rel[j] -= (1.0 - a) * av[0][j] + a * av[1][j];
    }
    vn = dot3(v_rel, nor);
    if (dot3(v_rel, v_rel) > sqr(vn))
        vt = sqrt(dot3(v_rel, v_rel) - sqr(vn));
    else
        vt = 0.0;
    if (vn < 0.0) {
        if ((sq[0] && sq[1]) || (sq[2] && sq[3])) {
            impulse = vn;
            rigid_impulse[0] = vn;
            rigid_impulse[1] = vn;
        } else if (mv[0] && mv[1] && mv[2] && mv[3]) {
            double m1 = c.body_mass[c.vbody[pts[0]]], m2 = c.body_mass[c.vbody[pts[2]]];
            rigid_impulse[0] = vn * m2 / (m1 + m2);
            rigid_impulse[1] = vn * m1 / (m1 + m2);
        } else if (mv[0] && mv[1]) {
            rigid_impulse[0] = 0.5 * vn;
            impulse = 0.5 * vn;
        } else if (mv[2] && mv[3]) {
            impulse = 0.5 * vn;
            rigid_impulse[1] = 0.5 * vn;
        } else {
            impulse = vn * 0.5;
        }
        if (sq[0]) wa[0] = 0.0;
        if (sq[1]) wa[1] = 0.0;
        if (sq[2]) wb[0] = 0.0;
        if (sq[3]) wb[1] = 0.0;
    }
    bool all_rigid = is_rigid(c, pts[0]) && is_rigid(c, pts[1]) && is_rigid(c, pts[2]) && is_rigid(c, pts[3]);
    if (vn * dt < 0.1 * dist) {
        if (all_rigid) {
            rigid_impulse[0] *= 1.0 + cr;
            rigid_impulse[1] *= 1.0 + cr;
        } else {
            double tmp = -smin(dt * k * dist / m, (0.1 * dist / dt - vn));
            impulse += tmp;
            rigid_impulse[0] += tmp;
            rigid_impulse[1] += tmp;
        }
    }
    if (wa[0] + wa[1] < kMachEps || wb[0] + wb[1] < kMachEps)
        m_impulse = impulse;
    else
        m_impulse = 2.0 * impulse / (wa[0] * wa[0] + wa[1] * wa[1] + wb[0] * wb[0] + wb[1] * wb[1]);
    if (all_rigid) {
        if (mv[0]) emit_body(c, st, pts[0], rigid_impulse[0], nor);
        if (mv[2]) emit_body(c, st, pts[2], -1.0 * rigid_impulse[1], nor);
        return;
    }
    int has_fric = fabs(vt) > kRoundEps;
    const double wgt[4] = {wa[0], wa[1], wb[0], wb[1]};
    const double inv_vt = 1.0 / vt;
    double imp[3], fric[3], slide[3];
    for (int j = 0; j < 3; ++j) slide[j] = v_rel[j] - vn * nor[j];
    for (int q = 0; q < 4; ++q) {
        if (sq[q]) continue;
        double t_impulse = mv[q] ? rigid_impulse[q < 2 ? 0 : 1] : m_impulse;
        const double share = wgt[q] * t_impulse;
        const double f = has_fric ? smax(-fabs(quotient(lambda * wgt[q] * t_impulse, vt, inv_vt)), -1.0) : 0.0;
        for (int j = 0; j < 3; ++j) {
            double d = share * nor[j];
            imp[j] = (q < 2) ? d : -d;
            fric[j] = has_fric ? f * slide[j] : 0.0;
        }
        emit(c, st, pts[q], imp, fric, has_fric);
    }
}

// ------------------------------------------------------- point / edge tests
// v / d, each component as rounded by the division.
__device__ __forceinline__ void divide3(double* v, double d) {
    const double inv = 1.0 / d;
    for (int i = 0; i < 3; ++i) v[i] = quotient(v[i], d, inv);
}

// PointToTri, dcollid3d.cpp:778-922. pts[0..2] the triangle, pts[3] the
// point; X holds the four positions the reference keeps in Coords.
static __device__ bool point_to_tri(const NarrowCtx& c, CallState& st, const int* pts, const double (*X)[3], double h) {
    double w[3] = {0.0, 0.0, 0.0};
    double x13[3], x23[3], x43[3];
    double nor[3] = {0.0, 0.0, 0.0}, nor_mag, dist, det;
    for (int i = 0; i < 3; ++i) {
        x13[i] = X[0][i] - X[2][i];
        x23[i] = X[1][i] - X[2][i];
        x43[i] = X[3][i] - X[2][i];
    }
    det = dot3(x13, x13) * dot3(x23, x23) - dot3(x13, x23) * dot3(x13, x23);
    if (fabs(det) < 1000 * kMachEps) return false;
    cross3(x13, x23, nor);
    nor_mag = mag3(nor);
    double xo[4][3];
    for (int q = 0; q < 4; ++q) load3(c.xo, pts[q], xo[q]);
    double x43_old[3];
    for (int i = 0; i < 3; ++i) x43_old[i] = xo[3][i] - xo[2][i];
    dist = dot3(x43_old, nor);
    divide3(nor, nor_mag * ((dist >= 0) ? 1.0 : -1.0));
    dist = fabs(dot3(x43, nor));
    const double inv_det = 1.0 / det;
    w[0] = quotient(dot3(x13, x43) * dot3(x23, x23) - dot3(x23, x43) * dot3(x13, x23), det, inv_det);
    w[1] = quotient(dot3(x13, x13) * dot3(x23, x43) - dot3(x13, x23) * dot3(x13, x43), det, inv_det);
    w[2] = 1 - w[0] - w[1];
    if (fabs(w[0]) < kRoundEps || fabs(w[1]) < kRoundEps || fabs(w[2]) < kRoundEps) {
        double vec[3];
        for (int j = 0; j < 3; ++j) vec[j] = xo[3][j];
        for (int i = 0; i < 3; ++i)
            for (int j = 0; j < 3; ++j) vec[j] -= w[i] * xo[i][j];
        double vec_mag = mag3(vec);
        if (vec_mag > kRoundEps)
            for (int j = 0; j < 3; ++j) nor[j] = vec[j];
    }
    nor_mag = mag3(nor);
    if (nor_mag > kRoundEps) {
        divide3(nor, nor_mag);
    } else {
        atomicOr(&c.ctr->err, kErrNan);  // "nan nor vec": the reference exits
        return false;
    }
    if (dist > h) return false;
    for (int i = 0; i < 3; ++i)
        if (w[i] > 1 + c.p.eps || w[i] < -c.p.eps) return false;
    if (c.check) return true;
    st.ncontacts++;
    point_to_tri_impulse(c, st, pts, nor, w, dist);
    return true;
}

// EdgeToEdge, dcollid3d.cpp:643-776. Edges (pts[0],pts[1]) and (pts[2],pts[3]).
static __device__ bool edge_to_edge(const NarrowCtx& c, CallState& st, const int* pts, const double (*X)[3], double h) {
    double x21[3], x43[3], x31[3], tmp[3], v1[3], v2[3], nor[3];
    double a, b, nor_mag, dist;
    for (int i = 0; i < 3; ++i) {
        x21[i] = X[1][i] - X[0][i];
        x43[i] = X[3][i] - X[2][i];
        x31[i] = X[2][i] - X[0][i];
    }
    cross3(x21, x43, tmp);
    if (mag3(tmp) < kRoundEps) return false;
    double d4343 = dot3(x43, x43), d2131 = dot3(x21, x31), d2143 = dot3(x21, x43), d4331 = dot3(x43, x31),
           d2121 = dot3(x21, x21);
    const double den = d2121 * d4343 - d2143 * d2143, inv_den = 1.0 / den;
    a = quotient(d4343 * d2131 - d2143 * d4331, den, inv_den);
    b = quotient(d2143 * d2131 - d2121 * d4331, den, inv_den);
    a = smax(smin(a, 1.0), 0.0);
    b = smax(smin(b, 1.0), 0.0);
    for (int i = 0; i < 3; ++i) {
        v1[i] = a * x21[i];
        v2[i] = b * x43[i];
    }
    for (int i = 0; i < 3; ++i) {
        v1[i] = X[0][i] + v1[i];
        v2[i] = X[2][i] + v2[i];
    }
    for (int i = 0; i < 3; ++i) nor[i] = v2[i] - v1[i];
    nor_mag = mag3(nor);
    // the distance: the same squares in the same order
    dist = nor_mag;
    if (nor_mag < 1000 * kMachEps) {
        double xo[4][3];
        for (int q = 0; q < 4; ++q) load3(c.xo, pts[q], xo[q]);
        for (int j = 0; j < 3; ++j) {
            nor[j] = (1.0 - b) * xo[2][j] + b * xo[3][j];
            nor[j] -= (1.0 - a) * xo[0][j] + a * xo[1][j];
        }
        nor_mag = mag3(nor);
    }
    if (dist > h) return false;
    if (nor_mag < kMachEps) {
        atomicOr(&c.ctr->err, kErrNan);  // "Normal vector is nan": the reference exits
        return false;
    }
    divide3(nor, nor_mag);
    if (c.check) return true;
    st.ncontacts++;
    edge_to_edge_impulse(c, st, pts, nor, a, b, dist);
    return true;
}

// ------------------------------------------------------------------- CCD
// The coplanarity cubic a t^3 + b t^2 + c t + d of four points
// (dcollid3d.cpp:371-408).
struct Cubic {
    double a, b, c, d;
};
// x, v: the positions and velocities of points 1 .. 3 from point 0's.
__device__ __forceinline__ Cubic coplanarity_cubic(const double (*xo4)[3], const double (*av4)[3], double (*x)[3],
                                                   double (*v)[3]) {
    Cubic q;
    for (int i = 1; i < 4; ++i)
        for (int j = 0; j < 3; ++j) {
            v[i][j] = av4[i][j] - av4[0][j];
            x[i][j] = xo4[i][j] - xo4[0][j];
        }
    double vv[3], vx[3], xx[3];
    vv[0] = v[1][1] * v[2][2] - v[1][2] * v[2][1];
    vv[1] = v[1][0] * v[2][2] - v[1][2] * v[2][0];
    vv[2] = v[1][0] * v[2][1] - v[1][1] * v[2][0];
    vx[0] = v[1][1] * x[2][2] - v[1][2] * x[2][1] - v[2][1] * x[1][2] + v[2][2] * x[1][1];
    vx[1] = v[1][0] * x[2][2] - v[1][2] * x[2][0] - v[2][0] * x[1][2] + v[2][2] * x[1][0];
    vx[2] = v[1][0] * x[2][1] - v[1][1] * x[2][0] - v[2][0] * x[1][1] + v[2][1] * x[1][0];
    xx[0] = x[1][1] * x[2][2] - x[1][2] * x[2][1];
    xx[1] = x[1][0] * x[2][2] - x[1][2] * x[2][0];
    xx[2] = x[1][0] * x[2][1] - x[1][1] * x[2][0];
    q.a = v[3][0] * vv[0] - v[3][1] * vv[1] + v[3][2] * vv[2];
    q.b = x[3][0] * vv[0] - x[3][1] * vv[1] + x[3][2] * vv[2] + v[3][0] * vx[0] - v[3][1] * vx[1] + v[3][2] * vx[2];
    q.c = x[3][0] * vx[0] - x[3][1] * vx[1] + x[3][2] * vx[2] + v[3][0] * xx[0] - v[3][1] * xx[1] + v[3][2] * xx[2];
    q.d = x[3][0] * xx[0] - x[3][1] * xx[1] + x[3][2] * xx[2];
    return q;
}

// Whether isCoplanar can find no root in its window [0, dt + 2 MACH_EPS],
// for |a| > MACH_EPS, from the coefficients alone: true only when it is
// certain, so that acos, cos and pow need not run. (They are most of a
// sub-test: ~400 of its ~500 FP64 instructions.)
//
// isCoplanar forms the roots of p(x) = x^3 + A x^2 + B x + C with A = b/a,
// B = c/a, C = d/a. Let u = 2^-53 and T >= max(|A|, sqrt|B|, cbrt|C|), so
// that |Q| <= 4/9 T^2, |R| <= 0.71 T^3 and Cardano's |A'| <= 1.2 T.
//  - The rounding of Q and R, of z, and of R^2 - Q^3 is that of exact
//    arithmetic on a cubic whose B and C are off by at most 16 u (A^2 + |B|)
//    <= 32 u T^2 and 32 u (|A|^3 + |A B| + |C|) <= 96 u T^3.
//  - The functions and the last operations move a root by at most
//    2^-44 (2 sqrt Q + 2 |A'| + |A|) <= 2560 u T (pow's exponent 1/3 is
//    rounded, which costs up to 120 u), and where |A'| < ROUND_EPS drops
//    Q / A' every root taken lies within 4e-10 of the real one.
//  - The double root taken when |A' - B'| < ROUND_EPS is the real part of
//    two roots at most 0.87e-10 away, where |p| <= 3 |A'| 0.75e-20.
// So if a root falls in the window, |p(x)| <= 32 u T^2 |x| + 96 u T^3 +
// 2e-19 T for some x within E = 2560 u T + 5e-10 of it. The Bernstein
// coefficients of the cubic on [0, dt] bound it there from below when they
// have one sign; outside [0, dt] it changes by at most E (|c| + 2 |b| X + 3
// |a| X^2). All terms are formed in FP32 from coefficients cut to FP32
// (errors below 2^-20 of the sum of the terms' magnitudes in all; 2^-19
// is taken).
__device__ __forceinline__ bool no_root_in_window(const Cubic& q, double dt) {
    const float a = cut32(q.a), b = cut32(q.b), c = cut32(q.c), d = cut32(q.d), w = (float)dt;
    const float fa = fabsf(a), fb = fabsf(b), fc = fabsf(c), fd = fabsf(d);
    const float w2 = w * w, w3 = w2 * w;
    const float third = 1.0f / 3.0f;
    const float b1 = d + c * w * third, b2 = d + (2.0f * c * w + b * w2) * third, b3 = d + c * w + b * w2 + a * w3;
    const float lo = fminf(fminf(d, b1), fminf(b2, b3)), hi = fmaxf(fmaxf(d, b1), fmaxf(b2, b3));
    const float low = fmaxf(lo, -hi);  // positive when the four have one sign: the least magnitude
    if (!(low > 0.f)) return false;
    const float ra = 1.0f / fa;
    const float T = 1.01f * fmaxf(fb * ra, fmaxf(sqrtf(fc * ra), exp2f(log2f(fd * ra) * third)));
    const float E = 3e-13f * T + 5e-10f;
    const float X = w + E;
    const float slope = fc + 2.0f * fb * X + 3.0f * fa * X * X;
    const float mag = fd + fc * w + fb * w2 + fa * w3;
    const float need = 0x1p-19f * mag + 1.01f * E * slope +
                       1.1f * fa * T * (4e-15f * T * X + 1.1e-14f * T * T + 2e-19f) + 1e-30f;
    return low > need;
}

// The roots where |a| <= MACH_EPS: quadratic or linear (dcollid3d.cpp:459-472).
__device__ __forceinline__ void low_degree_roots(double a, double b, double c, double* roots) {
    double delta = b * b - 4.0 * a * c;
    if (fabs(a) > kRoundEps && delta > 0) {
        double ds = sqrt(delta);
        roots[0] = (-b + ds) / (2.0 * a);
        roots[1] = (-b - ds) / (2.0 * a);
    } else if (fabs(a) < kRoundEps && fabs(b) > kRoundEps) {
        roots[0] = -c / b;
    }
}

// Roots outside [0, dt] dropped after the shift by MACH_EPS, the rest
// sorted; whether one is past MACH_EPS (dcollid3d.cpp:473-482).
__device__ __forceinline__ bool window_roots(double* roots, double dt) {
    for (int i = 0; i < 3; ++i) {
        roots[i] = roots[i] - kMachEps;
        if (roots[i] < 0 || roots[i] > dt) roots[i] = -1;
    }
    double t;
    if (roots[0] > roots[1]) { t = roots[0]; roots[0] = roots[1]; roots[1] = t; }
    if (roots[0] > roots[2]) { t = roots[0]; roots[0] = roots[2]; roots[2] = t; }
    if (roots[1] > roots[2]) { t = roots[1]; roots[1] = roots[2]; roots[2] = t; }
    return roots[0] > kMachEps || roots[1] > kMachEps || roots[2] > kMachEps;
}

// Whether a moving sub-test on these points can pass isCoplanar: false only
// when isCoplanar returns false.
__device__ __forceinline__ bool may_be_coplanar(const double (*xo4)[3], const double (*av4)[3], double dt) {
    double x[4][3], v[4][3];
    const Cubic q = coplanarity_cubic(xo4, av4, x, v);
    if (fabs(q.a) > kMachEps) return !no_root_in_window(q, dt);
    double roots[3] = {-1, -1, -1};
    low_degree_roots(q.b, q.c, q.d, roots);
    return window_roots(roots, dt);
}

// isCoplanar, dcollid3d.cpp:371-482: roots of the coplanarity cubic in
// [0, dt], shifted by -MACH_EPS and sorted; roots[3] holds dt. The functions
// are correctly rounded, as the reference's libm gives them (in fixed point
// they take less time than the FP64 library's). ncr counts the cubics with a
// root in the window.
static __device__ bool is_coplanar(const Cubic& q, double dt, double* roots, int* ncr) {
    if (!(fabs(q.a) > kMachEps)) {
        low_degree_roots(q.b, q.c, q.d, roots);
        return window_roots(roots, dt);
    }
    if (no_root_in_window(q, dt)) return false;
    const double inv_a = 1.0 / q.a;
    const double a = quotient(q.b, q.a, inv_a), b = quotient(q.c, q.a, inv_a), c = quotient(q.d, q.a, inv_a);
    double Q = (a * a - 3 * b) / 9;
    double R = (2 * a * a * a - 9 * a * b + 27 * c) / 54;
    double Q3 = Q * Q * Q;
    double R2 = R * R;
    if (R2 < Q3) {
        double Qsqrt = sqrt(Q);
        double z = R / sqrt(Q3);
        // A root that FP32 puts outside the window by 2^-9 of the roots'
        // scale is left out: z cut to FP32 moves theta by 2^-11 at most
        // (near |z| = 1), which moves a root by a third of that times 2 sqrt Q,
        // and the FP32 functions by 2^-20 of the scale.
        const float a32 = cut32(a), qs32 = cut32(Qsqrt), th32 = acosf(fminf(fmaxf(cut32(z), -1.f), 1.f));
        const float far = 0x1p-9f * (2.f * qs32 + fabsf(a32)) + 1e-30f, dt32 = (float)dt;
        const double theta = cr::acos(z);
#pragma unroll 1
        for (int i = 0; i < 3; ++i) {
            const float turn = i == 0 ? 0.f : i == 1 ? 6.2831853f : -6.2831853f;
            const float f32 = -2.f * qs32 * cosf((th32 + turn) * 0.33333333f) - a32 * 0.33333333f;
            if (f32 < -far || f32 > dt32 * 1.0001f + 1e-15f + far) continue;  // (roots[i] is -1)
            const double at = i == 0 ? theta / 3 : (i == 1 ? theta + 2 * kPi : theta - 2 * kPi) / 3;
            roots[i] = -2 * Qsqrt * cr::cos(at) - a / 3;
        }
    } else {
        double sgn = (R > 0) ? 1.0 : -1.0;
        double base = fabs(R) + sqrt(R2 - Q3);
        double A = -sgn * cr::pow(base, 1.0 / 3.0);
        double B = (fabs(A) < kRoundEps) ? 0.0 : Q / A;
        roots[0] = (A + B) - a / 3.0;
        if (fabs(A - B) < kRoundEps) roots[1] = roots[2] = -0.5 * (A + B) - a / 3.0;
    }
    const bool in = window_roots(roots, dt);
    *ncr += in;
    return in;
}

struct F3 {
    float x, y, z;
};
__device__ __forceinline__ F3 f3(float4 a) { return F3{a.x, a.y, a.z}; }
__device__ __forceinline__ F3 fsub(F3 a, F3 b) { return F3{a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ F3 fadd(F3 a, F3 b) { return F3{a.x + b.x, a.y + b.y, a.z + b.z}; }
__device__ __forceinline__ F3 fscale(F3 a, float s) { return F3{a.x * s, a.y * s, a.z * s}; }
__device__ __forceinline__ F3 cut_f3(const double* a) { return F3{cut32(a[0]), cut32(a[1]), cut32(a[2])}; }
__device__ __forceinline__ float fdot(F3 a, F3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ F3 fcross(F3 a, F3 b) {
    return F3{a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}
__device__ __forceinline__ float fnorm(F3 a) { return sqrtf(fdot(a, a)); }
__device__ __forceinline__ float fmaxabs(F3 a) { return fmaxf(fmaxf(fabsf(a.x), fabsf(a.y)), fabsf(a.z)); }
__device__ __forceinline__ float clamp01(float x) { return fminf(fmaxf(x, 0.f), 1.f); }

// Closest point of triangle (a, b, c) to p (Ericson 5.1.5), as an offset
// from a.
__device__ __forceinline__ F3 closest_on_tri(F3 ap, F3 ab, F3 ac) {
    float d1 = fdot(ab, ap), d2 = fdot(ac, ap);
    if (d1 <= 0.f && d2 <= 0.f) return F3{0.f, 0.f, 0.f};
    F3 bp = fsub(ap, ab);
    float d3 = fdot(ab, bp), d4 = fdot(ac, bp);
    if (d3 >= 0.f && d4 <= d3) return ab;
    float vc = d1 * d4 - d3 * d2;
    if (vc <= 0.f && d1 >= 0.f && d3 <= 0.f) return fscale(ab, d1 / (d1 - d3));
    F3 cp = fsub(ap, ac);
    float d5 = fdot(ab, cp), d6 = fdot(ac, cp);
    if (d6 >= 0.f && d5 <= d6) return ac;
    float vb = d5 * d2 - d1 * d6;
    if (vb <= 0.f && d2 >= 0.f && d6 <= 0.f) return fscale(ac, d2 / (d2 - d6));
    float va = d3 * d6 - d5 * d4;
    if (va <= 0.f && (d4 - d3) >= 0.f && (d5 - d6) >= 0.f) {
        float w = (d4 - d3) / ((d4 - d3) + (d5 - d6));
        return fadd(ab, fscale(fsub(ac, ab), w));
    }
    float den = 1.f / (va + vb + vc);
    return fadd(fscale(ab, vb * den), fscale(ac, vc * den));
}

// The least distance of two segments along the direction between their
// closest points, a lower bound of their distance whatever the rounding of
// that direction: segment d1 from r, segment d2 from 0. len: a bound on the
// lengths it was formed from. Negative infinity where they meet.
__device__ __forceinline__ float segment_gap(F3 d1, F3 d2, F3 r, float* len) {
    const float a = fdot(d1, d1), e = fdot(d2, d2), f = fdot(d2, r);
    float s = 0.f, t = 0.f;
    if (a > 0.f && e > 0.f) {
        const float cc = fdot(d1, r), b = fdot(d1, d2), den = a * e - b * b;
        s = den > 0.f ? clamp01((b * f - cc * e) / den) : 0.f;
        t = (b * s + f) / e;
        if (t < 0.f) {
            t = 0.f;
            s = clamp01(-cc / a);
        } else if (t > 1.f) {
            t = 1.f;
            s = clamp01((b - cc) / a);
        }
    } else if (a > 0.f) {
        s = clamp01(-fdot(d1, r) / a);
    } else if (e > 0.f) {
        t = clamp01(f / e);
    }
    // n from the second's closest point to the first's
    const F3 n = fsub(fadd(r, fscale(d1, s)), fscale(d2, t));
    const float nn = fnorm(n);
    const F3 q1 = fadd(r, d1);
    *len = fmaxf(fmaxf(fnorm(r), fnorm(q1)), fnorm(d2));
    if (!(nn > 0.f)) return -INFINITY;
    return (fminf(fdot(n, r), fdot(n, q1)) - fmaxf(0.f, fdot(n, d2))) / nn;
}

// The same of a point ap and the triangle (0, ab, ac).
__device__ __forceinline__ float triangle_gap(F3 ap, F3 ab, F3 ac, float* len) {
    const F3 n = fsub(ap, closest_on_tri(ap, ab, ac));
    const float nn = fnorm(n);
    *len = fmaxf(fmaxf(fnorm(ab), fnorm(ac)), fnorm(ap));
    if (!(nn > 0.f)) return -INFINITY;
    return (fdot(n, ap) - fmaxf(0.f, fmaxf(fdot(n, ab), fdot(n, ac)))) / nn;
}

// Whether a point that PointToTri (dcollid3d.cpp:778-922) calls a hit is
// certainly near the triangle, as every bound here assumes. Its coordinates
// come from det = |a|^2 |b|^2 - (a . b)^2 of two edges a, b: with u = 2^-53,
// det and the numerators round by at most 15 u |a|^2 |b|^2 (and |q| / |a| or
// |q| / |b| times that, q the point from the edges' corner), so a hit lies
// within r (2 |q| + 3 S) of where its coordinates put it, r = 15 u |a|^2
// |b|^2 / det and S the longest edge. The reach allows 2^-7 of the box's
// extents and 2^-10 of h, which holds for r <= 2^-12:
//  - extents up to 0.35 in all (|a| |b| <= 0.35^2), where the test's own cut
//    det >= 1000 MACH_EPS gives r < 2^-13; or
//  - an area |a x b| of at least 2^-16 of the extents squared: r < 2^-16.
// Of a thinner large triangle the test may call a point several lengths away
// a hit. ab, ac: its edges, up to err of them off at some time in the window;
// ext: its box's extents over the window, a bound on each edge.
__device__ __forceinline__ bool area_near(float area, float ext, float err) {
    return ext <= 0.35f || area - 4.0f * ext * err > ext * ext * 0x1p-16f;
}
__device__ __forceinline__ bool tri_near(F3 ab, F3 ac, float ext, float err) {
    return area_near(fnorm(fcross(ab, ac)), ext, err);
}
// err for points rounded to FP32 of magnitude up to M, whose velocities V
// differ by D at most and have magnitude up to Vm.
__device__ __forceinline__ float edge_error(float ext, float M, float D, float Vm, float dt32) {
    return (M + ext) * 0x1p-20f + dt32 * (D + Vm * 0x1p-18f) * 1.001f;
}

// Whether the static test at time t of a moving one certainly misses, in FP32
// on the points' positions x and velocities v from the first point's (cut
// from their FP64 differences, so that the error is relative to the
// elements' size S): a hit needs the elements within `reach` of each other
// (see sat_may_hit) and their gap along a direction is more. Positions here
// are within 2^-20 S of exact, the gap within 32 2^-24 of the lengths (at
// most 4 S), and the test's own positions within 2^-50 of the coordinates
// (slack: 2^-44 of them). An FP64 test is ~190 instructions of ~64 cycles;
// most of the times a pair's cubic gives are not near a hit. With the roots
// formed once, correctly rounded: sub-tests of a 257 x 257 sheet's step 1.51
// -> 0.87 ms, of 24 FP64 sheets 1.10 -> 0.55 ms.
template <bool EE>
__device__ __forceinline__ bool misses_at(const F3* x, const F3* v, float t, float slack, float h, float eps) {
    F3 P[4];
    float S = 0.f;
    for (int i = 1; i < 4; ++i) {
        P[i] = fadd(x[i], fscale(v[i], t));
        S = fmaxf(S, fmaxabs(x[i]) + t * fmaxabs(v[i]));
    }
    float len, gap, reach;
    if (EE) {
        // segments P0 P1 and P2 P3, origin P2
        const F3 d1 = P[1], d2 = fsub(P[3], P[2]), r = F3{-P[2].x, -P[2].y, -P[2].z};
        gap = segment_gap(d1, d2, r, &len);
        reach = h * 1.001f + S * 0x1p-16f;
    } else {
        gap = triangle_gap(P[3], P[1], P[2], &len);
        const float ext = (fmaxf(0.f, fmaxf(P[1].x, P[2].x)) - fminf(0.f, fminf(P[1].x, P[2].x))) +
                          (fmaxf(0.f, fmaxf(P[1].y, P[2].y)) - fminf(0.f, fminf(P[1].y, P[2].y))) +
                          (fmaxf(0.f, fmaxf(P[1].z, P[2].z)) - fminf(0.f, fminf(P[1].z, P[2].z)));
        reach = h * 1.001f + (ext * 1.001f + S * 0x1p-16f) * (8.0f * eps + 0x1p-10f) * 1.001f;
        if (!tri_near(P[1], P[2], ext * 1.001f + S * 0x1p-16f, S * 0x1p-18f)) return false;
    }
    return gap - (S * 0x1p-15f + 8.0f * slack) > reach;
}

// MovingPointToTri / MovingEdgeToEdge, dcollid3d.cpp:327-369: the static
// test with h = eps at each root of the cubic and at dt, first hit wins.
template <bool EE>
static __device__ bool moving_test(const NarrowCtx& c, CallState& st, const int* pts) {
    double xo4[4][3], av4[4][3];
    for (int q = 0; q < 4; ++q) {
        load3(c.xo, pts[q], xo4[q]);
        load3(c.av, pts[q], av4[q]);
    }
    double dt = c.p.dt;
    double roots[4] = {-1, -1, -1, dt};
    F3 x32[4], v32[4];
    float most = 0.f;  // of the coordinates
    {
        double x[4][3], v[4][3];
        const Cubic q = coplanarity_cubic(xo4, av4, x, v);
        if (!is_coplanar(q, dt, roots, &st.ncr)) return false;
        for (int i = 1; i < 4; ++i) {
            x32[i] = cut_f3(x[i]);
            v32[i] = cut_f3(v[i]);
            most = fmaxf(most, fmaxabs(x32[i]) + (float)dt * fmaxabs(v32[i]));
        }
        most += fmaxabs(cut_f3(xo4[0])) + (float)dt * fmaxabs(cut_f3(av4[0]));
    }
    for (int i = 0; i < 4; ++i) {
        if (roots[i] < 0) continue;
        if (misses_at<EE>(x32, v32, cut32(roots[i]), most * 0x1p-44f, (float)c.p.eps * 1.001f, (float)c.p.eps)) continue;
        double X[4][3];
        for (int q = 0; q < 4; ++q)
            for (int k = 0; k < 3; ++k) X[q][k] = xo4[q][k] + roots[i] * av4[q][k];
        bool hit = EE ? edge_to_edge(c, st, pts, X, c.p.eps) : point_to_tri(c, st, pts, X, c.p.eps);
        if (hit) return true;
    }
    return false;
}

template <bool EE>
__device__ __forceinline__ bool static_test(const NarrowCtx& c, CallState& st, const int* pts) {
    double X[4][3];
    for (int q = 0; q < 4; ++q) load3(c.xo, pts[q], X[q]);
    return EE ? edge_to_edge(c, st, pts, X, c.p.thickness) : point_to_tri(c, st, pts, X, c.p.thickness);
}

// tri_near of points a, b, c on the filters' FP32 data (v32 null: at rest).
// Only large triangles come here.
static __device__ bool points_near(const float4* p32, const float4* v32, int a, int b, int c, float ext,
                                   float dt32) {
    const F3 x0 = f3(p32[a]), x1 = f3(p32[b]), x2 = f3(p32[c]);
    float D = 0.f, Vm = 0.f;
    if (v32) {
        const F3 v0 = f3(v32[a]), v1 = f3(v32[b]), v2 = f3(v32[c]);
        D = fmaxf(fnorm(fsub(v1, v0)), fnorm(fsub(v2, v0)));
        Vm = fmaxf(fmaxabs(v0), fmaxf(fmaxabs(v1), fmaxabs(v2)));
    }
    const float M = fmaxf(fmaxabs(x0), fmaxf(fmaxabs(x1), fmaxabs(x2)));
    return tri_near(fsub(x1, x0), fsub(x2, x0), ext, edge_error(ext, M, D, Vm, dt32));
}

// Mixed-precision filter. Every position an FP64 test evaluates lies in its
// point's box (x_old and x_old + dt*avgVel, both rounded outward to FP32):
// the roots are in [0, dt] and x_old + t*avgVel rounds monotonically in t.
//  - Edge-edge (dcollid3d.cpp:643-776): the closest points v1, v2 lie on the
//    two segments, so dist >= the segments' distance >= the gap between
//    their boxes; a hit needs dist <= h.
//  - Point-triangle (dcollid3d.cpp:778-922): a hit needs the point within h
//    of the plane and barycentric coordinates in [-eps, 1+eps], so its
//    projection is within 4*eps*diameter of the triangle. The computed
//    coordinates carry a solve error; where tri_near holds, the reach padded
//    by (8*eps + 2^-10) times the triangle's box extent covers it, and no
//    other triangle is filtered.
// When the padded boxes do not overlap, the FP64 test returns false and is
// skipped; every other sub-test runs unchanged, so the results are the plain
// FP64 path's.
__device__ __forceinline__ bool mixed_may_hit(const NarrowCtx& c, const int* pts, bool ee, float* ext_out,
                                              float* extb_out) {
    float4 l0 = c.pbox_lo[pts[0]], h0 = c.pbox_hi[pts[0]];
    float4 l1 = c.pbox_lo[pts[1]], h1 = c.pbox_hi[pts[1]];
    float4 l2 = c.pbox_lo[pts[2]], h2 = c.pbox_hi[pts[2]];
    float4 l3 = c.pbox_lo[pts[3]], h3 = c.pbox_hi[pts[3]];
    float alo[3], ahi[3], blo[3], bhi[3];
    if (ee) {
        alo[0] = fminf(l0.x, l1.x); alo[1] = fminf(l0.y, l1.y); alo[2] = fminf(l0.z, l1.z);
        ahi[0] = fmaxf(h0.x, h1.x); ahi[1] = fmaxf(h0.y, h1.y); ahi[2] = fmaxf(h0.z, h1.z);
        blo[0] = fminf(l2.x, l3.x); blo[1] = fminf(l2.y, l3.y); blo[2] = fminf(l2.z, l3.z);
        bhi[0] = fmaxf(h2.x, h3.x); bhi[1] = fmaxf(h2.y, h3.y); bhi[2] = fmaxf(h2.z, h3.z);
    } else {
        alo[0] = fminf(fminf(l0.x, l1.x), l2.x); alo[1] = fminf(fminf(l0.y, l1.y), l2.y);
        alo[2] = fminf(fminf(l0.z, l1.z), l2.z);
        ahi[0] = fmaxf(fmaxf(h0.x, h1.x), h2.x); ahi[1] = fmaxf(fmaxf(h0.y, h1.y), h2.y);
        ahi[2] = fmaxf(fmaxf(h0.z, h1.z), h2.z);
        blo[0] = l3.x; blo[1] = l3.y; blo[2] = l3.z;
        bhi[0] = h3.x; bhi[1] = h3.y; bhi[2] = h3.z;
    }
    float ext = __fadd_ru(__fadd_ru(__fsub_ru(ahi[0], alo[0]), __fsub_ru(ahi[1], alo[1])), __fsub_ru(ahi[2], alo[2]));
    float pad;
    float extb = 0.f;
    if (ee) {
        extb = __fadd_ru(__fadd_ru(__fsub_ru(bhi[0], blo[0]), __fsub_ru(bhi[1], blo[1])), __fsub_ru(bhi[2], blo[2]));
        pad = __fadd_ru(c.hpad, __fmul_ru(__fadd_ru(ext, extb), 0x1p-20f));
    } else {
        pad = __fadd_ru(c.hpad, __fmul_ru(ext, __fadd_ru(__fmul_ru(8.0f, c.epad), 0x1p-10f)));
    }
    *ext_out = ext;
    *extb_out = extb;
    for (int d = 0; d < 3; ++d) {
        if (__fsub_rd(alo[d], pad) > bhi[d]) return false;
        if (__fadd_ru(ahi[d], pad) < blo[d]) return false;
    }
    return true;
}

// Second stage of the mixed-precision filter: a lower bound on the distance
// between the point and the triangle (PT) or between the two segments (EE)
// over the pass's time window, from FP32 copies of the points.
//
// Any direction n gives a lower bound: the gap between the projections of
// the two point sets onto n, divided by |n| (both sets are convex hulls of
// their points, so their projections are spanned by the points'). The
// direction is taken from FP32 closest points (Ericson, Real-Time Collision
// Detection, 2005, 5.1.5 ClosestPtPointTriangle and 5.1.9
// ClosestPtSegmentSegment); how well it is chosen affects only how often
// the bound rejects, never whether the bound holds. The bound is lowered by
//  - the rounding of its own FP32 evaluation, at most 13*u*L for dot
//    products over difference vectors of length <= L (u = 2^-24), and of the
//    points to FP32, at most 2*sqrt(3)*u*M for coordinates of magnitude <= M:
//    together below 32*u*(L + M);
//  - on moving passes, the distance the sets can close within [0, dt]: the
//    distance between two sets changes by at most the largest displacement
//    of a point of each relative to a common reference (a segment's or a
//    triangle's points move by at most the largest displacement of its
//    corners), dt*(D1 + D2) with D the largest |v - v_ref| of each side.
// A hit needs the distance within reach: for PT the plane distance <= h and
// barycentric coordinates >= -eps - dw (dw <= 2^-10, the solve error the
// box stage allows too; see tri_near) put the point within h + 6*(eps +
// dw)*diam of the triangle (padded to 8*(eps + 2^-10)*ext); for EE the clamped closest
// points within h are points of the segments, so the segments are within
// h + 2^-20*ext. Sub-tests whose bound exceeds the reach return false in
// FP64 too and are skipped.
// On given points (rounded to FP32, or cut to it by cut32, which is within
// the same bound) and velocities; ext, extb: the extents of the elements'
// boxes over the window.
// (The caller has seen to tri_near.)
template <bool MOVING, bool EE>
__device__ __forceinline__ bool gap_may_hit(const F3* X, const F3* V, float ext, float extb, float hpad, float epad,
                                            float dt32) {
    float M = fmaxf(fmaxf(fmaxabs(X[0]), fmaxabs(X[1])), fmaxf(fmaxabs(X[2]), fmaxabs(X[3])));
    float lb, L, reach;
    if (!EE) {
        // triangle X0 X1 X2, point X3; origin X0
        lb = triangle_gap(fsub(X[3], X[0]), fsub(X[1], X[0]), fsub(X[2], X[0]), &L);
        reach = __fadd_ru(hpad, __fmul_ru(ext, __fmul_ru(8.0f, __fadd_ru(epad, 0x1p-10f))));
    } else {
        // segments S1 = X0 X1, S2 = X2 X3; origin X2
        lb = segment_gap(fsub(X[1], X[0]), fsub(X[3], X[2]), fsub(X[0], X[2]), &L);
        reach = __fadd_ru(hpad, __fmul_ru(__fadd_ru(ext, extb), 0x1p-20f));
    }
    float err = __fmul_ru(32.0f * 0x1p-24f, __fadd_ru(L, M));
    float bound = __fsub_rd(lb, err);
    if (MOVING) {
        // reference velocity: the first point's
        float D1, D2;
        if (!EE) {
            D1 = fmaxf(fmaxf(fnorm(fsub(V[1], V[0])), fnorm(fsub(V[2], V[0]))), 0.f);
            D2 = fnorm(fsub(V[3], V[0]));
        } else {
            D1 = fnorm(fsub(V[1], V[0]));
            D2 = fmaxf(fnorm(fsub(V[2], V[0])), fnorm(fsub(V[3], V[0])));
        }
        float Vm = fmaxf(fmaxf(fmaxabs(V[0]), fmaxabs(V[1])), fmaxf(fmaxabs(V[2]), fmaxabs(V[3])));
        // FP32 rounding of the velocities and of the sums above
        float dv = __fadd_ru(__fmul_ru(__fadd_ru(D1, D2), 1.0f + 0x1p-16f), __fmul_ru(Vm, 32.0f * 0x1p-24f));
        bound = __fsub_rd(bound, __fmul_ru(dt32, dv));
    }
    return !(bound > reach);
}

// h as the filters take it: rounded up, with 2^-10 of it for the error of a
// hit's coordinates where h is much larger than the triangle (tri_near).
__device__ __forceinline__ float filter_reach(double h) { return cut32_up(h) * (1.0f + 0x1p-10f); }

// The extents of n points' box over the window, for gap_may_hit.
template <bool MOVING>
__device__ __forceinline__ float swept_extent(const F3* X, const F3* V, int n, float dt) {
    F3 lo = X[0], hi = X[0];
    auto take = [&](F3 p) {
        lo = F3{fminf(lo.x, p.x), fminf(lo.y, p.y), fminf(lo.z, p.z)};
        hi = F3{fmaxf(hi.x, p.x), fmaxf(hi.y, p.y), fmaxf(hi.z, p.z)};
    };
    for (int i = 0; i < n; ++i) {
        take(X[i]);
        if (MOVING) take(fadd(X[i], fscale(V[i], dt)));
    }
    const F3 d = fsub(hi, lo);
    return (d.x + d.y + d.z) * 1.001f;
}

// The gap bound of one sub-test on its points cut to FP32 (plain passes).
template <bool MOVING>
__device__ __forceinline__ bool plain_may_hit(const double4_32a* __restrict__ xo, const double4_32a* __restrict__ av,
                                              const int* pts, bool ee, const Params& prm) {
    const float dt32 = cut32_up(prm.dt);
    F3 X[4], V[4];
    for (int q = 0; q < 4; ++q) {
        double x[3];
        load3(xo, pts[q], x);
        X[q] = cut_f3(x);
        if (MOVING) {
            load3(av, pts[q], x);
            V[q] = cut_f3(x);
        }
    }
    float hpad = filter_reach(MOVING ? prm.eps : prm.thickness), epad = cut32_up(prm.eps);
    const float most = fmaxf(fmaxf(fmaxabs(X[0]), fmaxabs(X[1])), fmaxf(fmaxabs(X[2]), fmaxabs(X[3])));
    if (most * 0x1p-13f > fmaxabs(fsub(X[1], X[0]))) {
        // far from the origin for its size: positions from the first
        // point's, and the tests' own rounding on the reach
        double x0[3], x[3];
        load3(xo, pts[0], x0);
        X[0] = F3{0.f, 0.f, 0.f};
        for (int q = 1; q < 4; ++q) {
            load3(xo, pts[q], x);
            for (int k = 0; k < 3; ++k) x[k] -= x0[k];
            X[q] = cut_f3(x);
        }
        hpad += most * 0x1p-44f;
    }
    const int na = ee ? 2 : 3;
    const float ext = swept_extent<MOVING>(X, V, na, dt32);
    const float extb = swept_extent<MOVING>(X + na, V + na, 4 - na, dt32);
    if (ee) return gap_may_hit<MOVING, true>(X, V, ext, extb, hpad, epad, dt32);
    if (ext > 0.35f) {
        float M = 0.f, D = 0.f, Vm = 0.f;
        for (int q = 0; q < 3; ++q) {
            M = fmaxf(M, fmaxabs(X[q]));
            if (MOVING) Vm = fmaxf(Vm, fmaxabs(V[q])), D = fmaxf(D, fnorm(fsub(V[q], V[0])));
        }
        if (!tri_near(fsub(X[1], X[0]), fsub(X[2], X[0]), ext, edge_error(ext, M, D, Vm, dt32))) return true;
    }
    return gap_may_hit<MOVING, false>(X, V, ext, extb, hpad, epad, dt32);
}

template <bool MOVING, bool EE>
__device__ __forceinline__ bool sat_may_hit(const NarrowCtx& c, const int* pts, float ext, float extb) {
    F3 X[4], V[4];
    for (int q = 0; q < 4; ++q) X[q] = f3(c.p32[pts[q]]);
    if (MOVING)
        for (int q = 0; q < 4; ++q) V[q] = f3(c.v32[pts[q]]);
    return gap_may_hit<MOVING, EE>(X, V, ext, extb, c.hpad, c.epad, c.dt32);
}

// Element-pair stage of the mixed-precision filter: one lower bound on the
// distance between the two elements (as point sets) over the pass's time
// window. Every sub-test of the pair involves a point or an edge of each
// element, so its distance is at least this one, and when the bound exceeds
// the largest reach of the pair's sub-tests none of them can hit. The bound
// is the separating-axis gap (as in sat_may_hit, with the same rounding and
// motion allowances) maximised over a few axes: each triangle's normal and
// its three in-plane edge normals (for two disjoint coplanar triangles one of
// those separates them), for two segments their common normal and the
// in-plane normals of each, and the line between the centroids.
// Gap between the projections of two point sets (3 points each) onto ax,
// divided by |ax| (an): a lower bound on their distance (-1 for a zero axis).
__device__ __forceinline__ float axis_gap(F3 ax, const F3* R, float& an) {
    an = fnorm(ax);
    if (!(an > 0.f)) return -1.f;
    float amin = fdot(ax, R[0]), amax = amin, bmin = fdot(ax, R[3]), bmax = bmin;
#pragma unroll
    for (int q = 1; q < 3; ++q) {
        float ta = fdot(ax, R[q]), tb = fdot(ax, R[3 + q]);
        amin = fminf(amin, ta);
        amax = fmaxf(amax, ta);
        bmin = fminf(bmin, tb);
        bmax = fmaxf(bmax, tb);
    }
    return fmaxf(bmin - amax, amin - bmax) / an;
}

// The pair's decision from the gap lb: ia, ib its points (a segment's last
// one twice), L and M bounds of their distances and coordinates, areaA and
// areaB the lengths of the triangles' normals. kPairThin: it holds a triangle
// outside tri_near, whose point-triangle sub-tests no bound rules out.
enum PairBound { kPairFar = 0, kPairNear = 1, kPairThin = 2 };
template <bool MOVING>
__device__ __forceinline__ int pair_bound(const NarrowCtx& c, const int* ia, int na, const int* ib, int nb, float lb,
                                          float L, float M, float areaA, float areaB) {
    // the largest reach of the pair's sub-tests, with the boxes' extents
    float extA, extB;
    {
        float4 l = c.pbox_lo[ia[0]], h = c.pbox_hi[ia[0]];
        float lo[3] = {l.x, l.y, l.z}, hi[3] = {h.x, h.y, h.z};
#pragma unroll
        for (int q = 1; q < 3; ++q) {
            l = c.pbox_lo[ia[q]];
            h = c.pbox_hi[ia[q]];
            lo[0] = fminf(lo[0], l.x); lo[1] = fminf(lo[1], l.y); lo[2] = fminf(lo[2], l.z);
            hi[0] = fmaxf(hi[0], h.x); hi[1] = fmaxf(hi[1], h.y); hi[2] = fmaxf(hi[2], h.z);
        }
        extA = __fadd_ru(__fadd_ru(__fsub_ru(hi[0], lo[0]), __fsub_ru(hi[1], lo[1])), __fsub_ru(hi[2], lo[2]));
        l = c.pbox_lo[ib[0]];
        h = c.pbox_hi[ib[0]];
        float lo2[3] = {l.x, l.y, l.z}, hi2[3] = {h.x, h.y, h.z};
#pragma unroll
        for (int q = 1; q < 3; ++q) {
            l = c.pbox_lo[ib[q]];
            h = c.pbox_hi[ib[q]];
            lo2[0] = fminf(lo2[0], l.x); lo2[1] = fminf(lo2[1], l.y); lo2[2] = fminf(lo2[2], l.z);
            hi2[0] = fmaxf(hi2[0], h.x); hi2[1] = fmaxf(hi2[1], h.y); hi2[2] = fmaxf(hi2[2], h.z);
        }
        extB = __fadd_ru(__fadd_ru(__fsub_ru(hi2[0], lo2[0]), __fsub_ru(hi2[1], lo2[1])), __fsub_ru(hi2[2], lo2[2]));
    }
    float ext_tri = fmaxf(na == 3 ? extA : 0.f, nb == 3 ? extB : 0.f);
    float reach_pt = __fmul_ru(ext_tri, __fmul_ru(8.0f, __fadd_ru(c.epad, 0x1p-10f)));
    float reach_ee = __fmul_ru(__fadd_ru(extA, extB), 0x1p-20f);
    float reach = __fadd_ru(c.hpad, fmaxf(reach_pt, reach_ee));
    float err = __fmul_ru(32.0f * 0x1p-24f, __fadd_ru(L, M));
    float bound = __fsub_rd(lb, err);
    float DA = 0.f, DB = 0.f, Vm = 0.f;  // (DB from A's first point)
    if (MOVING) {
        F3 v0 = f3(c.v32[ia[0]]);
        Vm = fmaxabs(v0);
#pragma unroll
        for (int q = 1; q < 3; ++q) {
            F3 v = f3(c.v32[ia[q]]);
            DA = fmaxf(DA, fnorm(fsub(v, v0)));
            Vm = fmaxf(Vm, fmaxabs(v));
        }
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            F3 v = f3(c.v32[ib[q]]);
            DB = fmaxf(DB, fnorm(fsub(v, v0)));
            Vm = fmaxf(Vm, fmaxabs(v));
        }
        float dv = __fadd_ru(__fmul_ru(__fadd_ru(DA, DB), 1.0f + 0x1p-16f), __fmul_ru(Vm, 32.0f * 0x1p-24f));
        bound = __fsub_rd(bound, __fmul_ru(c.dt32, dv));
    }
    if (ext_tri > 0.35f) {
        if (na == 3 && extA > 0.35f && !area_near(areaA, extA, edge_error(extA, M, DA, Vm, c.dt32))) return kPairThin;
        if (nb == 3 && extB > 0.35f && !area_near(areaB, extB, edge_error(extB, M, 2.0f * DB, Vm, c.dt32)))
            return kPairThin;
    }
    return bound > reach ? kPairFar : kPairNear;
}

template <bool MOVING>
__device__ __forceinline__ int pair_may_hit(const NarrowCtx& c, const int* A, int na, const int* B, int nb) {
    // points relative to A's first; a segment's third point repeats its
    // second (the same convex hull, so the same projections)
    const int ia[3] = {A[0], A[1], na == 3 ? A[2] : A[1]};
    const int ib[3] = {B[0], B[1], nb == 3 ? B[2] : B[1]};
    F3 R[6];
    const F3 X0 = f3(c.p32[ia[0]]);
    float M = fmaxabs(X0), L = 0.f;
#pragma unroll
    for (int q = 0; q < 6; ++q) {
        F3 x = q < 3 ? f3(c.p32[ia[q]]) : f3(c.p32[ib[q - 3]]);
        M = fmaxf(M, fmaxabs(x));
        R[q] = fsub(x, X0);
        L = fmaxf(L, fnorm(R[q]));
    }
    float lb = -1.f, an, area[2];
    {
        F3 cA = fscale(fadd(fadd(R[0], R[1]), R[2]), 1.f / 3.f);
        F3 cB = fscale(fadd(fadd(R[3], R[4]), R[5]), 1.f / 3.f);
        lb = fmaxf(lb, axis_gap(fsub(cB, cA), R, an));
    }
#pragma unroll
    for (int side = 0; side < 2; ++side) {
        const F3* P = R + 3 * side;
        F3 e0 = fsub(P[1], P[0]), e1 = fsub(P[2], P[1]), e2 = fsub(P[0], P[2]);
        F3 nrm = fcross(e0, fsub(P[2], P[0]));  // zero for a segment: skipped
        lb = fmaxf(lb, axis_gap(nrm, R, area[side]));
        lb = fmaxf(lb, axis_gap(fcross(nrm, e0), R, an));
        lb = fmaxf(lb, axis_gap(fcross(nrm, e1), R, an));
        lb = fmaxf(lb, axis_gap(fcross(nrm, e2), R, an));
    }
    {
        F3 d1 = fsub(R[1], R[0]), d2 = fsub(R[4], R[3]);
        F3 nrm = fcross(d1, d2);
        lb = fmaxf(lb, axis_gap(nrm, R, an));
        lb = fmaxf(lb, axis_gap(fcross(nrm, d1), R, an));
        lb = fmaxf(lb, axis_gap(fcross(nrm, d2), R, an));
    }
    return pair_bound<MOVING>(c, ia, na, ib, nb, lb, L, M, area[0], area[1]);
}

template <bool MOVING, bool EE>
__device__ __forceinline__ bool sub_test(const NarrowCtx& c, CallState& st, const int* pts) {
    if (c.pbox_lo) {
        float ext, extb;
        const bool out = !mixed_may_hit(c, pts, EE, &ext, &extb) || !sat_may_hit<MOVING, EE>(c, pts, ext, extb);
        if (out && (EE || ext <= 0.35f || points_near(c.p32, MOVING ? c.v32 : nullptr, pts[0], pts[1], pts[2], ext, c.dt32)))
            return false;
    }
    st.nsub++;
    if (MOVING) return moving_test<EE>(c, st, pts);
    return static_test<EE>(c, st, pts);
}

// ------------------------------------------------------ element-pair tests
// TriToTri (dcollid3d.cpp:570-627) and MovingTriToTri (dcollid3d.cpp:274-325).
// A = found element, B = query element.
template <bool MOVING>
static __device__ bool tri_to_tri(const NarrowCtx& c, CallState& st, const int* A, const int* B) {
    int pts[4];
    bool status = false;
    for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j)
            if (A[i] == B[j]) return false;
    int sub = 0;
    for (int k = 0; k < 2; ++k)
        for (int i = 0; i < 3; ++i, ++sub) {
            // proximity tests B's triangle against A's points first; CCD the reverse
            const int* tri = MOVING ? ((k == 0) ? A : B) : ((k == 0) ? B : A);
            const int* pt = MOVING ? ((k == 0) ? B : A) : ((k == 0) ? A : B);
            for (int j = 0; j < 3; ++j) pts[j] = tri[j];
            pts[3] = pt[i];
            st.sub = sub;
            if (sub_test<MOVING, false>(c, st, pts)) status = true;
            if (MOVING && status && c.zone) create_imp_zone(c, st, pts);
        }
    for (int i = 0; i < 3; ++i) {
        pts[0] = A[i];
        pts[1] = A[(i + 1) % 3];
        for (int j = 0; j < 3; ++j, ++sub) {
            pts[2] = B[j];
            pts[3] = B[(j + 1) % 3];
            st.sub = sub;
            if (sub_test<MOVING, true>(c, st, pts)) status = true;
            if (MOVING && status && c.zone) create_imp_zone(c, st, pts);
        }
    }
    return status;
}

// TriToBond (dcollid3d.cpp:485-533) and MovingTriToBond (dcollid3d.cpp:203-244).
template <bool MOVING>
static __device__ bool tri_to_bond(const NarrowCtx& c, CallState& st, const int* T, const int* Bd) {
    int pts[4];
    bool status = false;
    for (int i = 0; i < 3; ++i)
        if (T[i] == Bd[0] || T[i] == Bd[1]) return false;
    for (int i = 0; i < 3; ++i) pts[i] = T[i];
    for (int e = 0; e < 2; ++e) {
        pts[3] = Bd[e];
        st.sub = e;
        if (sub_test<MOVING, false>(c, st, pts)) status = true;
        if (MOVING && status && c.zone) create_imp_zone(c, st, pts);
    }
    pts[2] = Bd[0];
    pts[3] = Bd[1];
    for (int i = 0; i < 3; ++i) {
        pts[0] = T[i];
        pts[1] = T[(i + 1) % 3];
        st.sub = 2 + i;
        if (sub_test<MOVING, true>(c, st, pts)) status = true;
        if (MOVING && status && c.zone) create_imp_zone(c, st, pts);
    }
    return status;
}

// BondToBond (dcollid3d.cpp:535-568) and MovingBondToBond (dcollid3d.cpp:246-272).
template <bool MOVING>
static __device__ bool bond_to_bond(const NarrowCtx& c, CallState& st, const int* A, const int* B) {
    int pts[4] = {A[0], A[1], B[0], B[1]};
    for (int i = 0; i < 4; ++i)
        for (int j = i + 1; j < 4; ++j)
            if (pts[i] == pts[j]) return false;
    st.sub = 0;
    bool status = sub_test<MOVING, true>(c, st, pts);
    if (MOVING && status && c.zone) create_imp_zone(c, st, pts);
    return status;
}

}  // namespace ccg
