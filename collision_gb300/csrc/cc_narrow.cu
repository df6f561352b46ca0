// Narrow-phase pass over the candidate pairs: one thread per pair.
//
// The reference visits each overlapping pair once, as (a = the leaf found
// later in its tree's inorder, b = the query leaf), in (b, a) inorder
// (AABB.cpp:254-343), and dispatches it by element type (isProximity /
// isCollision, dcollid.cpp:753-836). Here every pair is oriented by the
// leaf ranks of the reference tree, and each impulse contribution carries the
// key (rank b, rank a, sub-test) so the per-point sums can be formed later in
// exactly the reference's order.
#include "cc_launch.h"
#include "cc_narrow.cuh"
#include "cc_point_box.cuh"

namespace ccg {

namespace {

template <bool MOVING>
__global__ void __launch_bounds__(128) k_narrow(NarrowArgs a, int max_pairs) {
    NarrowCtx c;
    c.xo = a.xo; c.av = a.av; c.fixed = a.fixed; c.ev = a.ev; c.esurf = a.esurf; c.erigid = a.erigid;
    c.vbody = a.vbody; c.body_mass = a.body_mass; c.body_slot0 = a.body_slot0;
    c.rank = a.rank;
    c.contrib = a.contrib; c.contrib_cap = a.contrib_cap; c.ctr = a.ctr; c.urec = a.urec;
    c.urec_cap = a.urec_cap;
    c.rec = a.rec; c.rec_cap = a.rec_cap;
    c.pbox_lo = a.pbox_lo; c.pbox_hi = a.pbox_hi; c.p32 = a.p32; c.v32 = a.v32;
    c.check = a.check;
    int np = a.ctr->npairs;
    if (np > max_pairs) np = max_pairs;
    // counters summed per thread, added once per warp at the end
    int t_visits = 0, t_sub = 0, t_hits = 0, t_cr = 0, t_contacts = 0;
    for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < np; idx += gridDim.x * blockDim.x) {
        int2 pr = a.pairs[idx];
        if (!MOVING && a.static_only && !(pr.y & kPairStatic)) continue;
        pr.y &= kPairIdMask;
        int sc = a.escene[pr.x];
        const SceneRun run = a.run[sc];
        c.p = a.scenes[sc].p;
        c.zone = run.mode == kSceneZone && !a.check;
        c.pass = run.pass;
        // h of the sub-tests (thickness for proximity, eps for CCD) and the
        // barycentric tolerance eps, rounded up to FP32
        c.hpad = filter_reach(MOVING ? c.p.eps : c.p.thickness);
        c.epad = cut32_up(c.p.eps);
        c.dt32 = cut32_up(c.p.dt);
        int ri = c.rank ? c.rank[pr.x] : pr.x, rj = c.rank ? c.rank[pr.y] : pr.y;
        int ea = ri > rj ? pr.x : pr.y;  // found leaf
        int eb = ri > rj ? pr.y : pr.x;  // query leaf
        int ra = ri > rj ? ri : rj, rb = ri > rj ? rj : ri;
        bool ta = c.ev[3 * ea + 2] >= 0, tb = c.ev[3 * eb + 2] >= 0;
        int kind = (ta && tb) ? 0 : (!ta && !tb) ? 2 : 1;
        if (kind == 0 && c.esurf[ea] == c.esurf[eb] && c.erigid[ea]) continue;  // dcollid.cpp:762-763, 805-806
        // tri-bond pairs are always handed over as (tri, bond)
        int e1 = (kind == 1 && !ta) ? eb : ea;
        int e2 = (kind == 1 && !ta) ? ea : eb;
        const int* P1 = c.ev + 3 * e1;
        const int* P2 = c.ev + 3 * e2;
        CallState st;
        st.keybase = ((unsigned long long)rb << 26) | ((unsigned long long)ra << 4);
        int n1 = (P1[2] >= 0) ? 3 : 2, n2 = (P2[2] >= 0) ? 3 : 2;
        st.np = n1 + n2;
        for (int i = 0; i < 6; ++i) { st.dcount[i] = 0; st.plist[i] = -1; }
        for (int i = 0; i < n1; ++i) st.plist[i] = P1[i];
        for (int i = 0; i < n2; ++i) st.plist[n1 + i] = P2[i];
        st.sub = 0;
        st.nsub = 0;
        st.ncr = 0;
        st.ncontacts = 0;
        int A[3] = {P1[0], P1[1], n1 == 3 ? P1[2] : -1};
        int B[3] = {P2[0], P2[1], n2 == 3 ? P2[2] : -1};
        bool status;
        if (c.pbox_lo && !pair_may_hit<MOVING>(c, A, n1, B, n2))
            status = false;  // no sub-test of the pair can hit
        else if (kind == 0)
            status = tri_to_tri<MOVING>(c, st, A, B);
        else if (kind == 1)
            status = tri_to_bond<MOVING>(c, st, A, B);
        else
            status = bond_to_bond<MOVING>(c, st, A, B);
        t_visits++;
        t_sub += st.nsub;
        t_cr += st.ncr;
        t_contacts += st.ncontacts;
        if (status) {
            t_hits++;
            atomicAdd(&a.run[sc].hits, 1);
            for (int q = 0; q < 3; ++q) {
                if (A[q] >= 0) stamp_point(a.ps, A[q]);
                if (B[q] >= 0) stamp_point(a.ps, B[q]);
            }
        }
        if (c.rec) {
            int slot = atomicAdd(&c.ctr->nrec, 1);
            if (slot < c.rec_cap) {
                VisitRec& r = c.rec[slot];
                r.pass = c.pass; r.kind = kind; r.a = e1; r.b = e2; r.status = status ? 1 : 0;
                for (int i = 0; i < 6; ++i) r.dcount[i] = st.dcount[i];
                r.rank_b = rb; r.rank_a = ra;
            } else {
                atomicOr(&c.ctr->err, kErrRecordOverflow);
            }
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        t_visits += __shfl_xor_sync(0xffffffffu, t_visits, o);
        t_sub += __shfl_xor_sync(0xffffffffu, t_sub, o);
        t_hits += __shfl_xor_sync(0xffffffffu, t_hits, o);
        t_cr += __shfl_xor_sync(0xffffffffu, t_cr, o);
        t_contacts += __shfl_xor_sync(0xffffffffu, t_contacts, o);
    }
    if ((threadIdx.x & 31) == 0) {
        if (t_visits) atomicAdd(&c.ctr->nvisits, t_visits);
        if (t_sub) atomicAdd(&c.ctr->nsub, t_sub);
        if (t_hits) atomicAdd(&c.ctr->nhit_pairs, t_hits);
        if (t_cr) atomicAdd(&c.ctr->ncr, t_cr);
        if (t_contacts) atomicAdd(&c.ctr->ncontacts, t_contacts);
    }
}

// The sub-tests of an element pair in the order of tri_to_tri /
// tri_to_bond / bond_to_bond (A the found element, B the query element):
// f(sub, pts, ee) for each.
template <bool MOVING, class F>
__device__ __forceinline__ void for_each_subtest(int kind, const int* A, const int* B, F&& f) {
    int pts[4];
    if (kind == 0) {
        int sub = 0;
        for (int k = 0; k < 2; ++k)
            for (int i = 0; i < 3; ++i, ++sub) {
                // proximity tests B's triangle against A's points first; CCD the reverse
                const int* tri = MOVING ? ((k == 0) ? A : B) : ((k == 0) ? B : A);
                const int* pt = MOVING ? ((k == 0) ? B : A) : ((k == 0) ? A : B);
                pts[0] = tri[0]; pts[1] = tri[1]; pts[2] = tri[2]; pts[3] = pt[i];
                f(sub, pts, false);
            }
        for (int i = 0; i < 3; ++i)
            for (int j = 0; j < 3; ++j, ++sub) {
                pts[0] = A[i]; pts[1] = A[(i + 1) % 3]; pts[2] = B[j]; pts[3] = B[(j + 1) % 3];
                f(sub, pts, true);
            }
    } else if (kind == 1) {
        pts[0] = A[0]; pts[1] = A[1]; pts[2] = A[2];
        pts[3] = B[0];
        f(0, pts, false);
        pts[3] = B[1];
        f(1, pts, false);
        pts[2] = B[0];
        pts[3] = B[1];
        for (int i = 0; i < 3; ++i) {
            pts[0] = A[i];
            pts[1] = A[(i + 1) % 3];
            f(2 + i, pts, true);
        }
    } else {
        pts[0] = A[0]; pts[1] = A[1]; pts[2] = B[0]; pts[3] = B[1];
        f(0, pts, true);
    }
}

// A candidate pair as k_narrow orients it: kind (0 tri-tri, 1 tri-bond,
// 2 bond-bond), the points of the element handed over first (A) and second
// (B), and the visiting-order key base (rank of the query leaf, rank of the
// found leaf). False for a same-rigid-surface pair, which is not visited.
struct OrientedPair {
    int kind, n1, n2;
    int A[3], B[3];
    unsigned long long keybase;
};
__device__ __forceinline__ bool orient_pair(const NarrowArgs& a, int2 pr, OrientedPair& o) {
    int ri = a.rank ? a.rank[pr.x] : pr.x, rj = a.rank ? a.rank[pr.y] : pr.y;
    int ea = ri > rj ? pr.x : pr.y;  // found leaf
    int eb = ri > rj ? pr.y : pr.x;  // query leaf
    int ra = ri > rj ? ri : rj, rb = ri > rj ? rj : ri;
    bool ta = a.ev[3 * ea + 2] >= 0, tb = a.ev[3 * eb + 2] >= 0;
    o.kind = (ta && tb) ? 0 : (!ta && !tb) ? 2 : 1;
    if (o.kind == 0 && a.esurf[ea] == a.esurf[eb] && a.erigid[ea]) return false;  // dcollid.cpp:762-763, 805-806
    int e1 = (o.kind == 1 && !ta) ? eb : ea;  // tri-bond pairs are handed over as (tri, bond)
    int e2 = (o.kind == 1 && !ta) ? ea : eb;
    for (int i = 0; i < 3; ++i) {
        o.A[i] = a.ev[3 * e1 + i];
        o.B[i] = a.ev[3 * e2 + i];
    }
    o.n1 = o.A[2] >= 0 ? 3 : 2;
    o.n2 = o.B[2] >= 0 ? 3 : 2;
    o.keybase = ((unsigned long long)rb << 26) | ((unsigned long long)ra << 4);
    return true;
}

// The points of sub-test `sub` of a pair (for_each_subtest's numbering) and
// whether it is edge-edge; false past the pair's last.
template <bool MOVING>
__device__ __forceinline__ bool pair_subtest(const OrientedPair& o, int sub, int* pts, bool& ee) {
    const int npt = o.kind == 0 ? 6 : o.kind == 1 ? 2 : 0;
    const int n = o.kind == 0 ? 15 : o.kind == 1 ? 5 : 1;
    ee = sub >= npt;
    if (sub >= n) return false;
    if (!ee) {
        // moving: the triangle is A, the point B's, then the reverse; a
        // triangle against a bond's points only
        const bool tri_a = o.kind == 1 || (sub < 3) == MOVING;
        const int i = sub < 3 ? sub : sub - 3;
        for (int k = 0; k < 3; ++k) pts[k] = tri_a ? o.A[k] : o.B[k];
        const int* P = tri_a ? o.B : o.A;
        pts[3] = i == 0 ? P[0] : i == 1 ? P[1] : P[2];
        return true;
    }
    const int e = sub - npt;
    const int i = o.kind == 2 ? 0 : o.kind == 1 ? e : e / 3, j = o.kind == 0 ? e - 3 * i : 0;
    pts[0] = i == 0 ? o.A[0] : i == 1 ? o.A[1] : o.A[2];
    pts[1] = i == 0 ? o.A[1] : i == 1 ? o.A[2] : o.A[0];
    pts[2] = j == 0 ? o.B[0] : j == 1 ? o.B[1] : o.B[2];
    pts[3] = j == 0 ? o.B[1] : j == 1 ? o.B[2] : o.B[0];
    return true;
}

// One sub-test of a pair through the box and separating-axis filters; a
// survivor is queued with its key, and its pair, with its first, for stage 3.
template <bool MOVING>
__device__ __forceinline__ void queue_sub(const NarrowArgs& a, const NarrowCtx& c, bool ee, unsigned long long kb,
                                          int pair, int sc, const int* pts, int sub, bool thin, bool& first) {
    float ext, extb;
    if (ee || !thin) {
        if (!mixed_may_hit(c, pts, ee, &ext, &extb)) return;
        if (ee ? !sat_may_hit<MOVING, true>(c, pts, ext, extb) : !sat_may_hit<MOVING, false>(c, pts, ext, extb)) return;
    }
    int* cnt = ee ? &a.ctr->nsub_ee : &a.ctr->nsub_pt;
    int slot = aggregated_add(cnt, 1);
    if (slot >= a.sub_cap) {
        atomicOr(&a.ctr->err, kErrSubOverflow);
        return;
    }
    if (first) {
        a.pair_hit[pair] = 0;
        int q = aggregated_add(&a.ctr->npairq, 1);
        a.pairq[q] = pair;  // at most one entry per candidate pair: fits the pair buffer
        first = false;
    }
    SubRec r;
    r.keybase = kb;
    r.pair = pair;
    r.scene = sc;
    for (int i = 0; i < 4; ++i) r.p[i] = pts[i];
    r.sub = sub;
    r.counted = 0;
    (ee ? a.sub_ee : a.sub_pt)[slot] = r;
}

// Queues the sub-tests of the lanes with `queue` set, sixteen lanes (from lane
// `group` of the warp) per pair, and once each pair that has some. counted:
// the sub-test has been counted as evaluated in FP64.
__device__ __forceinline__ void queue_group(const NarrowArgs& a, bool queue, bool ee, unsigned long long keybase,
                                            int pair, int scene, const int* pts, int sub, int group, bool counted) {
    const unsigned in_pair = __ballot_sync(0xffffffffu, queue) >> group & 0xffffu;
    if (!queue) return;
    int slot;  // (the lanes that add together share one counter)
    if (ee)
        slot = aggregated_add(&a.ctr->nsub_ee, 1);
    else
        slot = aggregated_add(&a.ctr->nsub_pt, 1);
    if (slot >= a.sub_cap) {
        atomicOr(&a.ctr->err, kErrSubOverflow);
    } else {
        SubRec r;
        r.keybase = keybase;
        r.pair = pair;
        r.scene = scene;
        for (int i = 0; i < 4; ++i) r.p[i] = pts[i];
        r.sub = sub;
        r.counted = counted ? 1 : 0;
        (ee ? a.sub_ee : a.sub_pt)[slot] = r;
    }
    if ((in_pair & ((1u << sub) - 1u)) == 0) {  // the pair's first
        a.pair_hit[pair] = 0;
        a.pairq[aggregated_add(&a.ctr->npairq, 1)] = pair;
    }
}

// pair_may_hit on sixteen lanes (all of the group take part): lane s forms
// the gap along axis s of the twelve.
template <bool MOVING>
__device__ __forceinline__ int pair_may_hit16(const NarrowCtx& c, const OrientedPair& o, int s) {
    const int ia[3] = {o.A[0], o.A[1], o.n1 == 3 ? o.A[2] : o.A[1]};
    const int ib[3] = {o.B[0], o.B[1], o.n2 == 3 ? o.B[2] : o.B[1]};
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
    // axis 0 the line between the centroids; 1..4 and 5..8 each element's
    // normal and in-plane edge normals; 9..11 the first edges' common normal
    // and the in-plane normals of each
    float lb = -1.f, an = 0.f;
    if (s < 12) {
        F3 ax;
        if (s == 0) {
            F3 cA = fscale(fadd(fadd(R[0], R[1]), R[2]), 1.f / 3.f);
            F3 cB = fscale(fadd(fadd(R[3], R[4]), R[5]), 1.f / 3.f);
            ax = fsub(cB, cA);
        } else {
            const bool second = s >= 5, edges = s >= 9;
            const F3 P0 = second ? R[3] : R[0], P1 = second ? R[4] : R[1], P2 = second ? R[5] : R[2];
            const F3 e0 = fsub(P1, P0), e1 = fsub(P2, P1), e2 = fsub(P0, P2);
            const F3 d1 = fsub(R[1], R[0]), d2 = fsub(R[4], R[3]);
            const F3 nrm = edges ? fcross(d1, d2) : fcross(e0, fsub(P2, P0));
            const int k = edges ? s - 9 : second ? s - 5 : s - 1;
            const F3 e = edges ? (k == 1 ? d1 : d2) : k == 1 ? e0 : k == 2 ? e1 : e2;
            ax = k == 0 ? nrm : fcross(nrm, e);
        }
        lb = axis_gap(ax, R, an);
    }
    for (int d = 8; d > 0; d >>= 1) lb = fmaxf(lb, __shfl_xor_sync(0xffffffffu, lb, d));
    // the normals' lengths, from lanes 1 and 5
    return pair_bound<MOVING>(c, ia, o.n1, ib, o.n2, lb, L, M, __shfl_sync(0xffffffffu, an, 1, 16),
                              __shfl_sync(0xffffffffu, an, 5, 16));
}

// Passes of at most this many pairs take filter_wide. Moving filters of a
// step, with a thread per pair throughout / this line / sixteen threads
// throughout: sheet of 3,300 elements 0.032 / 0.015 / 0.015 ms, 48 sheets in
// contact (68 passes, the first of 1.46M pairs) 2.97 / 2.11 / 2.11, sheet of
// 136,000 elements 0.36 / 0.45 / 0.58 (0.34 with the line at 16,384 pairs).
constexpr int kWideFilter = 131072;

// Stage 1 with sixteen threads per pair, one per axis of the pair's bound and
// then one per sub-test. A thread's 12 axes and 15 sub-tests in turn (below)
// are ~36 us however few pairs a pass has.
template <bool MOVING>
__device__ __forceinline__ void filter_wide(const NarrowArgs& a, NarrowCtx& c, int np, int& t_visits) {
    const int sub = threadIdx.x & 15, group = (threadIdx.x & 31) & ~15;
    const int groups = (int)((gridDim.x * blockDim.x) >> 4);
    const int g0 = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 4);
    // every lane of a warp runs the same rounds: the pairs of its two groups
    for (int base = 0; base < np; base += groups) {
        const int idx = base + g0;
        bool on = idx < np, queue = false, ee = false;
        int pts[4] = {0, 0, 0, 0}, sc = 0;
        OrientedPair o;
        o.kind = 2;
        o.n1 = o.n2 = 2;
        o.keybase = 0;
        for (int k = 0; k < 3; ++k) o.A[k] = o.B[k] = 0;
        if (on) {
            int2 pr = a.pairs[idx];
            if (!MOVING && a.static_only && !(pr.y & kPairStatic)) on = false;
            pr.y &= kPairIdMask;
            if (on) on = orient_pair(a, pr, o);
            if (on) {
                t_visits += sub == 0;
                sc = a.escene[pr.x];
                bool shared = false;  // a shared point makes every test of the pair return false
                for (int i = 0; i < o.n1; ++i)
                    for (int j = 0; j < o.n2; ++j) shared |= o.A[i] == o.B[j];
                on = !shared;
            }
        }
        const double eps = a.scenes[sc].p.eps;
        c.hpad = filter_reach(MOVING ? eps : a.scenes[sc].p.thickness);
        c.epad = cut32_up(eps);
        c.dt32 = cut32_up(a.scenes[sc].p.dt);
        int bound = kPairNear;
        if (__any_sync(0xffffffffu, on)) bound = pair_may_hit16<MOVING>(c, o, sub);
        if (bound == kPairFar) on = false;
        if (on && pair_subtest<MOVING>(o, sub, pts, ee)) {
            float ext, extb;
            queue = (!ee && bound == kPairThin) ||
                    (mixed_may_hit(c, pts, ee, &ext, &extb) &&
                     (ee ? sat_may_hit<MOVING, true>(c, pts, ext, extb) : sat_may_hit<MOVING, false>(c, pts, ext, extb)));
        }
        queue_group(a, queue, ee, o.keybase, idx, sc, pts, sub, group, false);
    }
}

// Stage 1 of a split mixed pass: per candidate pair, the visit bookkeeping of
// k_narrow, the element-pair filter, and the box and separating-axis filter
// of every sub-test; survivors are queued, and pairs with survivors for
// stage 3. Sixteen threads per pair in passes of at most kWideFilter pairs,
// in larger ones, which fill the chip either way, a thread per pair.
// Registers held to 64 and 96, which let a block of 128 threads run eight and
// five times on an SM: with the moving kernel's own choice of 108 a step of 48
// sheets in contact took 29.2 ms against 28.8.
template <bool MOVING>
__global__ void __maxnreg__(MOVING ? 96 : 64) k_narrow_filter(NarrowArgs a, int max_pairs) {
    NarrowCtx c;
    c.pbox_lo = a.pbox_lo; c.pbox_hi = a.pbox_hi; c.p32 = a.p32; c.v32 = a.v32;
    int np = a.ctr->npairs;
    if (np > max_pairs) np = max_pairs;
    int t_visits = 0;
    if (np <= kWideFilter) filter_wide<MOVING>(a, c, np, t_visits);
    for (int idx = np <= kWideFilter ? np : blockIdx.x * blockDim.x + threadIdx.x; idx < np;
         idx += gridDim.x * blockDim.x) {
        int2 pr = a.pairs[idx];
        if (!MOVING && a.static_only && !(pr.y & kPairStatic)) continue;
        pr.y &= kPairIdMask;
        OrientedPair o;
        if (!orient_pair(a, pr, o)) continue;
        t_visits++;
        int sc = a.escene[pr.x];
        const double eps = a.scenes[sc].p.eps;
        c.hpad = filter_reach(MOVING ? eps : a.scenes[sc].p.thickness);
        c.epad = cut32_up(eps);
        c.dt32 = cut32_up(a.scenes[sc].p.dt);
        // a shared point makes every test of the pair return false
        bool shared = false;
        for (int i = 0; i < o.n1; ++i)
            for (int j = 0; j < o.n2; ++j) shared |= o.A[i] == o.B[j];
        const int bound = shared ? kPairFar : pair_may_hit<MOVING>(c, o.A, o.n1, o.B, o.n2);
        if (bound == kPairFar) continue;
        bool first = true;
        for_each_subtest<MOVING>(o.kind, o.A, o.B, [&](int sub, const int* pts, bool ee) {
            queue_sub<MOVING>(a, c, ee, o.keybase, idx, sc, pts, sub, bound == kPairThin, first);
        });
    }
    for (int o = 16; o > 0; o >>= 1) t_visits += __shfl_xor_sync(0xffffffffu, t_visits, o);
    if ((threadIdx.x & 31) == 0 && t_visits) atomicAdd(&a.ctr->nvisits, t_visits);
}

// Stage 1 of a plain FP64 pass, sixteen threads per pair: a sub-test whose
// elements stay farther apart than a hit allows (gap_may_hit, on the points
// cut to FP32) is done, the others are queued for the full test. Every
// sub-test counts as evaluated. An FP64 test
// of each of a pair's fifteen sub-tests took a static pass over 24 sheets
// 2.07 ms, and the moving passes of their step 2.0 ms; now 0.29 and 0.58 ms.
constexpr int kPlainBlock = 128;
template <bool MOVING>
__global__ void __launch_bounds__(kPlainBlock) k_plain_filter(NarrowArgs a, int max_pairs) {
    int np = a.ctr->npairs;
    if (np > max_pairs) np = max_pairs;
    const int sub = threadIdx.x & 15, group = (threadIdx.x & 31) & ~15;
    int t_visits = 0, t_sub = 0;
    const int groups = (int)(gridDim.x * (kPlainBlock / 16));
    const int g0 = (int)(blockIdx.x * (kPlainBlock / 16) + (threadIdx.x >> 4));
    for (int base = 0; base < np; base += groups) {
        const int idx = base + g0;
        bool queue = false, ee = false;
        int pts[4] = {0, 0, 0, 0}, sc = 0;
        OrientedPair o;
        o.keybase = 0;
        if (idx < np) {
            int2 pr = a.pairs[idx];
            const bool on = MOVING || !a.static_only || (pr.y & kPairStatic);
            pr.y &= kPairIdMask;
            if (on && orient_pair(a, pr, o)) {
                t_visits += sub == 0;
                bool shared = false;  // a shared point makes every test of the pair return false
                for (int i = 0; i < o.n1; ++i)
                    for (int j = 0; j < o.n2; ++j) shared |= o.A[i] == o.B[j];
                sc = a.escene[pr.x];
                if (!shared && pair_subtest<MOVING>(o, sub, pts, ee)) {
                    ++t_sub;
                    queue = plain_may_hit<MOVING>(a.xo, a.av, pts, ee, a.scenes[sc].p);
                }
            }
        }
        queue_group(a, queue, ee, o.keybase, idx, sc, pts, sub, group, true);
    }
    for (int o = 16; o > 0; o >>= 1) {
        t_visits += __shfl_xor_sync(0xffffffffu, t_visits, o);
        t_sub += __shfl_xor_sync(0xffffffffu, t_sub, o);
    }
    if ((threadIdx.x & 31) == 0) {
        if (t_visits) atomicAdd(&a.ctr->nvisits, t_visits);
        if (t_sub) atomicAdd(&a.ctr->nsub, t_sub);
    }
}

// Stage 3 (impact-zone scenes): createImpZone for every sub-test of a pair
// from its first hit on, in sub-test order - the reference's status stays
// true after the first hit (dcollid3d.cpp:300-321), whether or not the
// later sub-tests ran in FP64.
__global__ void __launch_bounds__(128) k_zone_unions(NarrowArgs a) {
    int n = a.ctr->npairq;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int pi = a.pairq[i];
        const int mask = a.pair_hit[pi];
        if (!mask) continue;
        int2 pr = a.pairs[pi];
        pr.y &= kPairIdMask;
        const int sc = a.escene[pr.x];
        if (a.run[sc].mode != kSceneZone) continue;
        OrientedPair o;
        if (!orient_pair(a, pr, o)) continue;
        const int kfirst = __ffs(mask) - 1;
        for_each_subtest<true>(o.kind, o.A, o.B, [&](int sub, const int* pts, bool) {
            if (sub < kfirst) return;
            int slot = aggregated_add(&a.ctr->nunion, 1);
            if (slot >= a.urec_cap) {
                atomicOr(&a.ctr->err, kErrUnionOverflow);
                return;
            }
            UnionRec r;
            r.key = o.keybase | (unsigned long long)sub;
            for (int q = 0; q < 4; ++q) r.p[q] = pts[q];
            a.urec[slot] = r;
        });
    }
}

// Stage 2: the FP64 test of k_narrow for each queued sub-test.
struct SubTally {
    int hits = 0, cr = 0, contacts = 0, sub = 0;
};

__device__ __forceinline__ NarrowCtx subtest_ctx(const NarrowArgs& a) {
    NarrowCtx c;
    c.xo = a.xo; c.av = a.av; c.fixed = a.fixed; c.ev = a.ev; c.esurf = a.esurf; c.erigid = a.erigid;
    c.vbody = a.vbody; c.body_mass = a.body_mass; c.body_slot0 = a.body_slot0;
    c.rank = a.rank;
    c.contrib = a.contrib; c.contrib_cap = a.contrib_cap; c.ctr = a.ctr; c.urec = nullptr; c.urec_cap = 0;
    c.rec = nullptr; c.rec_cap = 0;
    c.pbox_lo = nullptr; c.pbox_hi = nullptr; c.p32 = nullptr; c.v32 = nullptr;
    c.check = a.check;
    c.zone = 0;
    return c;
}

// One sub-test: its test, the stamps of its points and its pair's hit flag
// when it hits, the scene's hit count when it is the pair's first.
// counted: the sub-test has been counted (k_subtests_cubic).
template <bool MOVING, bool EE>
__device__ __forceinline__ void one_subtest(const NarrowArgs& a, NarrowCtx& c, const SubRec& r, bool counted,
                                            SubTally& t) {
    c.p = a.scenes[r.scene].p;
    c.pass = 0;
    CallState st;
    st.keybase = r.keybase;
    st.np = 0;
    st.sub = r.sub;
    st.nsub = 0;
    st.ncr = 0;
    st.ncontacts = 0;
    bool hit = MOVING ? moving_test<EE>(c, st, r.p) : static_test<EE>(c, st, r.p);
    t.sub += !counted && r.counted == 0;
    t.cr += st.ncr;
    t.contacts += st.ncontacts;
    if (hit)
        for (int q = 0; q < 4; ++q) stamp_point(a.ps, r.p[q]);
    if (hit && atomicOr(&a.pair_hit[r.pair], 1 << r.sub) == 0) {
        t.hits++;
        atomicAdd(&a.run[r.scene].hits, 1);
    }
}

// The pass's counters from every thread's tally (all lanes take part).
__device__ __forceinline__ void subtest_counts(const NarrowArgs& a, SubTally t) {
    for (int o = 16; o > 0; o >>= 1) {
        t.hits += __shfl_xor_sync(0xffffffffu, t.hits, o);
        t.cr += __shfl_xor_sync(0xffffffffu, t.cr, o);
        t.contacts += __shfl_xor_sync(0xffffffffu, t.contacts, o);
        t.sub += __shfl_xor_sync(0xffffffffu, t.sub, o);
    }
    if ((threadIdx.x & 31) == 0) {
        if (t.hits) atomicAdd(&a.ctr->nhit_pairs, t.hits);
        if (t.cr) atomicAdd(&a.ctr->ncr, t.cr);
        if (t.contacts) atomicAdd(&a.ctr->ncontacts, t.contacts);
        if (t.sub) atomicAdd(&a.ctr->nsub, t.sub);
    }
}

// Moving passes of more sub-tests than kSubSparse first form every cubic, a
// sub-test per thread, and list those that may have a root in the time window
// (may_be_coplanar); the tests then run on the lists. Most of a filter's
// survivors end here, and one lane's roots and tests otherwise hold up its
// warp. 257 x 257 points in contact: filters and sub-tests of a step 1.48 ->
// 1.09 ms (the filter formed the cubics of its survivors before, with almost
// every warp holding one).
// Passes of fewer give each sub-test its own warp (k_subtests) and need no
// list: two warps on each of the 608 SM sub-partitions. Sub-tests of a step
// without such passes / with this line / at 9,728 of them: 64 strings 0.25 /
// 0.14 / 0.15 ms, 48 sheets in contact 4.38 / 3.41 / 5.52, 24 FP64 sheets
// 0.51 / 0.40 / 0.52, sheet of 136,000 elements 0.67 / 0.67 / 0.74.
constexpr int kSubSparse = 1216;
struct SubLists {
    int npt, nee;
    bool listed;
};
template <bool MOVING>
__device__ __forceinline__ SubLists sub_lists(const NarrowArgs& a) {
    SubLists l;
    l.npt = a.ctr->nsub_pt < a.sub_cap ? a.ctr->nsub_pt : a.sub_cap;
    l.nee = a.ctr->nsub_ee < a.sub_cap ? a.ctr->nsub_ee : a.sub_cap;
    l.listed = MOVING && l.npt + l.nee > kSubSparse;
    if (l.listed) {
        l.npt = a.ctr->nlive_pt;
        l.nee = a.ctr->nlive_ee;
    }
    return l;
}

__global__ void __launch_bounds__(128) k_subtests_cubic(NarrowArgs a) {
    const int npt = a.ctr->nsub_pt < a.sub_cap ? a.ctr->nsub_pt : a.sub_cap;
    const int nee = a.ctr->nsub_ee < a.sub_cap ? a.ctr->nsub_ee : a.sub_cap;
    const int n = npt + nee;
    if (n <= kSubSparse) return;
    int t_sub = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const bool ee = i >= npt;
        const int k = ee ? i - npt : i;
        const SubRec& r = (ee ? a.sub_ee : a.sub_pt)[k];
        double xo4[4][3], av4[4][3];
        for (int q = 0; q < 4; ++q) {
            load3(a.xo, r.p[q], xo4[q]);
            load3(a.av, r.p[q], av4[q]);
        }
        t_sub += r.counted == 0;
        if (!may_be_coplanar(xo4, av4, a.scenes[r.scene].p.dt)) continue;
        if (ee)  // (the lanes that add together share one counter)
            a.live_ee[aggregated_add(&a.ctr->nlive_ee, 1)] = k;
        else
            a.live_pt[aggregated_add(&a.ctr->nlive_pt, 1)] = k;
    }
    for (int o = 16; o > 0; o >>= 1) t_sub += __shfl_xor_sync(0xffffffffu, t_sub, o);
    if ((threadIdx.x & 31) == 0 && t_sub) atomicAdd(&a.ctr->nsub, t_sub);
}

// Passes with more sub-tests than this give each kind blocks of its own:
// measured faster than both kinds in a warp when the pass is large, where the
// FP64 pipes are full either way.
constexpr int kSubMergeMax = 65536;

// Both lists in one launch. Up to kSubMergeMax sub-tests, point-triangle ones
// first, so that a small pass's two lists run side by side; above (and with
// merged = 0 throughout) point-triangle ones in the even blocks and edge-edge
// ones in the odd. A warp pays for an FP64 instruction the
// same whatever the number of its lanes that execute it, and the lanes of a
// warp running different sub-tests follow the union of their paths: a pass
// with at most kSubSparse sub-tests (two warps per SM sub-partition) gives
// each its own warp, which then follows one path; larger passes take one
// sub-test per thread, which keeps the FP64 pipe's issue slots full.
// Two blocks per SM: one warp per SM sub-partition already keeps its FP64
// pipe issuing, and the registers then hold both tests without spills.
template <bool MOVING>
__global__ void __launch_bounds__(128, 2) k_subtests(NarrowArgs a, int merged) {
    const SubLists l = sub_lists<MOVING>(a);
    const int n = l.npt + l.nee;
    NarrowCtx c = subtest_ctx(a);
    SubTally t;
    const bool by_kind = !merged || n > kSubMergeMax, sparse = !by_kind && n <= kSubSparse;
    if (!sparse || (threadIdx.x & 31) == 0) {
        // this thread's place among those that share its list, of `end` sub-tests from `i` on
        const int per = sparse ? (int)(blockDim.x >> 5) : (int)blockDim.x;
        const int block = by_kind ? blockIdx.x >> 1 : blockIdx.x, blocks = by_kind ? gridDim.x >> 1 : gridDim.x;
        const int first = by_kind && (blockIdx.x & 1) ? l.npt : 0, end = by_kind && !(blockIdx.x & 1) ? l.npt : n;
        for (int i = first + block * per + (sparse ? threadIdx.x >> 5 : threadIdx.x); i < end; i += blocks * per) {
            if (i < l.npt)
                one_subtest<MOVING, false>(a, c, a.sub_pt[l.listed ? a.live_pt[i] : i], l.listed, t);
            else
                one_subtest<MOVING, true>(a, c, a.sub_ee[l.listed ? a.live_ee[i - l.npt] : i - l.npt], l.listed, t);
        }
    }
    subtest_counts(a, t);
}

// dn (may be null): the point count in device memory; the grid strides.
template <bool MOVING>
__global__ void k_point_boxes(const double4_32a* __restrict__ xo, const double4_32a* __restrict__ av,
                              const int* __restrict__ vscene, const SceneDev* __restrict__ scenes,
                              const int* __restrict__ act, int n, const int* __restrict__ dn, float4* lo, float4* hi,
                              float4* p32, float4* v32) {
    if (dn) n = *dn;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x)
        point_box<MOVING>(xo, av, vscene, scenes, act ? act[k] : k, lo, hi, p32, v32);
}

}  // namespace

void point_boxes(const double4_32a* xo, const double4_32a* av, const int* vscene, const SceneDev* scenes,
                 const int* act_pts, int n, int moving, float4* lo, float4* hi, float4* p32, float4* v32,
                 cudaStream_t s, const int* dn) {
    if (n <= 0) return;
    int g = (n + 255) / 256;
    if (dn && g > 152 * 8) g = 152 * 8;
    if (moving)
        count_launch(), k_point_boxes<true><<<g, 256, 0, s>>>(xo, av, vscene, scenes, act_pts, n, dn, lo, hi, p32,
                                                              v32);
    else
        count_launch(), k_point_boxes<false><<<g, 256, 0, s>>>(xo, av, vscene, scenes, act_pts, n, dn, lo, hi, p32,
                                                               v32);
}

void narrow_pass(const NarrowArgs& a, int moving, int max_pairs, cudaStream_t s, int) {
    if (max_pairs <= 0) return;
    int threads = 128;
    int blocks = (max_pairs + threads - 1) / threads;
    if (blocks > 152 * 16) blocks = 152 * 16;
    if (moving)
        count_launch(), k_narrow<true><<<blocks, threads, 0, s>>>(a, max_pairs);
    else
        count_launch(), k_narrow<false><<<blocks, threads, 0, s>>>(a, max_pairs);
}

void narrow_pass_split(const NarrowArgs& args, int moving, int max_pairs, cudaStream_t s, int block, bool zone,
                       int parts) {
    if (max_pairs <= 0) return;
    const bool mixed = args.pbox_lo && args.p32 && (!moving || args.v32);  // the FP32 filters' point data (mode 1)
    const NarrowArgs& a = args;
    long long pb = (16ll * max_pairs + kPlainBlock - 1) / kPlainBlock;
    if (pb > 152 * 16) pb = 152 * 16;
    const int cap_blocks = 152 * 16 * 128 / block;
    int blocks = (max_pairs + block - 1) / block;
    // (sixteen threads per pair in passes of few pairs)
    const long long wide = (16ll * (max_pairs < kWideFilter ? max_pairs : kWideFilter) + block - 1) / block;
    if (blocks < wide) blocks = (int)wide;
    if (blocks > cap_blocks) blocks = cap_blocks;
    int sblocks = (a.sub_cap + 127) / 128;
    if (sblocks > 152 * 16) sblocks = 152 * 16;
    // one grid for any number of sub-tests, strided above kSubMergeMax, with at
    // least one warp per sub-test of a sparse pass and an even block count
    long long mb = (2ll * a.sub_cap + 127) / 128;
    if (mb > (kSubMergeMax + 127) / 128) mb = (kSubMergeMax + 127) / 128;
    if (mb < (kSubSparse + 3) / 4) mb = (kSubSparse + 3) / 4;
    const int mblocks = (int)(mb + 1) & ~1;
    if (moving) {
        if (parts & kSplitFilter) {
            if (mixed) {
                count_launch(), k_narrow_filter<true><<<blocks, block, 0, s>>>(a, max_pairs);
            } else {
                count_launch(), k_plain_filter<true><<<(int)pb, kPlainBlock, 0, s>>>(a, max_pairs);
            }
        }
        if (parts & kSplitSubtests) {
            count_launch(), k_subtests_cubic<<<sblocks < 152 * 8 ? sblocks : 152 * 8, 128, 0, s>>>(a);
            count_launch(), k_subtests<true><<<mblocks, 128, 0, s>>>(a, a.sub_merge);
            if (zone) count_launch(), k_zone_unions<<<blocks, 128, 0, s>>>(a);
        }
    } else {
        if (parts & kSplitFilter) {
            if (mixed)
                count_launch(), k_narrow_filter<false><<<blocks, block, 0, s>>>(a, max_pairs);
            else
                count_launch(), k_plain_filter<false><<<(int)pb, kPlainBlock, 0, s>>>(a, max_pairs);
        }
        if (parts & kSplitSubtests) {
            count_launch(), k_subtests<false><<<mblocks, 128, 0, s>>>(a, a.sub_merge);
        }
    }
}

}  // namespace ccg
