// Test shim: the strain sweeps' schedule (collision_gb300/csrc/cc_sweep_plan.cpp)
// and a host model of k_strain_sweeps that follows it: ten sweeps, each step
// taken in a random order that the sweeps' waits allow, against the
// sequential sweeps.
#include <cmath>
#include <cstring>
#include <random>

#include "cc_sweep_plan.h"

using namespace ccg;

namespace {

// Whether an edge averages: any fixed rule of the two velocities serves.
bool over(double a, double b) { return std::fabs(a - b) > 0.3; }

void take(const SweepElem& el, double* v0, double* v1, double* v2) {
    double* v[3] = {v0, v1, v2};
    for (int j = 0; j < ((el.s2n >> 16) == 1 ? 1 : 3); ++j) {
        double &a = *v[j], &b = *v[(j + 1) % 3];
        if (over(a, b)) a = b = 0.5 * (a + b);
    }
}

}  // namespace

// tris: nt x 3, bonds: nb x 2, point ids below nv. Returns 0 when the model
// equals the sequential sweeps bit for bit, else the first thing found wrong.
// info: levels, epochs, levels per epoch, widest level, slots, ring.
extern "C" int sweep_plan_check(const int* tris, int nt, const int* bonds, int nb, int nv, int seed, int* info) {
    const int v0 = 1000;
    std::vector<SweepElem> elems;
    for (int i = 0; i < nt + nb; ++i) {
        SweepElem e;
        std::memset(&e, 0, sizeof(e));
        const bool tri = i < nt;
        for (int k = 0; k < 3; ++k)
            e.p[k] = v0 + (tri ? tris[3 * i + k] : bonds[2 * (i - nt) + (k == 1 ? 1 : 0)]);
        e.s2n = (tri ? 3u : 1u) << 16;
        elems.push_back(e);
    }
    SweepArrays A;
    A.lev = {7, 7, 7};  // as after another scene
    A.load = {int2{0, 0}};
    SceneDev sd;
    std::memset(&sd, 0, sizeof(sd));
    append_sweep_plan(elems, v0, nv, A, sd);
    const int K = sd.sw_k, L = sd.sw_levels, E = sd.sw_epochs;
    const int out[6] = {L, E, K, sd.sw_width, sd.sw_slots, sd.sw_ring};
    std::memcpy(info, out, sizeof(out));
    if ((int)A.lev.size() != sd.sw_lev0 + L + 1 || (int)A.epoch.size() != E || (int)A.elems.size() != nt + nb) return 1;
    std::mt19937 rng((unsigned)seed);
    std::vector<double> start((size_t)nv);
    for (double& x : start) x = std::uniform_real_distribution<double>(-1.0, 1.0)(rng);
    constexpr int S = kStrainMaxIter;
    std::vector<double> seq = start;
    for (int k = 0; k < S; ++k)
        for (const SweepElem& e : elems) take(e, &seq[e.p[0] - v0], &seq[e.p[1] - v0], &seq[e.p[2] - v0]);
    // the model: per sweep its next step and published epochs, its slots and
    // the copies in flight (issued one step, landed the next)
    struct Sweep {
        int step = -2, published = 0;
        std::vector<double> slot;
        std::vector<int> owner;
        std::vector<std::pair<int, double>> flight;
    };
    std::vector<Sweep> sw(S);
    for (Sweep& s : sw) {
        s.slot.assign((size_t)sd.sw_slots, NAN);
        s.owner.assign((size_t)sd.sw_slots, -1);
    }
    std::vector<double> av = start;
    const int* lev = A.lev.data() + sd.sw_lev0;
    for (int left = S * (E + 3); left > 0;) {
        std::vector<int> ready;
        for (int k = 0; k < S; ++k) {
            const int t = sw[k].step;
            if (t > E) continue;
            const int e = t + 2;
            if (k == 0 || e >= E || sw[k - 1].published >= A.need[e]) ready.push_back(k);
        }
        if (ready.empty()) return 2;
        const int k = ready[rng() % ready.size()];
        Sweep& s = sw[k];
        const int t = s.step++;
        --left;
        // workers
        if (t >= 0)
            for (int l = t * K; l < (t + 1) * K && l < L; ++l)
                for (int i = lev[l]; i < lev[l + 1]; ++i) {
                    const SweepElem& el = A.elems[i];
                    const unsigned q[3] = {el.s01 & 0xffffu, el.s01 >> 16, el.s2n & 0xffffu};
                    for (int c = 0; c < 3; ++c)
                        if (q[c] >= s.slot.size() || s.owner[q[c]] != el.p[c]) return 3;
                    take(el, &s.slot[q[0]], &s.slot[q[1]], &s.slot[q[2]]);
                }
        // helpers: landed copies, new copies, write-backs
        for (auto& f : s.flight) s.slot[f.first] = f.second;
        s.flight.clear();
        if (t + 2 < E) {
            const int4 h = A.epoch[t + 2];
            for (int i = h.x; i < h.y; ++i) {
                const int2 ps = A.load[i];
                if (ps.y < 0 || ps.y >= sd.sw_slots || s.owner[ps.y] != -1) return 4;
                s.owner[ps.y] = ps.x;
                s.flight.push_back({ps.y, av[ps.x - v0]});
            }
        }
        if (t >= 1) {
            const int4 h = A.epoch[t - 1];
            for (int i = h.z; i < h.w; ++i) {
                const int2 ps = A.wb[i];
                if (s.owner[ps.y] != ps.x) return 5;
                av[ps.x - v0] = s.slot[ps.y];
                s.owner[ps.y] = -1;
            }
            s.published = t;
        }
    }
    return std::memcmp(av.data(), seq.data(), sizeof(double) * av.size()) == 0 ? 0 : 6;
}
