// Schedule of one scene's strain sweeps; see cc_sweep_plan.h.
#include "cc_sweep_plan.h"

#include <algorithm>
#include <cstdint>
#include <deque>

namespace ccg {

namespace {

// Slots needed with k levels per epoch: points alive per step, a point from
// step first/k - 2 (its copy-in) to step last/k + 1 (its write-back).
int slots_for(const std::vector<int>& first, const std::vector<int>& last, int nlevels, int k) {
    const int ne = (nlevels + k - 1) / k;
    std::vector<int> change((size_t)ne + 5, 0);
    for (size_t p = 0; p < first.size(); ++p)
        if (first[p] >= 0) {
            change[first[p] / k]++;       // step first/k - 2, shifted by 2
            change[last[p] / k + 4]--;    // free from step last/k + 2
        }
    int cur = 0, most = 0;
    for (int c : change) {
        cur += c;
        most = std::max(most, cur);
    }
    return most;
}

}  // namespace

int append_sweep_plan(const std::vector<SweepElem>& elems, int v0, int nv, SweepArrays& out, SceneDev& sd) {
    const int m = (int)elems.size();
    std::vector<int> lvl((size_t)m), last((size_t)nv, -1), first((size_t)nv, -1);
    int nlevels = 0;
    for (int i = 0; i < m; ++i) {
        const int np = elems[i].np();
        int l = 0;
        for (int k = 0; k < np; ++k) l = std::max(l, last[elems[i].p[k] - v0] + 1);
        for (int k = 0; k < np; ++k) {
            const int p = elems[i].p[k] - v0;
            last[p] = l;
            if (first[p] < 0) first[p] = l;
        }
        lvl[i] = l;
        nlevels = std::max(nlevels, l + 1);
    }
    std::vector<int> off((size_t)nlevels + 1, 0);
    for (int i = 0; i < m; ++i) off[lvl[i] + 1]++;
    int width = 0;
    for (int l = 0; l < nlevels; ++l) {
        width = std::max(width, off[l + 1]);
        off[l + 1] += off[l];
    }
    // The longest epoch whose shared memory lets two or more sweeps share an
    // SM; else the longest that fits with a record ring; else single-level
    // epochs with the records read from global memory.
    int k = 0, slots = 0, ring = 1;
    for (size_t want : {kSweepSharedBytes, kSweepMaxBytes}) {
        for (int c = kSweepMaxEpoch; c >= 1 && !k; c /= 2) {
            slots = slots_for(first, last, nlevels, c);
            if (sweep_smem(slots, width, 1) <= want) k = c;
        }
        if (k) break;
    }
    if (!k) {
        k = 1;
        ring = 0;
        slots = slots_for(first, last, nlevels, 1);
    }
    const int ne = (nlevels + k - 1) / k;
    sd.sw_lev0 = (int)out.lev.size();
    sd.sw_levels = nlevels;
    sd.sw_ep0 = (int)out.epoch.size();
    sd.sw_epochs = ne;
    sd.sw_k = k;
    sd.sw_width = width;
    sd.sw_slots = slots;
    sd.sw_ring = ring;
    sd.sw_e0 = (int)out.elems.size();
    sd.sw_ne = m;
    sd.sw_fits = sweep_smem(slots, width, ring) <= kSweepMaxBytes && slots <= 0xffff;

    // the points of each epoch in the order of their first levels, and in a
    // level of its elements; a freed slot goes to the back of the queue: the
    // elements side by side in a level mostly find their points in
    // neighbouring slots, whose loads meet no bank conflicts
    std::vector<int> by_level((size_t)m);
    {
        std::vector<int> cur(off.begin(), off.end() - 1);
        for (int i = 0; i < m; ++i) by_level[cur[lvl[i]]++] = i;
    }
    std::vector<std::vector<int>> by_first((size_t)ne), by_last((size_t)ne);
    std::vector<uint8_t> seen((size_t)nv, 0);
    int npts = 0;
    for (int l = 0; l < nlevels; ++l)
        for (int c = 0; c < 3; ++c)
            for (int i = off[l]; i < off[l + 1]; ++i) {
                const SweepElem& el = elems[by_level[i]];
                if (c >= el.np()) continue;
                const int p = el.p[c] - v0;
                if (seen[p]) continue;
                seen[p] = 1;
                by_first[l / k].push_back(p);
                by_last[last[p] / k].push_back(p);
                ++npts;
            }
    std::vector<int> slot((size_t)nv, -1);
    std::deque<int> free_slots;
    int nslots = 0, need = 0;
    const int lbase = (int)out.load.size(), wbase = (int)out.wb.size();
    int nl = 0, nw = 0;
    for (int e = 0; e < ne; ++e) {
        if (e >= 4)  // written back in step e - 3, before epoch e's copy-ins are issued in step e - 2
            for (int p : by_last[e - 4]) free_slots.push_back(slot[p]);
        int4 h;
        h.x = lbase + nl;
        for (int p : by_first[e]) {
            if (free_slots.empty()) free_slots.push_back(nslots++);
            slot[p] = free_slots.front();
            free_slots.pop_front();
            out.load.push_back(int2{v0 + p, slot[p]});
            need = std::max(need, last[p] / k + 1);
            ++nl;
        }
        h.y = lbase + nl;
        h.z = wbase + nw;
        for (int p : by_last[e]) {
            out.wb.push_back(int2{v0 + p, 0});
            ++nw;
        }
        h.w = wbase + nw;
        out.epoch.push_back(h);
        out.need.push_back(need);
    }
    for (int i = wbase; i < wbase + nw; ++i) out.wb[i].y = slot[out.wb[i].x - v0];
    for (int l = 0; l <= nlevels; ++l) out.lev.push_back(sd.sw_e0 + off[l]);
    out.elems.resize(out.elems.size() + (size_t)m);
    for (int i = 0; i < m; ++i) {
        SweepElem e = elems[by_level[i]];
        e.set_slots(slot[e.p[0] - v0], slot[e.p[1] - v0], slot[e.p[2] - v0]);
        out.elems[(size_t)sd.sw_e0 + i] = e;
    }
    return npts;
}

}  // namespace ccg
