// The reference tree's leaf order, built on the GPU.
//
// The reference builds each AABB tree by inserting leaves 0..n-1 one at a
// time, descending from the root into the child whose box grows least
// (ties go right) and splitting the leaf it reaches into a branch (new leaf
// left, old leaf right); every box on the path is then the union of its
// children's (AABB.cpp:129-197). Only the inorder rank of every leaf and the
// root volume are needed (cc_tree_order.h says why).
//
// The insertions are sequential in the reference, but their descents can
// overlap: insertion e, at a node of depth d, reads and writes only that
// node's record (its children's ids and boxes) and, splitting a leaf, makes
// the record below it. So one CTA runs the insertions as a pipeline, every
// active insertion one level per step with a block barrier between steps,
// and at most one insertion starting per step. Insertion e then reaches
// every depth at least one step after insertion e-1 and sees exactly the
// tree the reference's insertion e sees; in one step no two insertions touch
// the same record. Boxes are widened on the way down (the union with the new
// leaf's box), which gives the same box as the reference's bottom-up union
// of the children: min and max are exact.
//
// Leaves are ids 0..n-1 and insertion e (e >= 1) creates the internal node
// n+e-1. Each insertion also keeps parent links and leaf counts, from which
// k_tree_ranks gives each leaf its inorder rank by walking to the root.
#include <atomic>

#include "cc_launch.h"

namespace ccg {

namespace {

constexpr int kTreeThreads = 1024;
constexpr int kTreeGroups = kTreeThreads / 4;  // insertions in flight, by lanes
// Trees of at most this many leaves by lanes, larger ones by threads. One
// tree by lanes / by threads: 97 x 97 sheet on two obstacles (39,000 leaves)
// 45 / 67 ms, 85,000 leaves 173 / 198, 126,000 322 / 331, 152,000 443 / 435,
// 280,000 1,137 / 1,052, 545,000 3,218 / 2,777, 2.1 million 24.6 / 20.4 s.
// Two or more insertions per group in registers (512 and 1,024 in flight) are
// slower than either: 3.6 s and more for the 545,000.
constexpr int kTreeLaneMax = 131072;

// Box coordinates are kept as order-preserving integer keys: key(a) <
// key(b) exactly when a < b for doubles that are not NaN, except that -0
// orders below +0. So min and max run on the integer pipe (GB300's FP64
// rate is a small fraction of its integer rate). Where the reference's
// std::min/std::max would keep +0 and the key order keeps -0, the difference
// is only the sign of a zero coordinate, which changes no box extent, volume
// comparison or decision.
//
// A child as its parent's record holds it, in the halves that two lanes load:
// the keys of x and y, then those of z, the volume (AABB::volume of the box,
// AABB.cpp:51-54) and the child's id.
struct __align__(16) TreeChild {
    long long xlo, xhi, ylo, yhi;
    long long zlo, zhi;
    double vol;
    long long id;
};
struct TreeNode {
    TreeChild child[2];  // left, right
};

__device__ __forceinline__ long long okey(double d) {
    const long long b = __double_as_longlong(d);
    return b ^ ((b >> 63) & 0x7fffffffffffffffll);
}
__device__ __forceinline__ double odec(long long k) {
    return __longlong_as_double(k ^ ((k >> 63) & 0x7fffffffffffffffll));
}
__device__ __forceinline__ long long kmin(long long a, long long b) { return b < a ? b : a; }
__device__ __forceinline__ long long kmax(long long a, long long b) { return a < b ? b : a; }

// (hi - lo) products in the reference's order, never contracted
__device__ __forceinline__ double volume_k(const TreeChild& c) {
    return __dmul_rn(__dmul_rn(__dsub_rn(odec(c.xhi), odec(c.xlo)), __dsub_rn(odec(c.yhi), odec(c.ylo))),
                     __dsub_rn(odec(c.zhi), odec(c.zlo)));
}

// A child's box with another's (volume and id left out), and whether it holds
// the other already.
__device__ __forceinline__ TreeChild joined(const TreeChild& a, const TreeChild& b) {
    TreeChild c;
    c.xlo = kmin(a.xlo, b.xlo); c.xhi = kmax(a.xhi, b.xhi);
    c.ylo = kmin(a.ylo, b.ylo); c.yhi = kmax(a.yhi, b.yhi);
    c.zlo = kmin(a.zlo, b.zlo); c.zhi = kmax(a.zhi, b.zhi);
    return c;
}
__device__ __forceinline__ bool holds(const TreeChild& a, const TreeChild& b) {
    return a.xlo <= b.xlo && a.ylo <= b.ylo && a.zlo <= b.zlo && b.xhi <= a.xhi && b.yhi <= a.yhi && b.zhi <= a.zhi;
}

// One lane's half of a child: lane h = 0 xlo, xhi, ylo, yhi; h = 1 zlo, zhi,
// the volume's bits, the id.
struct Half {
    long long a, b, c, d;
};
__device__ __forceinline__ Half load_half(const TreeChild* p, int h) {
    const longlong2* q = reinterpret_cast<const longlong2*>(p) + 2 * h;
    const longlong2 u = q[0], v = q[1];
    return Half{u.x, u.y, v.x, v.y};
}
__device__ __forceinline__ void store_half(TreeChild* p, int h, const Half& x) {
    longlong2* q = reinterpret_cast<longlong2*>(p) + 2 * h;
    q[0] = make_longlong2(x.a, x.b);
    q[1] = make_longlong2(x.c, x.d);
}

// Insertions 2 .. n - 1, four lanes each (lane 2 s + h: half h of child s).
// What bounds a build is the time of a step, one level of every insertion in
// flight: with a thread per insertion it was ~14 FP64 instructions of each
// warp (GB300 takes ~64 cycles for one however many lanes it serves, and 32
// insertions' lanes rarely all skip them), two dependent loads (the child ids,
// then the children) and the barrier. Here both children's unions are formed
// side by side, x and z too, which leaves five FP64 instructions; a node's
// record holds both children, so a level is one round of loads; a new leaf's
// record is loaded an insertion ahead; and the leaf counts are adds that
// nothing waits for.
__device__ void insert_by_lanes(TreeNode* nd, const TreeChild* leaf, int* parent, int* extra, int n) {
    const int tid = threadIdx.x;
    const int g = tid >> 2, side = (tid >> 1) & 1, h = tid & 1;
    const int lane = tid & 31, base = lane & ~3;  // the group's first lane in its warp
    const Half none{0, 0, 0, 0};
    int my_e = -1, p = n;
    Half mine = none;
    int ahead = g < 2 ? g + kTreeGroups : g;  // this group's next insertion, and its leaf
    Half next_leaf = ahead < n ? load_half(&leaf[ahead], h) : none;
    int next = 2;  // the next insertion to start; the same in every thread
    __syncthreads();
    for (;;) {
        const bool start = next < n && my_e < 0 && next == ahead;
        if (start) {
            my_e = next;
            p = n;
            mine = next_leaf;
            ahead += kTreeGroups;
            if (ahead < n) next_leaf = load_half(&leaf[ahead], h);
        }
        if (__any_sync(0xffffffffu, my_e >= 0)) {
            const bool on = my_e >= 0;
            // one level: p is an internal node on the path
            const Half old = on ? load_half(&nd[p - n].child[side], h) : none;
            Half u = old;  // the child's half with the new leaf
            u.a = kmin(old.a, mine.a);
            u.b = kmax(old.b, mine.b);
            if (h == 0) {
                u.c = kmin(old.c, mine.c);
                u.d = kmax(old.d, mine.d);
            }
            // the volume growth of each child's box by the new leaf's
            // (AABB::merge, AABB.cpp:38-49), in the lanes h = 0; ties go
            // right. A box that holds the new leaf's gives its own volume
            // again, and no growth: if every right child of the warp's does,
            // there is nothing to form.
            const bool same = u.a == old.a && u.b == old.b && u.c == old.c && u.d == old.d;
            const unsigned holds = __ballot_sync(0xffffffffu, same) >> base;
            const bool right_holds = (holds & 12u) == 12u;
            bool go_left = false;
            double vol = __longlong_as_double(__shfl_sync(0xffffffffu, old.c, lane | 1));
            if (__any_sync(0xffffffffu, on && !right_holds)) {
                const double e_a = __dsub_rn(odec(u.b), odec(u.a));
                const double e_b = __dsub_rn(odec(u.d), odec(u.c));  // h = 1: not used
                const double e_z = __shfl_sync(0xffffffffu, e_a, lane | 1);
                const double grown = __dmul_rn(__dmul_rn(e_a, e_b), e_z);
                const double growth = __dsub_rn(grown, vol);
                const double gl = __shfl_sync(0xffffffffu, growth, base);
                const double gr = __shfl_sync(0xffffffffu, growth, base + 2);
                go_left = gl < gr;
                vol = __shfl_sync(0xffffffffu, grown, lane & ~1);
            }
            const int chosen = go_left ? 0 : 1;
            const int c = (int)__shfl_sync(0xffffffffu, old.d, base + 2 * chosen + 1);
            const bool split = on && c < n;
            const int q = n + my_e - 1;
            if (on && side == chosen && (split || !((holds >> (2 * chosen) & 3u) == 3u))) {
                Half w = u;
                if (h == 1) {
                    w.c = __double_as_longlong(vol);
                    if (split) w.d = q;
                }
                store_half(&nd[p - n].child[side], h, w);
            }
            if (__any_sync(0xffffffffu, split)) {
                Half was;  // the leaf's half, in both lanes h
                was.a = __shfl_sync(0xffffffffu, old.a, base + 2 * chosen + h);
                was.b = __shfl_sync(0xffffffffu, old.b, base + 2 * chosen + h);
                was.c = __shfl_sync(0xffffffffu, old.c, base + 2 * chosen + h);
                was.d = __shfl_sync(0xffffffffu, old.d, base + 2 * chosen + h);
                if (split) {
                    // new leaf left, old leaf right
                    store_half(&nd[q - n].child[side], h, side == 0 ? mine : was);
                    const int l4 = lane & 3;
                    if (l4 == 0) parent[q] = p;
                    if (l4 == 1) parent[my_e] = q;
                    if (l4 == 2) parent[c] = q;
                }
            }
            if (split) {
                my_e = -1;
            } else if (on) {
                p = c;
                if ((lane & 3) == 3) atomicAdd(&extra[c - n], 1);
            }
        }
        next += __syncthreads_or(start) ? 1 : 0;
        if (next >= n && !__syncthreads_or(my_e >= 0)) break;
    }
}

// The same, a thread each: four times as many in flight, for trees so deep
// (a flat sheet's are ~1.4 times its side) that insertions wait for a free
// group more than shorter steps make up for.
__device__ void insert_by_threads(TreeNode* nd, const TreeChild* leaf, int* parent, int* extra, int n) {
    const int tid = threadIdx.x;
    int my_e = -1, p = n;
    TreeChild mine;
    int next = 2;
    __syncthreads();
    for (;;) {
        const bool start = next < n && my_e < 0 && next % kTreeThreads == tid;
        if (start) {
            my_e = next;
            p = n;
            mine = leaf[my_e];
        }
        if (my_e >= 0) {
            TreeNode* at = &nd[p - n];
            const TreeChild l = at->child[0], r = at->child[1];
            // a box that holds the new leaf's does not grow (the same
            // doubles), and a growth is never below 0
            bool go_left, grows;
            double vol;  // the chosen child's with the new leaf
            if (holds(r, mine)) {
                go_left = false;  // the right one's growth is 0
                grows = false;
                vol = r.vol;
            } else {
                const double vr = volume_k(joined(r, mine));
                if (holds(l, mine)) {
                    go_left = __dsub_rn(l.vol, l.vol) < __dsub_rn(vr, r.vol);  // (0, or NaN if it is infinite)
                    grows = !go_left;
                    vol = go_left ? l.vol : vr;
                } else {
                    const double vl = volume_k(joined(l, mine));
                    go_left = __dsub_rn(vl, l.vol) < __dsub_rn(vr, r.vol);
                    grows = true;
                    vol = go_left ? vl : vr;
                }
            }
            const TreeChild was = go_left ? l : r;
            const int c = (int)was.id;
            const bool split = c < n;
            const int q = n + my_e - 1;
            if (grows || split) {
                TreeChild w = joined(was, mine);
                w.vol = vol;
                w.id = split ? q : c;
                at->child[go_left ? 0 : 1] = w;
            }
            if (split) {
                // new leaf left, old leaf right
                mine.id = my_e;  // (needs no register until here)
                nd[q - n].child[0] = mine;
                nd[q - n].child[1] = was;
                parent[q] = p;
                parent[my_e] = q;
                parent[c] = q;
                my_e = -1;
            } else {
                p = c;
                atomicAdd(&extra[c - n], 1);
            }
        }
        next += __syncthreads_or(start) ? 1 : 0;
        if (next >= n && !__syncthreads_or(my_e >= 0)) break;
    }
}

// One CTA per tree, of those that are inserted by threads or by lanes.
template <bool BY_THREADS>
__global__ void __launch_bounds__(kTreeThreads) k_tree_build(const Box6* __restrict__ boxes, const int* __restrict__ jobs,
                                                            TreeNode* nodes_all, TreeChild* leaves_all, int* parent_all,
                                                            int* extra_all, int* root_out, double* vol_out) {
    const int e0 = jobs[3 * blockIdx.x + 1], n = jobs[3 * blockIdx.x + 2];
    if ((n > kTreeLaneMax) != BY_THREADS) return;
    TreeNode* nd = nodes_all + e0;         // internal node q is nd[q - n]
    TreeChild* leaf = leaves_all + e0;
    int* parent = parent_all + 2 * (size_t)e0;
    int* extra = extra_all + e0;           // node q has 2 + extra[q - n] leaves
    const int tid = threadIdx.x;
    for (int e = tid; e < n; e += kTreeThreads) {
        const Box6 b = boxes[e0 + e];
        TreeChild L;
        L.xlo = okey(b.lo[0]); L.xhi = okey(b.hi[0]);
        L.ylo = okey(b.lo[1]); L.yhi = okey(b.hi[1]);
        L.zlo = okey(b.lo[2]); L.zhi = okey(b.hi[2]);
        L.vol = volume_k(L);
        L.id = e;
        leaf[e] = L;
        parent[e] = -1;
        extra[e] = 0;
    }
    __syncthreads();
    if (n < 2) {
        if (tid == 0) {
            root_out[blockIdx.x] = n - 1;
            vol_out[blockIdx.x] = n == 1 ? leaf[0].vol : 0.0;
        }
        return;
    }
    if (tid == 0) {  // insertion 1 splits the root leaf 0 into node n
        nd[0].child[0] = leaf[1];
        nd[0].child[1] = leaf[0];
        parent[n] = -1;
        parent[0] = parent[1] = n;
    }
    if (BY_THREADS)
        insert_by_threads(nd, leaf, parent, extra, n);
    else
        insert_by_lanes(nd, leaf, parent, extra, n);
    if (tid == 0) {
        root_out[blockIdx.x] = n;
        vol_out[blockIdx.x] = volume_k(joined(nd[0].child[0], nd[0].child[1]));
    }
}

// Inorder rank of each leaf: the leaves of every left sibling on its path.
__global__ void k_tree_ranks(const int* __restrict__ jobs, const TreeNode* __restrict__ nodes_all,
                             const int* __restrict__ parent_all, const int* __restrict__ extra_all, int* rank) {
    const int e0 = jobs[3 * blockIdx.y + 1], n = jobs[3 * blockIdx.y + 2];
    const TreeNode* nd = nodes_all + e0;
    const int* parent = parent_all + 2 * (size_t)e0;
    const int* extra = extra_all + e0;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x) {
        int r = 0, x = e;
        for (int a = parent[x]; a >= 0; x = a, a = parent[a]) {
            const int lft = (int)nd[a - n].child[0].id;
            if (lft != x) r += lft < n ? 1 : 2 + extra[lft - n];
        }
        rank[e0 + e] = r;
    }
}

}  // namespace

size_t tree_scratch_bytes(long long ne) {
    return (size_t)(ne + 1) * (sizeof(TreeNode) + sizeof(TreeChild) + 3 * sizeof(int));
}

void tree_configure() {
    // Once per device: kernels stay loaded, and asking for these takes
    // 0.25 ms each time, loaded or not. (After a device reset they are loaded
    // at their first launch again.)
    static std::atomic<unsigned long long> loaded{0};
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess || device > 63) return;
    if (loaded.load() >> device & 1) return;
    cudaFuncAttributes a;
    if (cudaFuncGetAttributes(&a, k_tree_build<false>) == cudaSuccess &&
        cudaFuncGetAttributes(&a, k_tree_build<true>) == cudaSuccess &&
        cudaFuncGetAttributes(&a, k_tree_ranks) == cudaSuccess)
        loaded.fetch_or(1ull << device);
}

void tree_order_gpu(const Box6* boxes, const int* jobs, int njobs, int max_ne, void* scratch, long long ne_total,
                    int* rank, int* root_out, double* vol_out, cudaStream_t s) {
    if (njobs <= 0) return;
    TreeNode* nodes = static_cast<TreeNode*>(scratch);
    TreeChild* leaves = reinterpret_cast<TreeChild*>(nodes + ne_total + 1);
    int* parent = reinterpret_cast<int*>(leaves + ne_total + 1);
    int* extra = parent + 2 * (ne_total + 1);
    k_tree_build<false><<<njobs, kTreeThreads, 0, s>>>(boxes, jobs, nodes, leaves, parent, extra, root_out, vol_out);
    if (max_ne > kTreeLaneMax)
        k_tree_build<true><<<njobs, kTreeThreads, 0, s>>>(boxes, jobs, nodes, leaves, parent, extra, root_out, vol_out);
    const int bx = std::max(1, std::min((max_ne + 255) / 256, 1024));
    k_tree_ranks<<<dim3(bx, njobs), 256, 0, s>>>(jobs, nodes, parent, extra, rank);
}

}  // namespace ccg
