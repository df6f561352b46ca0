// Device primitives: exclusive scan and a stable LSD radix sort of
// (64-bit key, 32-bit value) pairs with 8-bit digits. Hand-written (no CUB):
// the sort ranks keys inside a tile with __match_any_sync and per-warp digit
// counts in shared memory, so equal digits keep their input order.
#include "cc_launch.h"

namespace ccg {

long long g_kernel_launches = 0;

namespace {

constexpr int kScanThreads = 1024;
constexpr int kScanItems = 2;
constexpr int kScanTile = kScanThreads * kScanItems;

__device__ __forceinline__ int warp_incl_scan(int v) {
    int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
    }
    return v;
}

// Exclusive scan of one tile per block; block totals to sums[blockIdx.x].
__global__ void k_scan_tile(const int* in, int* out, int n, int* sums) {
    __shared__ int wsum[kScanThreads / 32];
    int base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
    int v[kScanItems];
    int local = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        v[k] = (base + k < n) ? in[base + k] : 0;
        local += v[k];
    }
    int incl = warp_incl_scan(local);
    int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        int s = (lane < kScanThreads / 32) ? wsum[lane] : 0;
        s = warp_incl_scan(s);
        if (lane < kScanThreads / 32) wsum[lane] = s;
    }
    __syncthreads();
    int run = incl - local + (warp > 0 ? wsum[warp - 1] : 0);
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        if (base + k < n) out[base + k] = run;
        run += v[k];
    }
    if (threadIdx.x == kScanThreads - 1 && sums) sums[blockIdx.x] = run;
}

__global__ void k_scan_add(int* out, int n, const int* block_off) {
    int i = blockIdx.x * kScanTile + threadIdx.x;
    int add = block_off[blockIdx.x];
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        int j = i + k * kScanThreads;
        if (j < n) out[j] += add;
    }
}

inline int ceil_div(int a, int b) { return (a + b - 1) / b; }

// Scans of up to kScanOne elements take one block, a run of consecutive
// elements per thread: one launch instead of three (~1.2 us each). At 32,768
// elements that serial run costs more than it saves (a build of 136,000
// leaves 0.22 -> 0.23 ms, of 196,000 0.265 -> 0.313 ms).
constexpr int kScanOne = 4 * kScanTile;
__global__ void __launch_bounds__(kScanThreads) k_scan_one(const int* in, int* out, int n) {
    __shared__ int wsum[kScanThreads / 32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int per = (n + kScanThreads - 1) / kScanThreads;  // consecutive elements per thread
    const int i0 = threadIdx.x * per, i1 = i0 + per < n ? i0 + per : n;
    int local = 0;
    for (int i = i0; i < i1; ++i) local += in[i];
    const int incl = warp_incl_scan(local);
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    if (warp == 0) wsum[lane] = warp_incl_scan(wsum[lane]);
    __syncthreads();
    int run = incl - local + (warp > 0 ? wsum[warp - 1] : 0);
    for (int i = i0; i < i1; ++i) {
        const int v = in[i];
        out[i] = run;
        run += v;
    }
}

// Levels of block sums for an n-element scan.
size_t scan_levels_bytes(int n) {
    size_t bytes = 0;
    while (n > kScanTile) {
        n = ceil_div(n, kScanTile);
        bytes += ((size_t)n * sizeof(int) + 255) & ~(size_t)255;
    }
    return bytes;
}

void scan_rec(const int* in, int* out, int n, char* temp, cudaStream_t s) {
    int nb = ceil_div(n, kScanTile);
    if (nb <= 1) {
        count_launch(), k_scan_tile<<<1, kScanThreads, 0, s>>>(in, out, n, nullptr);
        return;
    }
    if (n <= kScanOne) {
        count_launch(), k_scan_one<<<1, kScanThreads, 0, s>>>(in, out, n);
        return;
    }
    int* sums = (int*)temp;
    char* rest = temp + (((size_t)nb * sizeof(int) + 255) & ~(size_t)255);
    count_launch(), k_scan_tile<<<nb, kScanThreads, 0, s>>>(in, out, n, sums);
    scan_rec(sums, sums, nb, rest, s);
    count_launch(), k_scan_add<<<nb, kScanThreads, 0, s>>>(out, n, sums);
}

// ------------------------------------------------------------------ sort
constexpr int kSortThreads = 256;
constexpr int kSortItems = 8;
constexpr int kSortTile = kSortThreads * kSortItems;
constexpr int kRadix = 256;

// dn (may be null): the number of pairs to sort is min(*dn, n).
__device__ __forceinline__ int sort_count(const int* dn, int n) {
    if (!dn) return n;
    const int m = *dn;
    return m < n ? (m > 0 ? m : 0) : n;
}

__global__ void k_radix_hist(const unsigned long long* keys, int n, int shift, int* hist, int nblocks,
                             const int* dn) {
    n = sort_count(dn, n);
    __shared__ int h[kRadix];
    h[threadIdx.x] = 0;
    __syncthreads();
    int base = blockIdx.x * kSortTile;
#pragma unroll
    for (int r = 0; r < kSortItems; ++r) {
        int i = base + r * kSortThreads + threadIdx.x;
        if (i < n) atomicAdd(&h[(keys[i] >> shift) & 0xff], 1);
    }
    __syncthreads();
    hist[threadIdx.x * nblocks + blockIdx.x] = h[threadIdx.x];
}

__global__ void k_radix_scatter(const unsigned long long* keys, const unsigned int* vals, unsigned long long* okeys,
                                unsigned int* ovals, int n, int shift, const int* off, int nblocks, const int* dn) {
    n = sort_count(dn, n);
    __shared__ int run[kRadix];
    __shared__ int wcnt[kSortThreads / 32][kRadix];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned lt_mask = (1u << lane) - 1u;
    run[threadIdx.x] = 0;
    int base = blockIdx.x * kSortTile;
    for (int r = 0; r < kSortItems; ++r) {
#pragma unroll
        for (int w = 0; w < kSortThreads / 32; ++w) wcnt[w][threadIdx.x] = 0;
        __syncthreads();
        int i = base + r * kSortThreads + threadIdx.x;
        bool valid = i < n;
        unsigned long long k = valid ? keys[i] : 0ull;
        int d = valid ? (int)((k >> shift) & 0xff) : kRadix;
        unsigned peers = __match_any_sync(0xffffffffu, d);
        int lrank = __popc(peers & lt_mask);
        if (valid && lrank == 0) wcnt[warp][d] = __popc(peers);
        __syncthreads();
        if (valid) {
            int pre = run[d] + lrank;
            for (int w = 0; w < warp; ++w) pre += wcnt[w][d];
            int pos = off[d * nblocks + blockIdx.x] + pre;
            okeys[pos] = k;
            ovals[pos] = vals[i];
        }
        __syncthreads();
        int tot = 0;
#pragma unroll
        for (int w = 0; w < kSortThreads / 32; ++w) tot += wcnt[w][threadIdx.x];
        run[threadIdx.x] += tot;
    }
}

// Small sorts in one CTA: up to kSmallSort pairs, each key extended by its
// input position (so the keys are distinct and a bitonic network gives the
// stable order). Thread t holds elements t * ITEMS .. t * ITEMS + ITEMS - 1
// in registers: partners of the same thread meet there, of the same warp by
// shuffle, and only the wider strides go through shared memory - 15 of 78
// stages for 4,096 elements, where a barrier per stage took 43 us (now 25 us).
constexpr int kSmallThreads = 1024;
constexpr int kIdxBits = 13;
static_assert(1 << kIdxBits == kSmallSort, "an index per pair");
constexpr size_t kSmallBytes = (size_t)kSmallSort * (sizeof(unsigned long long) + sizeof(unsigned int));

template <int ITEMS, int J>
__device__ __forceinline__ void bitonic_in_thread(unsigned long long (&v)[ITEMS], int e0, int k) {
    if constexpr (J < ITEMS) {
#pragma unroll
        for (int r = 0; r < ITEMS; ++r)
            if ((r & J) == 0) {
                const unsigned long long a = v[r], b = v[r | J];
                if ((a > b) == (((e0 + r) & k) == 0)) {
                    v[r] = b;
                    v[r | J] = a;
                }
            }
    }
}

// The first P elements (a power of two, at least 32; P = 1024 * ITEMS for
// ITEMS > 1) of the whole CTA in ascending order; x: ITEMS * 1024 slots.
template <int ITEMS>
__device__ __forceinline__ void cta_bitonic(unsigned long long (&v)[ITEMS], int P, unsigned long long* x) {
    const int tid = threadIdx.x, e0 = tid * ITEMS;
    for (int k = 2; k <= P; k <<= 1)
        for (int j = k >> 1; j > 0; j >>= 1) {
            if (j >= ITEMS) {
                const int d = j / ITEMS;  // partner threads' distance
                const bool keep_min = ((e0 & k) == 0) == ((tid & d) == 0);
                if (d >= 32) {
                    __syncthreads();
#pragma unroll
                    for (int r = 0; r < ITEMS; ++r) x[r * kSmallThreads + tid] = v[r];
                    __syncthreads();
                }
#pragma unroll
                for (int r = 0; r < ITEMS; ++r) {
                    const unsigned long long o =
                        d >= 32 ? x[r * kSmallThreads + (tid ^ d)] : __shfl_xor_sync(0xffffffffu, v[r], d);
                    v[r] = (o < v[r]) == keep_min ? o : v[r];
                }
            } else if (j == 4) {
                bitonic_in_thread<ITEMS, 4>(v, e0, k);
            } else if (j == 2) {
                bitonic_in_thread<ITEMS, 2>(v, e0, k);
            } else {
                bitonic_in_thread<ITEMS, 1>(v, e0, k);
            }
        }
}

template <int ITEMS>
__device__ __forceinline__ void sort_small(unsigned long long* keys, unsigned int* vals, int m, int P,
                                           unsigned long long* s_k, unsigned int* s_v) {
    const int tid = threadIdx.x;
    unsigned long long v[ITEMS];
    for (int i = tid; i < m; i += kSmallThreads) s_v[i] = vals[i];
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) {
        const int e = tid * ITEMS + r;
        v[r] = e < m ? (keys[e] << kIdxBits) | (unsigned long long)e : ~0ull;
    }
    cta_bitonic<ITEMS>(v, P, s_k);
    __syncthreads();  // every key and value has been read
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) {
        const int e = tid * ITEMS + r;
        if (e < m) {
            keys[e] = v[r] >> kIdxBits;
            vals[e] = s_v[v[r] & (kSmallSort - 1)];
        }
    }
}

// Sorts the first m = min(*dn, n) pairs when m <= kSmallSort and sets *eff
// to 0; otherwise leaves them and sets *eff = m.
__global__ void __launch_bounds__(kSmallThreads) k_sort_small(unsigned long long* keys, unsigned int* vals,
                                                             const int* dn, int n, int* eff) {
    extern __shared__ unsigned long long s_k[];
    unsigned int* s_v = reinterpret_cast<unsigned int*>(s_k + kSmallSort);
    const int m = sort_count(dn, n);
    if (m > kSmallSort) {
        if (threadIdx.x == 0 && eff) *eff = m;
        return;
    }
    int P = 32;
    while (P < m) P <<= 1;
    if (P <= 1024)
        sort_small<1>(keys, vals, m, P, s_k, s_v);
    else if (P == 2048)
        sort_small<2>(keys, vals, m, P, s_k, s_v);
    else if (P == 4096)
        sort_small<4>(keys, vals, m, P, s_k, s_v);
    else
        sort_small<8>(keys, vals, m, P, s_k, s_v);
    if (threadIdx.x == 0 && eff) *eff = 0;
}

}  // namespace

cudaError_t small_sort_ready() {
    return cudaFuncSetAttribute(k_sort_small, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmallBytes);
}

void sort_pairs_dev(unsigned long long* keys, unsigned int* vals, const int* dn, int cap, int bits, void* temp,
                    int* eff, cudaStream_t s, bool small, bool general) {
    if (cap <= 1 || bits <= 0) return;
    if (small)
        count_launch(), k_sort_small<<<1, kSmallThreads, kSmallBytes, s>>>(keys, vals, dn, cap, eff);
    if (general) radix_sort_pairs_dev(keys, vals, small ? eff : dn, cap, bits, temp, s);
}

size_t scan_temp_bytes(int n) { return scan_levels_bytes(n) + 256; }

void exclusive_scan(const int* in, int* out, int n, void* temp, cudaStream_t s) {
    if (n > 0) scan_rec(in, out, n, (char*)temp, s);
}

size_t radix_sort_temp_bytes(int n) {
    int nb = ceil_div(n > 0 ? n : 1, kSortTile);
    size_t hist = (size_t)kRadix * nb;
    auto al = [](size_t b) { return (b + 255) & ~(size_t)255; };
    return al((size_t)n * sizeof(unsigned long long)) + al((size_t)n * sizeof(unsigned int)) +
           2 * al(hist * sizeof(int)) + al(scan_temp_bytes((int)hist));
}

void radix_sort_pairs(unsigned long long* keys, unsigned int* vals, int n, int bits, void* temp, cudaStream_t s) {
    // up to kSmallSort pairs in one CTA: the same stable order in one launch
    // (a 33 x 33 sheet's build: 0.13 -> 0.085 ms)
    if (n > 1 && n <= kSmallSort && bits <= 64 - kIdxBits && small_sort_ready() == cudaSuccess) {
        count_launch(), k_sort_small<<<1, kSmallThreads, kSmallBytes, s>>>(keys, vals, nullptr, n, nullptr);
        return;
    }
    radix_sort_pairs_dev(keys, vals, nullptr, n, bits, temp, s);
}

void radix_sort_pairs_dev(unsigned long long* keys, unsigned int* vals, const int* dn, int n, int bits, void* temp,
                          cudaStream_t s) {
    if (n <= 1 || bits <= 0) return;
    int nb = ceil_div(n, kSortTile);
    size_t hist_n = (size_t)kRadix * nb;
    auto al = [](size_t b) { return (b + 255) & ~(size_t)255; };
    char* t = (char*)temp;
    unsigned long long* k2 = (unsigned long long*)t;
    t += al((size_t)n * sizeof(unsigned long long));
    unsigned int* v2 = (unsigned int*)t;
    t += al((size_t)n * sizeof(unsigned int));
    int* hist = (int*)t;
    t += al(hist_n * sizeof(int));
    int* off = (int*)t;
    t += al(hist_n * sizeof(int));
    void* stemp = t;
    unsigned long long* ka = keys;
    unsigned int* va = vals;
    unsigned long long* kb = k2;
    unsigned int* vb = v2;
    int passes = (bits + 7) / 8;
    for (int ps = 0; ps < passes; ++ps) {
        int shift = ps * 8;
        count_launch(), k_radix_hist<<<nb, kSortThreads, 0, s>>>(ka, n, shift, hist, nb, dn);
        exclusive_scan(hist, off, (int)hist_n, stemp, s);
        count_launch(), k_radix_scatter<<<nb, kSortThreads, 0, s>>>(ka, va, kb, vb, n, shift, off, nb, dn);
        unsigned long long* tk = ka; ka = kb; kb = tk;
        unsigned int* tv = va; va = vb; vb = tv;
    }
    if (ka != keys) {
        cudaMemcpyAsync(keys, ka, (size_t)n * sizeof(unsigned long long), cudaMemcpyDeviceToDevice, s);
        cudaMemcpyAsync(vals, va, (size_t)n * sizeof(unsigned int), cudaMemcpyDeviceToDevice, s);
    }
}

}  // namespace ccg
