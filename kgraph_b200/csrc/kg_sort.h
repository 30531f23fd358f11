// Introsort exactly as the GNU C++ library's std::sort performs it, for the
// three places where the reference sorts Neighbor records by distance alone
// and the order of equal-distance records is therefore fixed by the library's
// algorithm, not by the data:
//   kgraph.cpp:476  sort(knn.begin(), knn.begin() + L)   -- search seed pool
//   kgraph.cpp:697  std::sort(v.begin(), v.end())         -- reverse edges
//   kgraph.cpp:793  sort(pool.begin(), pool.begin() + L)  -- build init pool
// Reproducing the same permutation on the GPU keeps search bit-identical to
// the reference even when distances tie (integer-valued data ties often).
//
// The algorithm is the published introsort (Musser 1997) with the GNU
// choices: depth limit 2*floor(log2 n); partitions while more than 16
// elements remain, recursing on the right part; median-of-three of
// (first+1, mid, last-1) moved to first; unguarded Hoare partition; heapsort
// (make_heap + sort_heap) when the depth limit is spent; a final insertion
// sort (guarded for the first 16, unguarded after).  Comparisons are `a < b`
// on the key only.
//
// gnu_sort is written as a template over an accessor so the same code runs in a CUDA
// thread (device) and in the host tests that check it against std::sort;
// warp_gnu_sort is the same sort by a warp.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define KG_HD __host__ __device__ __forceinline__
#else
#define KG_HD inline
#endif

namespace kgb {

// A: struct with  float key(int i); void swap(int i, int j);
//                 Rec get(int i); void put(int i, Rec r); float rkey(Rec r)
template <typename A>
KG_HD void gs_move_median_to_first(A &a, int result, int x, int y, int z) {
    if (a.key(x) < a.key(y)) {
        if (a.key(y) < a.key(z)) a.swap(result, y);
        else if (a.key(x) < a.key(z)) a.swap(result, z);
        else a.swap(result, x);
    } else if (a.key(x) < a.key(z)) a.swap(result, x);
    else if (a.key(y) < a.key(z)) a.swap(result, z);
    else a.swap(result, y);
}

template <typename A>
KG_HD int gs_unguarded_partition(A &a, int first, int last, int pivot) {
    while (true) {
        while (a.key(first) < a.key(pivot)) ++first;
        --last;
        while (a.key(pivot) < a.key(last)) --last;
        if (!(first < last)) return first;
        a.swap(first, last);
        ++first;
    }
}

template <typename A, typename R>
KG_HD void gs_push_heap(A &a, int first, int hole, int top, R value) {
    int parent = (hole - 1) / 2;
    while (hole > top && a.key(first + parent) < a.rkey(value)) {
        a.put(first + hole, a.get(first + parent));
        hole = parent;
        parent = (hole - 1) / 2;
    }
    a.put(first + hole, value);
}

template <typename A, typename R>
KG_HD void gs_adjust_heap(A &a, int first, int hole, int len, R value) {
    const int top = hole;
    int second = hole;
    while (second < (len - 1) / 2) {
        second = 2 * (second + 1);
        if (a.key(first + second) < a.key(first + (second - 1))) second--;
        a.put(first + hole, a.get(first + second));
        hole = second;
    }
    if ((len & 1) == 0 && second == (len - 2) / 2) {
        second = 2 * (second + 1);
        a.put(first + hole, a.get(first + (second - 1)));
        hole = second - 1;
    }
    gs_push_heap(a, first, hole, top, value);
}

template <typename A>
KG_HD void gs_heapsort(A &a, int first, int last) {
    int len = last - first;
    if (len >= 2) {   // make_heap
        int parent = (len - 2) / 2;
        while (true) {
            auto v = a.get(first + parent);
            gs_adjust_heap(a, first, parent, len, v);
            if (parent == 0) break;
            parent--;
        }
    }
    while (last - first > 1) {   // sort_heap: pop_heap(first, last, last)
        --last;
        auto v = a.get(last);
        a.put(last, a.get(first));
        gs_adjust_heap(a, first, 0, last - first, v);
    }
}

template <typename A>
KG_HD void gs_unguarded_linear_insert(A &a, int last) {
    auto val = a.get(last);
    int next = last - 1;
    while (a.rkey(val) < a.key(next)) {
        a.put(last, a.get(next));
        last = next;
        --next;
    }
    a.put(last, val);
}

template <typename A>
KG_HD void gs_insertion_sort(A &a, int first, int last) {
    if (first == last) return;
    for (int i = first + 1; i != last; ++i) {
        if (a.key(i) < a.key(first)) {
            auto val = a.get(i);
            for (int j = i; j > first; --j) a.put(j, a.get(j - 1));
            a.put(first, val);
        } else {
            gs_unguarded_linear_insert(a, i);
        }
    }
}

KG_HD int gs_lg(int n) {
    int r = 0;
    while (n > 1) { n >>= 1; ++r; }
    return r;
}

template <typename A>
KG_HD void gnu_sort(A &a, int first, int last) {
    if (first == last) return;
    // __introsort_loop with an explicit stack.  The recursive form is
    //   while (n > 16) { if (!depth) heapsort, return; --depth;
    //                    cut = partition; recurse(cut, last, depth); last = cut; }
    // so the right part is finished before the left part continues with the
    // same (decremented) depth: the left frame is pushed under the right one.
    struct Frame { int first, last, depth; };
    Frame stack[72];
    int sp = 0;
    stack[sp++] = Frame{first, last, gs_lg(last - first) * 2};
    while (sp > 0) {
        Frame f = stack[--sp];
        if (f.last - f.first <= 16) continue;
        if (f.depth == 0) { gs_heapsort(a, f.first, f.last); continue; }
        int depth = f.depth - 1;
        int mid = f.first + (f.last - f.first) / 2;
        gs_move_median_to_first(a, f.first, f.first + 1, mid, f.last - 1);
        int cut = gs_unguarded_partition(a, f.first + 1, f.last, f.first);
        stack[sp++] = Frame{f.first, cut, depth};
        stack[sp++] = Frame{cut, f.last, depth};
    }
    // __final_insertion_sort
    if (last - first > 16) {
        gs_insertion_sort(a, first, first + 16);
        for (int i = first + 16; i != last; ++i) gs_unguarded_linear_insert(a, i);
    } else {
        gs_insertion_sort(a, first, last);
    }
}

#ifdef __CUDACC__
// gnu_sort of n <= WARP_SORT_MAX records (key d[i], payload id[i] and, unless
// null, m[i]; shared or global memory) by one warp: the same permutation, ties
// included.  tmp: WARP_SORT_TMP words of the warp's own shared memory; nan:
// whether a lane has met a NaN among the keys.
//  * Which ranges are partitioned, and around which pivots, depends only on the
//    data, and ranges are disjoint, so their order is free.
//  * A Hoare partition swaps the t-th stop of its left scan (a record not below
//    the pivot) with the t-th stop of its right scan (one not above it) while
//    they have not crossed; the swaps lie behind both scans.  So stops are found
//    32 at a time, paired by rank and swapped in parallel; the cut is the next
//    left stop, or the last right stop swapped if that comes first.
//  * The final insertion sort is stable, and ranges that were left have at most
//    16 records: a record's place is its own plus the smaller ones up to 15
//    behind it minus the larger ones up to 15 before it.  Among NaN a place
//    is not a record's own any more: there one lane inserts.
// A range whose depth limit is spent is heap-sorted by one lane.
constexpr int WARP_SORT_MAX = 8191, WARP_SORT_TMP = 48;

struct WarpSortAcc {   // the serial accessor, for the heap sort
    float *d; uint32_t *i, *m;
    struct Rec { float d; uint32_t i, m; };
    __device__ float key(int x) const { return d[x]; }
    __device__ void swap(int x, int y) const {
        const float td = d[x]; d[x] = d[y]; d[y] = td;
        const uint32_t ti = i[x]; i[x] = i[y]; i[y] = ti;
        if (m) { const uint32_t tm = m[x]; m[x] = m[y]; m[y] = tm; }
    }
    __device__ Rec get(int x) const { return Rec{d[x], i[x], m ? m[x] : 0u}; }
    __device__ void put(int x, Rec r) const { d[x] = r.d; i[x] = r.i; if (m) m[x] = r.m; }
    __device__ float rkey(Rec r) const { return r.d; }
};

__device__ inline int warp_partition(float *d, uint32_t *id, uint32_t *m, int f, int l, uint8_t *rank, int lane) {
    const unsigned ALL = 0xFFFFFFFFu, below = (1u << lane) - 1u;
    const float piv = d[f];
    int lp = f + 1, rp = l - 1;      // next positions to scan
    int lb = 0, rb = 0, rlast = l;   // bases of the scanned pieces; the last right stop swapped
    unsigned ml = 0, mr = 0;         // their stops not yet paired
    for (;;) {
        while (!ml) {
            if (lp >= rlast) return rlast;
            lb = lp;
            const int p = lb + lane;
            ml = __ballot_sync(ALL, p < l && !(d[p] < piv));
            lp += 32;
        }
        while (!mr && rp > f) {
            rb = rp;
            const int p = rb - lane;
            mr = __ballot_sync(ALL, p > f && !(piv < d[p]));
            rp -= 32;
        }
        if (!mr) return min(lb + __ffs(ml) - 1, rlast);
        const int t = min(__popc(ml), __popc(mr));
        if ((ml >> lane) & 1u) rank[__popc(ml & below)] = (uint8_t)lane;
        if ((mr >> lane) & 1u) rank[32 + __popc(mr & below)] = (uint8_t)lane;
        __syncwarp();
        int L = 0, R = 0;
        if (lane < t) { L = lb + rank[lane]; R = rb - rank[32 + lane]; }
        const unsigned okm = __ballot_sync(ALL, lane < t && L < R);
        if ((okm >> lane) & 1u) {
            const float td = d[L]; d[L] = d[R]; d[R] = td;
            const uint32_t ti = id[L]; id[L] = id[R]; id[R] = ti;
            if (m) { const uint32_t tm = m[L]; m[L] = m[R]; m[R] = tm; }
        }
        __syncwarp();
        const int n = __popc(okm);
        if (n) rlast = __shfl_sync(ALL, R, n - 1);
        if (n < t) return min(__shfl_sync(ALL, L, n), rlast);
        ml = __ballot_sync(ALL, ((ml >> lane) & 1u) && __popc(ml & below) >= t);
        mr = __ballot_sync(ALL, ((mr >> lane) & 1u) && __popc(mr & below) >= t);
    }
}

__device__ inline void warp_gnu_sort(float *d, uint32_t *id, uint32_t *m, int n, uint32_t *tmp, bool nan, int lane) {
    uint8_t *rank = reinterpret_cast<uint8_t *>(tmp + 32);   // 64 bytes behind 32 frames
    int sp = 0, f = 0, l = n, depth = n > 1 ? 2 * (31 - __clz(n)) : 0;
    for (;;) {
        if (l - f <= 16 || depth == 0) {
            if (l - f > 16) {
                if (lane == 0) { WarpSortAcc a{d, id, m}; gs_heapsort(a, f, l); }
                __syncwarp();
            }
            if (sp == 0) break;
            const uint32_t w = tmp[--sp];
            __syncwarp();
            f = (int)(w & 8191u); l = (int)((w >> 13) & 8191u); depth = (int)(w >> 26);
            continue;
        }
        --depth;
        const int mid = f + (l - f) / 2;
        const float a = d[f + 1], b = d[mid], c = d[l - 1];
        int at;   // gs_move_median_to_first
        if (a < b) at = b < c ? mid : a < c ? l - 1 : f + 1;
        else at = a < c ? f + 1 : b < c ? l - 1 : mid;
        __syncwarp();
        if (lane == 0) { WarpSortAcc s{d, id, m}; s.swap(f, at); }
        __syncwarp();
        const int cut = warp_partition(d, id, m, f, l, rank, lane);
        if (cut - f > 16) {
            if (lane == 0) tmp[sp] = (uint32_t)f | (uint32_t)cut << 13 | (uint32_t)depth << 26;
            ++sp;
            __syncwarp();
        }
        f = cut;
    }
    if (__any_sync(0xFFFFFFFFu, nan)) {
        if (lane == 0) {
            WarpSortAcc a{d, id, m};
            gs_insertion_sort(a, 0, n < 16 ? n : 16);
            for (int i = 16; i < n; ++i) {   // gs_unguarded_linear_insert, with a guard
                const WarpSortAcc::Rec val = a.get(i);
                int at = i;
                for (; at > 0 && val.d < d[at - 1]; --at) a.put(at, a.get(at - 1));
                a.put(at, val);
            }
        }
        __syncwarp();
        return;
    }
    // the final insertion sort; a piece of 32 is written once the next one has been ranked
    float pd = 0.f;
    uint32_t pi = 0, pm = 0;
    int pp = -1;
    for (int base = 0; base < n + 32; base += 32) {
        const int p = base + lane;
        float v = 0.f;
        uint32_t vi = 0, vm = 0;
        int np = -1;
        if (p < n) {
            v = d[p];
            vi = id[p];
            if (m) vm = m[p];
            np = p;
#pragma unroll 5
            for (int o = 1; o <= 15; ++o) {
                if (p + o < n && d[p + o] < v) ++np;
                if (p - o >= 0 && v < d[p - o]) --np;
            }
        }
        __syncwarp();
        if (pp >= 0) { d[pp] = pd; id[pp] = pi; if (m) m[pp] = pm; }
        __syncwarp();
        pd = v; pi = vi; pm = vm; pp = np;
    }
}
#endif

}  // namespace kgb
