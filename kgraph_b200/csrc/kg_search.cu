// Batched graph-walk search: KGraphImpl::search (kgraph.cpp:423-564) for a
// whole batch of queries in one persistent launch.
//
// Layout.  One warp owns one query at a time and pulls the next query index
// from a global counter, so queries with uneven K and P balance themselves.
// The warp keeps the query vector and its candidate pool (K+P+1 entries:
// dist, id|flag, m|M<<16 -- the reference's NeighborX) in shared memory, and
// a private N-bit visited set in global memory (the reference's
// dynamic_bitset, kgraph.cpp:438).  The compact pool (CP) packs an entry
// into 8 bytes -- dist, and id (the bits N needs) | expansion progress m/S
// (the remaining bits up to 31) | flag -- and reads M again from the node's
// {M, degree} when the entry is expanded, together with its first adjacency
// window: a third fewer bytes per entry, so more queries fit on an SM where
// the pool limits residency.
//
// Exactness.  The walk is the reference's, step for step: the same P seeds
// for every query (host mt19937(seed) + GenRandom, kgraph.cpp:444-453), the
// seed pool sorted by the GNU introsort (kgraph.cpp:476), neighbours visited
// in adjacency order S at a time, each inserted with UpdateKnnList
// semantics, k reset to the insert position (kgraph.cpp:478-514).  The
// distances of a run of neighbours -- of several batches of S -- are computed
// in parallel (they are pure), then merged up to the batch after which the
// reference turns to another entry, which is what its interleaved loop
// produces.  With the canonical distance this reproduces the reference's ids,
// distances, result count and SearchInfo.cost exactly.
#include <cuda_fp16.h>
#include <cuda_fp8.h>
#include <algorithm>
#include "kg_common.cuh"
#include "kg_warp.cuh"
#include "kg_sort.h"
#include "kg_search.h"

namespace kgb {

namespace {

struct WarpSmem {
    float *q;          // ld floats
    float *pd;         // cap
    uint32_t *pid;     // cap   id | FLAG_BIT
    uint32_t *pm;      // cap   m | (M << 16)
    float *rd;         // rcap  (T > 1 result merge)
    uint32_t *rid;     // rcap
    float *cd;         // 32    batch distances (seeds, brute force)
    uint32_t *cid;     // 32    batch ids
    // the walk's use of the same 96 words: a window's unvisited neighbours in order
    uint32_t *lid;     // 64    ids
    uint8_t *lpos;     // 64    positions in the window
    uint8_t *lsel;     // 32    group lanes the compressed-row filter kept
};
constexpr uint32_t LIST = 64;   // entries of lid / lpos

template <int CP>
__device__ __forceinline__ WarpSmem carve(char *base, const SearchArgs &a) {
    WarpSmem s;
    char *p = base;
    s.q = reinterpret_cast<float *>(p); p += sizeof(float) * a.D.ld;
    s.pd = reinterpret_cast<float *>(p); p += sizeof(float) * a.cap;
    s.pid = reinterpret_cast<uint32_t *>(p); p += sizeof(uint32_t) * a.cap;
    s.pm = nullptr;
    if constexpr (!CP) { s.pm = reinterpret_cast<uint32_t *>(p); p += sizeof(uint32_t) * a.cap; }
    s.rd = reinterpret_cast<float *>(p); p += sizeof(float) * a.rcap;
    s.rid = reinterpret_cast<uint32_t *>(p); p += sizeof(uint32_t) * a.rcap;
    s.cd = reinterpret_cast<float *>(p);
    s.cid = reinterpret_cast<uint32_t *>(p + sizeof(float) * 32);
    s.lid = reinterpret_cast<uint32_t *>(p); p += sizeof(uint32_t) * LIST;
    s.lpos = reinterpret_cast<uint8_t *>(p); p += LIST;
    s.lsel = reinterpret_cast<uint8_t *>(p);
    return s;
}

// actual_M (kgraph.cpp:284-286) as stored in NeighborX::M (uint16_t).
__device__ __forceinline__ uint32_t actual_M(const SearchArgs &a, uint32_t pM, uint32_t id) {
    uint32_t deg, M;
    if (a.meta) {
        uint2 md = a.meta[id];
        M = md.x;
        deg = md.y;
    } else {
        deg = (uint32_t)(a.offsets[id + 1] - a.offsets[id]);
        M = a.Mnode[id];
    }
    return min(max(M, pM), deg) & 0xFFFFu;
}

// Neighbour p of node: the ELL copy for p < ell_w, else the CSR.
__device__ __forceinline__ uint32_t neighbour(const SearchArgs &a, uint32_t node, uint32_t p) {
    if (a.ell && p < a.ell_w) return a.ell[(size_t)node * a.ell_w + p];
    return a.nbr[a.offsets[node] + p];
}

// Distances for cnt candidates cid[0..cnt) -> cd[], 32/G per pass (G-lane groups).
template <int G>
__device__ __forceinline__ void batch_dist(const SearchArgs &a, const WarpSmem &s, float qn, uint32_t cnt,
                                           int lane) {
    constexpr uint32_t PER = 32 / G;
    const int g = lane / G, t = lane % G;
    for (uint32_t base = 0; base < cnt; base += PER) {
        uint32_t c = base + g;
        uint32_t id = c < cnt ? s.cid[c] : 0u;
        float dd = query_dist_g<G>(a.D, s.q, qn, id, t, FULL);
        if (c < cnt && t == 0) s.cd[c] = dd;
    }
    __syncwarp();
}

// SearchOracle::search (kgraph.cpp:231-252) by one warp: every row in id
// order, epsilon filter, sorted insert into K slots (+1 overflow).
template <int G>
__device__ uint32_t warp_bruteforce(const SearchArgs &a, const WarpSmem &s, float qn, uint32_t K, int lane) {
    const uint32_t N = a.D.n;
    uint32_t L = 0;
    for (uint32_t base = 0; base < N; base += 32) {
        uint32_t cnt = min(32u, N - base);
        if (lane < (int)cnt) s.cid[lane] = base + lane;
        __syncwarp();
        batch_dist<G>(a, s, qn, cnt, lane);
        for (uint32_t c = 0; c < cnt; ++c) {
            float dd = s.cd[c];
            if (dd > a.epsilon) continue;
            if (L == K && (K == 0 || dd >= s.pd[K - 1])) continue;   // would land at slot K
            warp_update_knn(s.pd, s.pid, (uint32_t *)nullptr, L, dd, base + c, 0u, lane);
            if (L < K) ++L;
        }
        __syncwarp();
    }
    return L;
}

// Distances of the n <= 32 candidates list[0 .. n), computed 32/G at a time by
// the G-lane groups; lane i < n returns candidate i's.  With `sel`, candidate i
// is list[sel[i]].
template <int G>
__device__ __forceinline__ float warp_list_dist(const SearchArgs &a, const float *q, float qn, const uint32_t *list,
                                               const uint8_t *sel, uint32_t n, int lane) {
    constexpr uint32_t PER = 32 / G;
    const int g = lane / G, t = lane % G;
    float mine = 0.f;
    for (uint32_t base = 0; base < n; base += PER) {
        const uint32_t i = base + g;
        const float dd = query_dist_g<G>(a.D, q, qn, i < n ? list[sel ? sel[i] : i] : 0u, t, FULL);
        const float got = __shfl_sync(FULL, dd, (int)(G * (lane % PER)));
        if ((uint32_t)lane / PER == base / PER) mine = got;
    }
    return mine;
}

// Hint: bring dataset row `id` into L2 (four 128-byte lines for D = 128).
__device__ __forceinline__ void prefetch_row(const DataView &D, uint32_t id) {
    const char *p = reinterpret_cast<const char *>(D.X + (size_t)id * D.ld);
    const uint32_t bytes = D.ld * 4;
    for (uint32_t o = 0; o < bytes; o += 128) asm volatile("prefetch.global.L2 [%0];" ::"l"(p + o));
}

__device__ __forceinline__ bool visited_test_set(uint32_t *vis, uint32_t id) {
    uint32_t bit = 1u << (id & 31);
    uint32_t old = atomicOr(vis + (id >> 5), bit);
    return (old & bit) != 0;
}

// ---- the distance filter on compressed rows (kg_precision.cu) ----
constexpr float U32 = 5.9604645e-8f;   // unit roundoff of FP32, 2^-24

// The W reconstructed values of `row` at elements [off, off + W): BF16 values,
// or FP8 E4M3 values times the row's scale (rounded to FP32, as the error
// bound of the compressed row assumes).
template <int PREC, int W>
__device__ __forceinline__ void load_y(const void *Xc, uint32_t ld, uint32_t row, uint32_t off, float scale,
                                       float *y) {
    if constexpr (PREC == 1) {
        const uint16_t *p = reinterpret_cast<const uint16_t *>(Xc) + (size_t)row * ld + off;
        uint32_t w[W / 2];
        if constexpr (W == 8) { const uint4 v = *reinterpret_cast<const uint4 *>(p); w[0] = v.x; w[1] = v.y; w[2] = v.z; w[3] = v.w; }
        else if constexpr (W == 4) { const uint2 v = *reinterpret_cast<const uint2 *>(p); w[0] = v.x; w[1] = v.y; }
        else { w[0] = *reinterpret_cast<const uint32_t *>(p); }
#pragma unroll
        for (int j = 0; j < W / 2; ++j) {
            y[2 * j] = __uint_as_float(w[j] << 16);
            y[2 * j + 1] = __uint_as_float(w[j] & 0xFFFF0000u);
        }
    } else {
        const uint8_t *p = reinterpret_cast<const uint8_t *>(Xc) + (size_t)row * ld + off;
        uint16_t h[W / 2];
        if constexpr (W == 8) {
            const uint2 v = *reinterpret_cast<const uint2 *>(p);
            h[0] = (uint16_t)v.x; h[1] = (uint16_t)(v.x >> 16); h[2] = (uint16_t)v.y; h[3] = (uint16_t)(v.y >> 16);
        } else if constexpr (W == 4) {
            const uint32_t v = *reinterpret_cast<const uint32_t *>(p);
            h[0] = (uint16_t)v; h[1] = (uint16_t)(v >> 16);
        } else {
            h[0] = *reinterpret_cast<const uint16_t *>(p);
        }
#pragma unroll
        for (int j = 0; j < W / 2; ++j) {
            const __half2_raw r = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)h[j], __NV_E4M3);
            const float2 f = __half22float2(__half2(r));
            y[2 * j] = __fmul_rn(f.x, scale);
            y[2 * j + 1] = __fmul_rn(f.y, scale);
        }
    }
}

// Sum over the row of (q - y)^2 (dot q.y for angular) with FP32 accumulation,
// by the G-lane group of this lane; every lane of the group gets the sum.
template <int PREC, int G>
__device__ __forceinline__ float approx_raw(const SearchArgs &a, const float *q, uint32_t row, int t, float scale) {
    constexpr int W = 16 / G;
    const bool dot = a.D.metric == METRIC_ANGULAR;
    float acc = 0.f;
    const uint32_t chunks = a.D.ld >> 4;
    for (uint32_t c = 0; c < chunks; ++c) {
        const uint32_t off = 16 * c + W * t;
        float y[W];
        load_y<PREC, W>(a.Xc, a.D.ld, row, off, scale, y);
#pragma unroll
        for (int j = 0; j < W; ++j) {
            const float qj = q[off + j];
            if (dot) acc = __fmaf_rn(qj, y[j], acc);
            else { const float df = __fsub_rn(qj, y[j]); acc = __fmaf_rn(df, df, acc); }
        }
    }
#pragma unroll
    for (int o = G / 2; o; o >>= 1) acc = __fadd_rn(acc, __shfl_xor_sync(FULL, acc, o));
    return acc;
}

// Rigorous lower bound of the canonical FP32 distance (kg_common.cuh) of a row
// x from `raw` (approx_raw over its reconstruction y, ||x - y|| <= e), the
// query's and the row's norm terms nq, nx.  gamma_k = k u bounds the relative
// error of a k-deep FP32 sum: ld + 8 deep for approx_raw, d/16 + 24 for the
// canonical distance (16 lanes, a 4-level tree, up to 15 tail terms).  Every
// step rounds towards the bound.
__device__ __forceinline__ float filter_lb(int metric, float raw, float e, float nq, float nx, uint32_t d,
                                           uint32_t ld) {
    const float ga = (float)(ld + 8) * U32 * 1.01f;
    const float gc = (float)(d / 16 + 24) * U32 * 1.01f;
    if (metric == METRIC_ANGULAR) {
        // -dot_c >= -dot' - ||q|| (e + ga ||y|| + gc ||x||);  ||q|| <= nq (1 + 2 gc), ||x|| <= nx (1 + 2 gc),
        // ||y|| <= ||x|| + e; the canonical denominator is recomputed bit for bit, and rounding is monotone
        const float qn = __fmul_ru(nq, 1.f + 2.f * gc);
        const float xn = __fmul_ru(nx, 1.f + 2.f * gc);
        const float yn = __fadd_ru(xn, e);
        const float B = __fmul_ru(qn, __fadd_ru(e, __fadd_ru(__fmul_ru(ga, yn), __fmul_ru(gc, xn))));
        const float num = __fsub_rd(-raw, B);
        return __fdiv_rd(num, __fmaf_rn(nx, nq, FLT_EPSILON));
    }
    // ||q - y||^2 >= raw (1 - ga) and ||q - x|| >= ||q - y|| - e
    const float r = __fsqrt_rd(fmaxf(__fmul_rd(raw, 1.f - ga), 0.f));
    const float b = fmaxf(__fsub_rd(r, e), 0.f);
    const float t2 = __fmul_rd(b, b);   // <= ||q - x||^2
    if (metric == METRIC_L2SQR) return __fmul_rd(t2, 1.f - 2.f * gc);   // canonical >= ||q-x||^2 (1 - gamma)
    // euclidean: canonical (n_q + n_x) - dot >= ||q - x||^2 / 2 - 2.2 gc (n_q + n_x)
    return __fsub_rd(__fmul_rd(t2, 0.5f), __fmul_ru(2.2f * gc, __fadd_ru(nq, nx)));
}

// Lower bounds of the n <= 32 candidates list[0 .. n) from their compressed
// rows, 32/G per pass; lane i < n returns candidate i's.
template <int PREC, int G>
__device__ __forceinline__ float warp_list_lb(const SearchArgs &a, const float *q, float qn, const uint32_t *list,
                                              uint32_t n, int lane) {
    constexpr uint32_t PER = 32 / G;
    const int g = lane / G, t = lane % G;
    float mine = 0.f;
    for (uint32_t base = 0; base < n; base += PER) {
        const uint32_t i = base + g;
        const uint32_t row = i < n ? list[i] : 0u;
        const float4 md = a.cmeta[row];   // {error bound, scale, norm term, 0}
        const float raw = approx_raw<PREC, G>(a, q, row, t, md.y);
        const float lb = filter_lb(a.D.metric, raw, md.x, qn, md.z, a.D.d, a.D.ld);
        const float got = __shfl_sync(FULL, lb, (int)(G * (lane % PER)));
        if ((uint32_t)lane / PER == base / PER) mine = got;
    }
    return mine;
}

// L2 prefetch of a compressed row.
template <int PREC>
__device__ __forceinline__ void prefetch_crow(const SearchArgs &a, uint32_t id) {
    const uint32_t bytes = a.D.ld * (PREC == 1 ? 2u : 1u);
    const char *p = reinterpret_cast<const char *>(a.Xc) + (size_t)id * bytes;
    for (uint32_t o = 0; o < bytes; o += 128) asm volatile("prefetch.global.L2 [%0];" ::"l"(p + o));
}

}  // namespace

// G: lanes per distance (the D-split, 32/G candidates per pass); PF: neighbour
// batches whose rows are prefetched into L2 ahead of the walk; PREC: 0, or the
// compressed rows (1 BF16, 2 FP8) that filter candidates once the pool is full.
// MB: resident blocks of 256 threads per SM the register allocation is sized
// for (4: 64 registers per thread; 3: 80, fewer spills for large pools, whose
// shared memory limits residency anyway), or 9: blocks of at most 128
// threads at 56 registers (36 warps per SM instead of 32).  CP: the compact 8-byte pool entry
// (the host selects it only when every node's expansion fits the progress
// field: a.cp_idbits id bits, 31 - a.cp_idbits progress bits).
template <int G, int PF, int PREC, int MB, int CP>
__global__ void __launch_bounds__(MB == 9 ? 128 : 256, MB) search_kernel(SearchArgs a) {
    extern __shared__ __align__(16) char smem[];
    const uint32_t IDM = CP ? (1u << a.cp_idbits) - 1u : ID_MASK;   // the id bits of a pool word
    const uint32_t PMASK = CP ? ID_MASK >> a.cp_idbits : 0u;        // the progress bits, shifted down
    const int lane = threadIdx.x & 31;
    const int wib = threadIdx.x >> 5;
    const uint32_t slot = blockIdx.x * a.warps_per_block + wib;
    WarpSmem s = carve<CP>(smem + (size_t)wib * a.warp_smem_bytes, a);
    uint32_t *vis = a.visited + (size_t)slot * a.vwords;
    const uint32_t N = a.D.n;

    for (;;) {
        uint32_t qi = 0;
        if (lane == 0) qi = atomicAdd(a.qcounter, 1u);
        qi = __shfl_sync(FULL, qi, 0);
        if (qi >= a.nq) break;
        const uint32_t K = a.Kq ? a.Kq[qi] : a.K;
        const uint32_t P = a.Pq ? a.Pq[qi] : a.P;
        const uint32_t T = a.T;
        const uint32_t S = min(a.S, 0x10000u);   // an expansion has at most 65535 neighbours (NeighborX::M)
        // x / S by multiplication, exact for x < 2^16 and 2 <= S <= 2^16
        const uint32_t inv_S = S > 1 ? 0xFFFFFFFFu / S + 1 : 0u;
        const uint32_t cap = K + P + 1;   // knn.size(), kgraph.cpp:434

        // query -> smem, and its norm term (SearchOracle ctor, python-api.cpp:98-101).  The padding
        // columns [d, ld) of a caller's row may hold anything; the smem copy holds zeros there, so the
        // compressed-row filter, which sums over whole 16-column chunks, sees (0 - 0)^2 terms.
        const float *qg = a.Q + (size_t)qi * a.q_ld;
        for (uint32_t x = lane * 4; x < a.D.ld; x += 128) {
            float4 v = ld4(qg + x);
            if (x + 4 > a.D.d) {
                if (x + 0 >= a.D.d) v.x = 0.f;
                if (x + 1 >= a.D.d) v.y = 0.f;
                if (x + 2 >= a.D.d) v.z = 0.f;
                if (x + 3 >= a.D.d) v.w = 0.f;
            }
            *reinterpret_cast<float4 *>(s.q + x) = v;
        }
        __syncwarp();
        float qn = 0.f;
        if (a.D.metric != METRIC_L2SQR) {
            float n2 = group4_raw(s.q, s.q, a.D.d, METRIC_EUCLIDEAN, lane & 3, FULL);
            qn = norm_term(n2, a.D.metric);
        }

        uint32_t count = 0;
        float cost = 0.f;
        uint32_t *out_i = a.out_ids + (size_t)qi * a.out_ld;
        float *out_d = a.out_dists ? a.out_dists + (size_t)qi * a.out_ld : nullptr;

        if (P >= N) {   // kgraph.cpp:427-433: brute force, cost 1
            count = warp_bruteforce<G>(a, s, qn, K, lane);
            for (uint32_t k = lane; k < count; k += 32) {
                out_i[k] = s.pid[k] & ID_MASK;
                if (out_d) out_d[k] = s.pd[k];
            }
            if (lane == 0) { a.out_count[qi] = count; if (a.out_cost) a.out_cost[qi] = 1.0f; }
            __syncwarp();
            continue;
        }
        if (a.init && !(a.init < K)) {   // kgraph.cpp:463
            if (lane == 0) { raise_error(a.err, ERR_INIT_K); a.out_count[qi] = 0; }
            __syncwarp();
            continue;
        }

        for (uint32_t w = lane * 4; w < a.vwords; w += 128)
            *reinterpret_cast<uint4 *>(vis + w) = make_uint4(0u, 0u, 0u, 0u);
        __syncwarp();

        uint32_t n_comps = 0, n_adj = 0, n_seed = 0, n_apx = 0, n_skip = 0;
        uint32_t rn = 0;          // results.size() - 1
        bool have_results = false;
        for (uint32_t trial = 0; trial < T; ++trial) {
            uint32_t L = 0;
            if (a.init == 0) {
                const uint32_t *seeds = a.seeds + a.seed_index[qi] + (size_t)trial * P;
                // kgraph.cpp:454-459: keep seeds not visited by an earlier trial
                for (uint32_t base = 0; base < P; base += 32) {
                    uint32_t j = base + lane;
                    uint32_t sid = j < P ? seeds[j] : 0u;
                    bool keep = j < P && !((__ldcg(vis + (sid >> 5)) >> (sid & 31)) & 1u);
                    unsigned m = __ballot_sync(FULL, keep);
                    if (keep) s.pid[L + __popc(m & ((1u << lane) - 1u))] = sid;
                    L += __popc(m);
                }
            } else {
                L = a.init;
                const uint32_t *init = a.init_ids + (size_t)qi * a.out_ld;
                for (uint32_t j = lane; j < L; j += 32) s.pid[j] = init[j];
            }
            __syncwarp();
            n_seed += L;
            bool nan = false;   // a distance this lane stored
            // kgraph.cpp:468-475: mark, flag, distance, m = 0, M = actual_M
            for (uint32_t base = 0; base < L; base += 32) {
                uint32_t j = base + lane;
                uint32_t id = j < L ? s.pid[j] : 0u;
                bool bad = j < L && id >= N;
                if (__any_sync(FULL, bad)) {
                    if (lane == 0) raise_error(a.err, ERR_BAD_ID);
                }
                if (j < L && !bad) {
                    atomicOr(vis + (id >> 5), 1u << (id & 31));
                    if constexpr (!CP) s.pm[j] = actual_M(a, a.Mp, id) << 16;
                }
                __syncwarp();
                uint32_t cnt = min(32u, L - base);
                if (j < L) s.cid[lane] = bad ? 0u : id;
                __syncwarp();
                batch_dist<G>(a, s, qn, cnt, lane);
                // an out-of-range starting point (the error is raised above) enters as id 0,
                // unflagged: it is never expanded, so no adjacency row is read for it
                if (j < L) {
                    const float dd = s.cd[lane];
                    nan |= dd != dd;
                    s.pd[j] = dd;
                    s.pid[j] = bad ? 0u : (id | FLAG_BIT);
                }
                __syncwarp();
            }
            // kgraph.cpp:476: std::sort by dist (GNU introsort order for ties)
            if (L <= (uint32_t)WARP_SORT_MAX) {
                warp_gnu_sort(s.pd, s.pid, s.pm, (int)L, s.lid, nan, lane);
            } else {
                if (lane == 0) {
                    WarpSortAcc acc{s.pd, s.pid, s.pm};
                    gnu_sort(acc, 0, (int)L);
                }
                __syncwarp();
            }

            uint32_t k = 0;
            // Each expansion advances m or clears a flag of an entry that was inserted
            // once, so the walk ends; the bound only turns a defect into an error.
            const uint64_t step_limit = 64ull * (N + cap) + 4096;
            uint64_t steps = 0;
            // The expansion loop of kgraph.cpp:478-514.  The reference expands the entry
            // at k batch after batch (S neighbours each) while no insert of a batch
            // lands at or before k, else it moves on to another entry after the batch.
            // Here an entry's adjacency comes in windows of up to 128 ids (four per
            // lane; one round trip for the ids, one for their visited bits -- this
            // warp's private set, so only this walk changes them), whose unvisited
            // neighbours form a list in order.  Batches without one change nothing but
            // the entry's progress and cost nothing.  The others are taken in groups of up
            // to 32 candidates, whatever batches they belong to: one round trip confirms
            // the group's candidates with an atomic test-and-set and brings their rows,
            // and their insertion positions show the first batch with an insert at or
            // before k.  The batches up to that one are merged into the pool in one
            // step; the candidates after it are put back to unvisited, as the reference
            // has not reached them (their rows were read for nothing).
            // What bounds it: a chain of dependent round trips per entry (ids, bits,
            // rows), so trips are what counts, not the rows' bytes.  Against one trip per
            // batch of S (1M x 128 mixture, 10k queries, K=10): P=1000 78.2 -> 45.7 ms,
            // 3 good starting points and P=5 5.62 -> 4.43 ms; one query on 100k x 16
            // 1.33 -> 0.79 ms.  Groups bounded to 8 or 16 candidates were slower
            // everywhere (49.2 / 47.1 ms, 4.98 / 4.77 ms, 1.03 / 0.88 ms).
            if (S == 0 && L > 0 && warp_next_flagged(s.pid, 0, L, lane) < L) {   // the reference would not end
                if (lane == 0) raise_error(a.err, ERR_STEP_LIMIT);
                L = 0;
            }
            while (true) {
                k = warp_next_flagged(s.pid, k, L, lane);
                if (k >= L) break;
                const uint32_t pk = s.pid[k];
                const uint32_t node = pk & IDM;
                uint32_t eM, m, bq = 0;
                uint32_t wid[4];
                bool pre = false;   // CP: wid holds the ELL ids of the window at m
                if constexpr (CP) {
                    // the node's {M, degree} and its first window's ELL ids in flight together
                    bq = (pk >> a.cp_idbits) & PMASK;
                    m = bq * S;
                    if (a.ell) {
#pragma unroll
                        for (int c = 0; c < 4; ++c) {
                            const uint32_t p = m + 32 * c + lane;
                            wid[c] = p < a.ell_w ? a.ell[(size_t)node * a.ell_w + p] : 0xFFFFFFFFu;
                        }
                        pre = true;
                    }
                    eM = actual_M(a, a.Mp, node);
                } else {
                    const uint32_t mM0 = s.pm[k];
                    eM = mM0 >> 16;
                    m = mM0 & 0xFFFFu;
                }
                uint32_t wlo = m, whi = m;     // loaded window [wlo, whi)
                uint32_t lb = 0, nl = 0;       // its unvisited neighbours not yet taken: list entries [lb, nl)
                uint32_t lim = eM;             // end of the positions to read: after an insert at or before k,
                bool moved = false;            //  the end of its batch
                uint32_t endM = eM;            // the entry's progress when the walk leaves it
                bool done = true;              // every neighbour read
                while (true) {
                    if (lb >= nl) {   // the next window
                        if (whi >= lim) break;
                        if (++steps > step_limit) {
                            if (lane == 0) raise_error(a.err, ERR_STEP_LIMIT);
                            k = L;
                            break;
                        }
                        wlo = whi;
                        whi = min(wlo + 128u, lim);
                        bool wuv[4];
#pragma unroll
                        for (int c = 0; c < 4; ++c) {
                            const uint32_t p = wlo + 32 * c + lane;
                            const bool act = p < whi;
                            if (!act) wid[c] = 0xFFFFFFFFu;
                            else if (!(CP && pre && p < a.ell_w)) wid[c] = neighbour(a, node, p);
                            const bool bad = act && wid[c] >= N;
                            if (__any_sync(FULL, bad)) { if (lane == 0) raise_error(a.err, ERR_BAD_ID); }
                            wuv[c] = act && !bad;
                        }
#pragma unroll
                        for (int c = 0; c < 4; ++c)
                            if (wuv[c]) wuv[c] = !((__ldcg(vis + (wid[c] >> 5)) >> (wid[c] & 31)) & 1u);
                        pre = false;
                        uint32_t tot = 0;
                        uint32_t cut = 0xFFFFFFFFu;
#pragma unroll
                        for (int c = 0; c < 4; ++c) {
                            const unsigned um = __ballot_sync(FULL, wuv[c]);
                            const uint32_t at = tot + __popc(um & ((1u << lane) - 1u));
                            if (wuv[c]) {
                                if (at < LIST) { s.lid[at] = wid[c]; s.lpos[at] = (uint8_t)(32 * c + lane); }
                                else if (at == LIST) cut = wlo + 32 * c + lane;
                            }
                            tot += __popc(um);
                        }
                        if (tot > LIST) whi = __reduce_min_sync(FULL, cut);   // the rest comes with the next window
                        lb = 0;
                        nl = min(tot, LIST);
                        __syncwarp();
                        continue;
                    }
                    // the group: lane j holds list entry lb + j, in its batch b
                    const uint32_t c = min(nl - lb, 32u);
                    const uint32_t at = lb + min((uint32_t)lane, c - 1);
                    const uint32_t id = s.lid[at];
                    const uint32_t x = wlo + s.lpos[at] - m;
                    const uint32_t b = S == 1 ? x : __umulhi(x, inv_S);
                    const bool act = (uint32_t)lane < c && x < lim - m;
                    const uint32_t n = __popc(__ballot_sync(FULL, act));   // act is a prefix of the lanes
                    if (n == 0) break;   // moved, and the rest lies behind the batch
                    const uint32_t *list = s.lid + lb;
                    const bool again = lb > 0;   // the window's second group or later
                    lb += n;
                    // an id that recurs in the group: its first position only, as the reference's
                    // in-order loop marks it visited there (kgraph.cpp:497-498)
                    const unsigned same = __match_any_sync(FULL, act ? id : 0xFFFFFFFFu);
                    const bool cand = act && (__ffs(same) - 1) == lane;
                    // L2 prefetch of the rows the next groups of this window will read, behind this
                    // group's loads
                    if constexpr (PF > 0) {
                        if (lane < PF * 8 && lb + lane < nl) {
                            const uint32_t pid2 = s.lid[lb + lane];
                            if (PREC && L == cap - 1) prefetch_crow<PREC>(a, pid2);
                            else prefetch_row(a.D, pid2);
                        }
                    }
                    // FP32 walk: the exact test-and-set of the visited bits in flight with the
                    // candidates' {M, degree} and rows.  Filtered walk: most candidates end with
                    // their compressed rows, which are there before a test-and-set would be; a
                    // candidate is new unless its id came up in an earlier group of the window,
                    // and is marked once the batches that are taken are known (10k queries on
                    // 200k x 100, angular, P=700: 82 -> 65 ms).
                    constexpr bool EARLY = PREC == 0;
                    bool isnew = cand;
                    uint32_t aM = 0;
                    if (cand) {
                        const uint32_t bit = 1u << (id & 31);
                        if (EARLY) isnew = !(atomicOr(vis + (id >> 5), bit) & bit);
                        else if (again) isnew = !(__ldcg(vis + (id >> 5)) & bit);
                    }
                    float dd = 0.f;
                    unsigned nm, im, sm = 0;   // new candidates; those that may enter the pool; those skipped
                    const bool full = L == cap - 1;
                    if (PREC && full) {
                        // Full pool: the lower bound from the compressed rows drops candidates that would
                        // land in the spare slot; the others take the FP32 distance.
                        const float lbd = warp_list_lb<PREC, G>(a, s.q, qn, list, n, lane);
                        const float worst = s.pd[L - 1];
                        const bool keep = isnew && !(lbd >= worst);
                        nm = __ballot_sync(FULL, isnew);
                        const unsigned km = __ballot_sync(FULL, keep);
                        sm = nm & ~km;
                        im = 0;
                        if (km) {
                            if (!CP && keep) aM = actual_M(a, a.Mp, id);
                            const uint32_t my = __popc(km & ((1u << lane) - 1u));
                            if (keep) s.lsel[my] = (uint8_t)lane;
                            __syncwarp();
                            const float got = warp_list_dist<G>(a, s.q, qn, list, s.lsel, __popc(km), lane);
                            dd = __shfl_sync(FULL, got, (int)my);
                            im = __ballot_sync(FULL, keep && dd < worst);
                            __syncwarp();
                        }
                    } else {
                        if (!CP && cand) aM = actual_M(a, a.Mp, id);
                        dd = warp_list_dist<G>(a, s.q, qn, list, nullptr, n, lane);
                        nm = __ballot_sync(FULL, isnew);
                        // A full pool takes a candidate only below its last entry: one at or
                        // above it lands in the spare slot (kgraph.cpp:503-506), and so does
                        // every later candidate that is not closer than it, so leaving those
                        // out of the merge changes no position.
                        im = full ? __ballot_sync(FULL, isnew && dd < s.pd[L - 1]) : nm;
                    }
                    unsigned taken = FULL;   // the lanes of the batches the reference reads
                    if (im) {
                        uint32_t ai, f;
                        const uint32_t r = warp_rank_batch(s.pd, L, cap, im, dd, ai, f, lane);
                        const unsigned hm = __ballot_sync(FULL, r <= k);
                        if (hm && !moved) {
                            // the expanded entry is no longer at k after this batch: its progress
                            // is written where it still stands
                            const uint32_t bs = __shfl_sync(FULL, b, __ffs(hm) - 1);
                            const uint32_t end = m + (bs + 1) * S;
                            moved = true;
                            done = end > eM;
                            endM = min(end, eM);
                            lim = endM;
                            if (lane == 0) {
                                if constexpr (CP) {   // progress in batches of S
                                    s.pid[k] = done ? node : (node | FLAG_BIT | ((bq + bs + 1) << a.cp_idbits));
                                } else {
                                    if (done) s.pid[k] = s.pid[k] & ID_MASK;
                                    s.pm[k] = (endM & 0xFFFFu) | (eM << 16);
                                }
                            }
                            taken = __ballot_sync(FULL, b <= bs);
                            if (EARLY && isnew && b > bs) atomicAnd(vis + (id >> 5), ~(1u << (id & 31)));
                            if (im & ~taken) {
                                im &= taken;
                                f = warp_rank_again(im, dd, lane);
                            }
                            __syncwarp();
                        }
                        const uint32_t mr = __reduce_min_sync(FULL, ((im >> lane) & 1u) ? r : 0xFFFFFFFFu);
                        L = warp_apply_batch(s.pd, s.pid, CP ? nullptr : s.pm, L, cap, im, ai, f, dd, id | FLAG_BIT,
                                             aM << 16, lane);   // new entries: flag set, m = 0, M = actual_M
                        if (mr < k) k = mr;
                    }
                    if (!EARLY) {
                        if (((nm & taken) >> lane) & 1u) atomicOr(vis + (id >> 5), 1u << (id & 31));
                        __syncwarp();   // the bits before the next look at them
                    }
                    n_comps += __popc(nm & taken);
                    if (PREC && full) {
                        n_apx += __popc(nm & taken);
                        n_skip += __popc(sm & taken);
                    }
                }
                if (k >= L) break;
                n_adj += endM - m;
                if (!moved) {   // every neighbour read, and the entry still at k
                    if (lane == 0) {
                        if constexpr (CP) {
                            s.pid[k] = node;
                        } else {
                            s.pid[k] = s.pid[k] & ID_MASK;
                            s.pm[k] = (eM & 0xFFFFu) | (eM << 16);
                        }
                    }
                    __syncwarp();
                }
            }
            if (L > K) L = K;   // kgraph.cpp:515
            if (!have_results) {
                for (uint32_t j = lane; j < L; j += 32) { s.rd[j] = s.pd[j]; s.rid[j] = s.pid[j] & (IDM | FLAG_BIT); }
                rn = L;
                have_results = true;
                __syncwarp();
            } else {   // kgraph.cpp:521-528
                for (uint32_t l = 0; l < L; ++l) {
                    uint32_t r = warp_update_knn(s.rd, s.rid, (uint32_t *)nullptr, rn, s.pd[l], s.pid[l] & (IDM | FLAG_BIT),
                                                 0u, lane);
                    if (r < rn + 1 && rn + 1 < K + 1) ++rn;
                }
            }
        }
        // kgraph.cpp:531-540: drop the spare slot, epsilon filter
        count = rn;
        for (uint32_t base = 0; base < count; base += 32) {
            uint32_t j = base + lane;
            unsigned m = __ballot_sync(FULL, j < count && s.rd[j] > a.epsilon);
            if (m) { count = base + __ffs(m) - 1; break; }
        }
        for (uint32_t k = lane; k < count; k += 32) {
            out_i[k] = s.rid[k] & ID_MASK;
            if (out_d) out_d[k] = s.rd[k];
        }
        cost = __fdiv_rn((float)n_comps, (float)N);   // kgraph.cpp:561
        if (lane == 0) {
            a.out_count[qi] = count;
            if (a.out_cost) a.out_cost[qi] = cost;
            if (a.work) {
                atomicAdd(a.work, (unsigned long long)(n_comps + n_seed));
                atomicAdd(a.work + 1, (unsigned long long)n_adj);
                if (PREC && n_apx) {
                    atomicAdd(a.work + 2, (unsigned long long)n_apx);
                    atomicAdd(a.work + 3, (unsigned long long)n_skip);
                }
            }
        }
        __syncwarp();
    }
}

// The filter's lower bound and the canonical distance for `per` dataset rows
// per query (one warp per query, one 4-lane group per row): the check of the
// bound's arithmetic, lb <= dist for every pair.
template <int PREC>
__global__ void __launch_bounds__(256) filter_bounds_kernel(SearchArgs a, const uint32_t *ids, uint32_t per, float *lb,
                                                            float *dist) {
    __shared__ __align__(16) float qs[8][256];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t qi = blockIdx.x * 8 + w;
    if (qi >= a.nq) return;   // whole warps
    float *q = qs[w];
    for (uint32_t x = lane; x < a.D.ld; x += 32) q[x] = x < a.D.d ? a.Q[(size_t)qi * a.q_ld + x] : 0.f;
    __syncwarp();
    float qn = 0.f;
    if (a.D.metric != METRIC_L2SQR) qn = norm_term(group4_raw(q, q, a.D.d, METRIC_EUCLIDEAN, lane & 3, FULL), a.D.metric);
    const int g = lane >> 2, t = lane & 3;
    for (uint32_t base = 0; base < per; base += 8) {
        const uint32_t j = base + g;
        const uint32_t row = j < per ? ids[(size_t)qi * per + j] : 0u;
        const float4 md = a.cmeta[row];
        const float raw = approx_raw<PREC, 4>(a, q, row, t, md.y);
        const float b = filter_lb(a.D.metric, raw, md.x, qn, md.z, a.D.d, a.D.ld);
        const float dd = query_dist(a.D, q, qn, row, t, FULL);
        if (j < per && t == 0) {
            lb[(size_t)qi * per + j] = b;
            dist[(size_t)qi * per + j] = dd;
        }
    }
}

cudaError_t launch_filter_bounds(const SearchArgs &a, const uint32_t *ids, uint32_t per, float *lb, float *dist,
                                 cudaStream_t st) {
    if (a.D.ld > 256) return cudaErrorInvalidValue;
    const uint32_t grid = (a.nq + 7) / 8;
    if (a.prec == 1) filter_bounds_kernel<1><<<grid, 256, 0, st>>>(a, ids, per, lb, dist);
    else if (a.prec == 2) filter_bounds_kernel<2><<<grid, 256, 0, st>>>(a, ids, per, lb, dist);
    else return cudaErrorInvalidValue;
    return cudaGetLastError();
}

// Two lanes per distance put 16 candidates in a pass instead of 8: half the
// passes, each a memory round trip, for twice the loads per lane.  That wins
// where a row is few chunks of 16 columns (or ends in a tail, which every lane of
// a group adds up by itself).  Measured on 60k uniform and 300k mixture rows, 2 /
// 1,000 / 30,000 queries, 4 lanes against 2: FP32 d = 12 to 60 1.00-1.36x, d = 64
// 0.94-1.07x, d = 96 0.90-1.05x; BF16 filter d = 12 to 96 0.99-1.29x; FP8 filter
// (whose row chunk is 4 bytes a lane) d <= 26 1.07-1.22x, above it 1.01-1.27x for
// up to 1,000 queries and 0.91-0.99x for 30,000.
uint32_t search_split(uint32_t d, uint32_t ld, uint32_t prec, size_t nq, int num_sms) {
    bool two;
    if (prec == 0) two = d < 64;
    else if (prec == 1) two = ld <= 96;
    else two = d < 32 || (ld <= 96 && nq <= (size_t)num_sms * 8);
    return two ? 2 : 4;
}

size_t search_warp_smem_bytes(uint32_t ld, uint32_t cap, uint32_t rcap, bool compact) {
    size_t b = sizeof(float) * ld + (compact ? 8ull : 12ull) * cap + 8ull * rcap + 12ull * 32;
    return (b + 15) & ~size_t(15);
}

namespace {

using SearchFn = void (*)(SearchArgs);
template <int PREC, int MB, int CP>
SearchFn search_fn_prec(uint32_t split, bool pf) {
    switch (split) {
        case 2: return pf ? search_kernel<2, 2, PREC, MB, CP> : search_kernel<2, 0, PREC, MB, CP>;
        case 8: return pf ? search_kernel<8, 2, PREC, MB, CP> : search_kernel<8, 0, PREC, MB, CP>;
        default: return pf ? search_kernel<4, 2, PREC, MB, CP> : search_kernel<4, 0, PREC, MB, CP>;
    }
}
// The compiled (D-split, prefetch, filter precision, register budget, pool
// entry) variants; the 80-register budget and the compact pool exist for the
// FP32 walk.
SearchFn search_fn(uint32_t split, uint32_t prefetch, uint32_t prec, uint32_t regs, bool compact) {
    const bool pf = prefetch > 0;
    if (prec == 1) return search_fn_prec<1, 4, 0>(split, pf);
    if (prec == 2) return search_fn_prec<2, 4, 0>(split, pf);
    if (compact) {
        if (regs == 56) return search_fn_prec<0, 9, 1>(split, pf);
        return regs == 80 ? search_fn_prec<0, 3, 1>(split, pf) : search_fn_prec<0, 4, 1>(split, pf);
    }
    return regs == 80 ? search_fn_prec<0, 3, 0>(split, pf) : search_fn_prec<0, 4, 0>(split, pf);
}
// The compact pool runs where the shape asks for it and the graph allows it.
bool use_compact(const SearchArgs &a, const SearchShape &sh) { return search_uses_compact(a, sh); }

// Warps per block: the requested query tile, or as many as fit 200 KB of
// shared memory (at most 8); halved until the block fits.
uint32_t pick_wpb(const SearchShape &sh, size_t warp_bytes) {
    const uint32_t most = sh.regs == 56 ? 4u : 8u;   // the 56-register variant takes blocks of at most 128 threads
    uint32_t wpb = sh.warps_per_block ? std::min<uint32_t>(sh.warps_per_block, most) : most;
    while (wpb > 1 && (size_t)wpb * warp_bytes > 200 * 1024) wpb >>= 1;
    return wpb;
}

}  // namespace

bool search_uses_compact(const SearchArgs &a, const SearchShape &sh) {
    return sh.compact && a.compact_ok && a.prec == 0;
}

bool search_shape_valid(const SearchShape &sh) {
    const bool split_ok = sh.split == 0 || sh.split == 2 || sh.split == 4 || sh.split == 8;
    const bool wpb_ok = sh.warps_per_block == 0 || sh.warps_per_block == 1 || sh.warps_per_block == 2 ||
                        sh.warps_per_block == 4 || sh.warps_per_block == 8;
    const bool pf_ok = sh.prefetch == 0 || sh.prefetch == 2;
    const bool regs_ok = sh.regs == 0 || sh.regs == 56 || sh.regs == 64 || sh.regs == 80;
    return split_ok && wpb_ok && pf_ok && regs_ok && sh.compact <= 1;
}

cudaError_t launch_search(SearchArgs &a, const SearchShape &sh, int num_sms, cudaStream_t st, uint32_t *grid_out) {
    const bool cp = use_compact(a, sh);
    a.warp_smem_bytes = (uint32_t)search_warp_smem_bytes(a.D.ld, a.cap, a.rcap, cp);
    const uint32_t wpb = pick_wpb(sh, a.warp_smem_bytes);
    if ((size_t)wpb * a.warp_smem_bytes > 227 * 1024) return cudaErrorInvalidValue;
    a.warps_per_block = wpb;
    size_t smem = (size_t)wpb * a.warp_smem_bytes;
    SearchFn fn = search_fn(sh.split, sh.prefetch, a.prec, sh.regs, cp);
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, wpb * 32, smem);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) per_sm = 1;
    uint32_t grid = (uint32_t)(num_sms * per_sm);
    uint32_t need = (a.nq + wpb - 1) / wpb;
    if (grid > need) grid = need;
    if (grid < 1) grid = 1;
    if (grid_out) *grid_out = grid;
    if (grid * wpb > a.visited_slots) return cudaErrorInvalidValue;
    fn<<<grid, wpb * 32, smem, st>>>(a);
    return cudaGetLastError();
}

uint32_t search_max_slots(const SearchArgs &a, const SearchShape &sh, int num_sms) {
    const bool cp = use_compact(a, sh);
    const size_t wb = search_warp_smem_bytes(a.D.ld, a.cap, a.rcap, cp);
    const uint32_t wpb = pick_wpb(sh, wb);
    const size_t smem = (size_t)wpb * wb;
    SearchFn fn = search_fn(sh.split, sh.prefetch, a.prec, sh.regs, cp);
    cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, wpb * 32, smem);
    if (per_sm < 1) per_sm = 1;
    return (uint32_t)(num_sms * per_sm) * wpb;
}

}  // namespace kgb
