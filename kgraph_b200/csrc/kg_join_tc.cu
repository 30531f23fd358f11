// Local join on the fifth-generation tensor cores (tcgen05), for D >= 64.
//
// KGraphConstructor::join + Nhood::join (kgraph.cpp:740-751, 797-815) visit,
// for every node n, the pairs new x new (i < j) and new x old of n's sample
// lists and try each pair's distance against both endpoints' pools.  Here one
// CTA takes one node at a time:
//
//   1. U = new ++ old (positions 0..a-1 are new).  U's rows are staged into
//      shared memory as BF16, CENTERED on x_n (row - x_n, in FP32, then
//      rounded): the distances are translation invariant, and centering makes
//      the BF16 error scale with |x_u - x_n| |x_j - x_n| -- neighbour
//      distances -- instead of the raw norms.  The same pass keeps, per row,
//      h = |x_u - x_n|^2 / 2 and c = (x_u - x_n) . x_n in FP32.
//   2. tcgen05.mma (kind::f16, BF16 x BF16 -> FP32 in TMEM) forms the Gram
//      block of 32 new rows (N) against themselves and 96 of the entries after
//      them (M = 128); the new rows are the tile's first 32, so B is read from
//      the same staged buffer.  A node has 10 to 30 new entries and 20 to 70 in
//      all: with 128 columns and a second 128-row buffer an SM held three CTAs
//      of eight warps, half of them without a row; four warps, 32 TMEM columns
//      and one buffer make that six nodes at a time, each with its next list in
//      flight.  200k x 96 (K=50 L=100 S=12) whole build 178 -> 153 ms, 100k x
//      128 97 -> 79, 60k x 64 36 -> 28; E4M3 tiles 200k x 96 331 -> 290.
//   3. Each epilogue thread owns one U row (one TMEM lane) and derives the
//      approximate distance of each of its pairs: euclidean h_u + h_j - g,
//      l2sqr twice that, angular -(g + c_u + c_j + |x_n|^2) / (n_u n_j + eps).
//      The test is arranged so that a pair costs a dozen multiply-adds
//      (filter_terms): with a square root and a division per pair this epilogue
//      was two thirds of the kernel (200k x 96 unit-norm mixture, K=50 L=100
//      S=12, whole build 386 -> 193 ms; E4M3 tiles 551 -> 345 ms).
//      A pair whose approximate distance minus a rigorous error margin E is
//      above BOTH endpoints' radius cannot pass the reference's unlocked
//      radius test (kgraph.cpp:725, radii only shrink during a join), so it is
//      skipped.  Every other pair is recomputed with the canonical FP32
//      distance and offered as the CUDA-core join offers its pairs (to the
//      record of deferred inserts, or inserted under the pools' locks): every
//      insert, ordering and stored distance is decided in FP32.
//
// The margin E bounds |approx - exact| + |canonical FP32 - exact| with a
// factor 2 of slack: BF16 rounding of both operands (2^-8 + 2^-17 relative to
// |x_u - x_n| |x_j - x_n|), FP32 accumulation of D products (up to 2^-23 each),
// the FP32 centering and norm sums, and the canonical distance's own error
// (D + 4 ulps of the uncentered norms).  On a sample of nodes (about 1 in 2048)
// every pair is also evaluated in FP64 and in canonical FP32: the tile error and
// its ratio to E are recorded (JoinTcStats), and a pair whose lower bound, as the
// test itself formed it, lies above its distance, or that was skipped although a
// pool would take it, is a violation.
//
// All waits are bounded: the MMA completion barrier gives up after ~1 s,
// raises ERR_TC_TIMEOUT and the CTA drains, frees its TMEM and returns.
#include <algorithm>
#include <cfloat>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>
#include "kg_build.h"
#include "kg_insert.cuh"
#include "kg_join_filter.h"
#include "kg_tc.cuh"

namespace kgb {
namespace {

constexpr int TC_THREADS = 128;          // warp w reads TMEM lanes 32 w .. 32 w + 31
constexpr uint32_t TC_M = 128;           // rows per tile = TMEM lanes
constexpr uint32_t TC_N = 32;            // new columns per tile = TMEM columns
constexpr uint32_t TC_REST = TC_M - TC_N;   // partners per tile besides the columns' own rows
constexpr uint32_t TC_TMEM_COLS = 32;
constexpr long long TC_WAIT_CYCLES = 2000000000ll;
constexpr uint32_t TC_CLAIM = 8;         // nodes claimed per CTA at a time

static_assert((int)FILTER_EUCLIDEAN == METRIC_EUCLIDEAN && (int)FILTER_ANGULAR == METRIC_ANGULAR &&
              (int)FILTER_L2SQR == METRIC_L2SQR, "FilterMetric");

__device__ __forceinline__ bool sampled_node(uint32_t n) { return ((n * 0x9E3779B1u) >> 21) == 0; }

// Approximate distance of a pair from its Gram entry g, and the margin E.
struct Approx { float d, e; };
__device__ __forceinline__ Approx approx_dist(int metric, float g, float hu, float hj, float cu, float cj, float nu,
                                              float nj, float qn, float et, float gam) {
    const float pt = 2.0f * sqrtf(hu * hj);   // |x_u - x_n| |x_j - x_n|
    Approx r;
    if (metric == METRIC_ANGULAR) {
        const float full = g + cu + cj + qn;
        const float den = nu * nj + FLT_EPSILON;
        r.d = -full / den;
        const float edot = et * pt + gam * (sqrtf(2.0f * hu) + sqrtf(2.0f * hj)) * sqrtf(qn) + gam * qn +
                           4.0f * 5.96e-8f * (fabsf(cu) + fabsf(cj) + qn + fabsf(g));
        r.e = 2.0f * (edot / den + gam * (nu * nj) / den + 2.0f * gam * fabsf(r.d)) + 1e-30f;
    } else if (metric == METRIC_L2SQR) {
        r.d = 2.0f * ((hu + hj) - g);
        r.e = 2.0f * (2.0f * et * pt + 6.0f * gam * (hu + hj)) + 1e-30f;
    } else {
        r.d = (hu + hj) - g;
        r.e = 2.0f * (et * pt + gam * (hu + hj) + 2.0f * gam * (nu + nj)) + 1e-30f;
    }
    return r;
}

// The pair's distance in FP64 from the FP32 rows, by one warp (every lane
// returns it).
__device__ double warp_dist64(const DataView &D, uint32_t i, uint32_t j, int lane) {
    const float *a = D.X + (size_t)i * D.ld, *b = D.X + (size_t)j * D.ld;
    double s = 0, na = 0, nb = 0;
    for (uint32_t k = lane; k < D.d; k += 32) {
        const double x = a[k], y = b[k];
        if (D.metric == METRIC_ANGULAR) { s += x * y; na += x * x; nb += y * y; }
        else s += (x - y) * (x - y);
    }
    for (int o = 16; o; o >>= 1) {
        s += __shfl_xor_sync(FULL, s, o);
        na += __shfl_xor_sync(FULL, na, o);
        nb += __shfl_xor_sync(FULL, nb, o);
    }
    if (D.metric == METRIC_ANGULAR) return -s / (sqrt(na) * sqrt(nb) + (double)FLT_EPSILON);
    return D.metric == METRIC_L2SQR ? s : 0.5 * s;
}

// What a warp's sampled pairs add to the join's statistics.
struct SampleTally {
    unsigned long long sampled, violations, rel_count;
    double sum_abs, sum_ratio, sum_rel;
    uint32_t max_abs, max_ratio, max_rel;   // bits of non-negative floats
    __device__ void add(JoinTcStats *t) const {
        atomicAdd(&t->sampled, sampled);
        atomicAdd(&t->sum_abs, sum_abs);
        atomicAdd(&t->sum_ratio, sum_ratio);
        atomicMax(&t->max_abs_bits, max_abs);
        atomicMax(&t->max_ratio_bits, max_ratio);
        if (rel_count) {
            atomicAdd(&t->rel_count, rel_count);
            atomicAdd(&t->sum_rel, sum_rel);
            atomicMax(&t->max_rel_bits, max_rel);
        }
        if (violations) atomicAdd(&t->violations, violations);
    }
};

// Whole warp: the error of the approximate distance of rows ia and ib of node
// n's lists (Gram entry g) against FP64, and the filter's own decision against
// the distances.  f: {product error, the filter's lower bound, the larger radius as
// it held it, 1 where it skipped the pair}.
__device__ __noinline__ void sample_pair(const BuildState &s, uint32_t n, uint32_t ia, uint32_t ib, float g, float4 f,
                                         int lane, SampleTally &t) {
    const float etp = f.x;
    const uint32_t Dp = s.D.ld;
    const float gam = (float)(s.D.d + 4) * 5.9605e-8f;
    const float *xn = s.D.X + (size_t)n * Dp;
    float qn = 0.f, hc[4] = {0.f, 0.f, 0.f, 0.f};   // |x_n|^2; h and c of both rows (filter_terms)
    for (uint32_t k = lane; k < Dp; k += 32) {
        const float x = xn[k], ea = s.D.X[(size_t)ia * Dp + k] - x, eb = s.D.X[(size_t)ib * Dp + k] - x;
        qn += x * x;
        hc[0] += ea * ea; hc[1] += eb * eb; hc[2] += ea * x; hc[3] += eb * x;
    }
    for (int o = 16; o; o >>= 1) {
        qn += __shfl_xor_sync(FULL, qn, o);
#pragma unroll
        for (int k = 0; k < 4; ++k) hc[k] += __shfl_xor_sync(FULL, hc[k], o);
    }
    const Approx ap = approx_dist(s.D.metric, g, 0.5f * hc[0], 0.5f * hc[1], hc[2], hc[3], s.D.norms[ia], s.D.norms[ib],
                                  qn, etp, gam);
    const float dc = pair_dist(s.D, ia, ib, lane & 3, FULL);
    const double d64 = warp_dist64(s.D, ia, ib, lane), err = fabs((double)ap.d - d64), ratio = err / (double)ap.e;
    ++t.sampled;
    t.sum_abs += err;
    t.sum_ratio += ratio;
    t.max_abs = max(t.max_abs, __float_as_uint((float)err));
    t.max_ratio = max(t.max_ratio, __float_as_uint((float)ratio));
    if (d64 != 0.0) {
        const double rel = err / fabs(d64);
        ++t.rel_count;
        t.sum_rel += rel;
        t.max_rel = max(t.max_rel, __float_as_uint((float)rel));
    }
    const bool wrong = filter_wrong((FilterMetric)s.D.metric, f.y, f.w != 0.f, f.z, s.D.norms ? s.D.norms[ia] : 0.f,
                                    s.D.norms ? s.D.norms[ib] : 0.f, d64, dc);
    if (err > (double)ap.e || wrong) ++t.violations;
}

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t *>(&v);
}

struct TcShared {
    uint8_t *buf;           // the 128-row tile (BF16 or E4M3), K-major core-matrix layout
    float *xn;              // x_n, FP32
    float4 *tA;             // per U row {A, s, radius, id (NO_ID for a bad id)} (filter_terms)
    float2 *tC;             // {C, canonical norm term}
    float2 *tF;             // E4M3 tiles: {scale, 1 + rel}, rel = ||v - scale q|| / ||v||
};
constexpr uint32_t TC_PAD = 16;   // the epilogue reads columns 16 at a time, past the last row

__device__ __forceinline__ void filter_terms(int metric, float h, float c, float nrm, float qn, float gam, float rad,
                                             uint32_t id, float4 &tA, float2 &tC) {
    const FilterRow r = filter_row((FilterMetric)metric, h, c, nrm, qn, gam, rad);
    tA = make_float4(r.A, r.s, r.rad, __uint_as_float(id));
    tC = make_float2(r.C, r.nrm);
}

// The tile's rows: entries [j0, j0 + nb) of U in rows 0 .. nb - 1, entries
// [us, us + nr) in rows 32 .. 32 + nr - 1.  Groups of 8 rows go to the warps in
// turn: lane l owns row (l & 7) of the group and 16-byte chunks (l >> 3) + 4i, so
// each quarter-warp store covers one contiguous 128-byte core matrix.
struct TileRows {
    uint32_t j0, nb, us, nr;
    __device__ __forceinline__ uint32_t groups() const { return (nb + 7) / 8 + (nr + 7) / 8; }
    // row r = 8 g + k of the staging order: its tile row and entry; false past the end
    __device__ __forceinline__ bool at(uint32_t g, uint32_t k, uint32_t &row, uint32_t &u) const {
        const uint32_t gb = (nb + 7) / 8;
        const bool first = g < gb;
        const uint32_t r = (first ? g : g - gb) * 8 + k;
        row = first ? r : TC_N + r;
        u = (first ? j0 : us) + r;
        return r < (first ? nb : nr);
    }
};
template <int PREC>
__device__ void stage_rows(const BuildState &s, const TcShared &sh, const TileRows &tr, float qn, float gam, int warp,
                           int lane);

// E4M3 rows with a per-row scale: v = x_u - x_n in FP32 (as the BF16 rows),
// scale = max|v| / 448, q = e4m3_satfinite(v / scale); per row the exact
// ||v - scale q|| (FP64, every term exact there) relative to ||v||, rounded up.
// Lane l owns row (l & 7) of a group of 8 and 16-byte chunks (16 elements)
// (l >> 3) + 4i; the row's maximum needs a first pass over its elements.
template <>
__device__ void stage_rows<1>(const BuildState &s, const TcShared &sh, const TileRows &tr, float qn, float gam,
                              int warp, int lane) {
    const uint32_t Dp = s.D.ld, nk16 = Dp >> 4;
    for (uint32_t g = warp; g < tr.groups(); g += TC_THREADS / 32) {
        uint32_t rl, u;
        const bool valid = tr.at(g, lane & 7, rl, u);
        const uint32_t id = valid ? __float_as_uint(sh.tA[u].w) : NO_ID;
        const bool ok = id != NO_ID;
        float nrm = 0.f, rd = -FLT_MAX;
        if (ok && lane < 8) {
            nrm = s.D.norms[id];
            rd = *reinterpret_cast<volatile const float *>(s.radius + id);
        }
        const float *row = s.D.X + (size_t)(ok ? id : 0u) * Dp;
        float hs = 0.f, cs = 0.f, mx = 0.f;
        for (uint32_t k16 = lane >> 3; k16 < nk16; k16 += 4) {
#pragma unroll
            for (int h = 0; h < 4; ++h) {
                const float4 n0 = *reinterpret_cast<const float4 *>(sh.xn + 16 * k16 + 4 * h);
                const float4 a0 = ok ? ld4(row + 16 * k16 + 4 * h) : n0;
                const float e0 = a0.x - n0.x, e1 = a0.y - n0.y, e2 = a0.z - n0.z, e3 = a0.w - n0.w;
                hs += e0 * e0 + e1 * e1 + e2 * e2 + e3 * e3;
                cs += e0 * n0.x + e1 * n0.y + e2 * n0.z + e3 * n0.w;
                mx = fmaxf(mx, fmaxf(fmaxf(fabsf(e0), fabsf(e1)), fmaxf(fabsf(e2), fabsf(e3))));
            }
        }
        hs += __shfl_xor_sync(FULL, hs, 8);
        hs += __shfl_xor_sync(FULL, hs, 16);
        cs += __shfl_xor_sync(FULL, cs, 8);
        cs += __shfl_xor_sync(FULL, cs, 16);
        mx = fmaxf(mx, __shfl_xor_sync(FULL, mx, 8));
        mx = fmaxf(mx, __shfl_xor_sync(FULL, mx, 16));
        const float scale = mx > 0.f ? mx / 448.f : 1.f;
        double err2 = 0.0;
        for (uint32_t k16 = lane >> 3; k16 < nk16; k16 += 4) {
            uint32_t wv[4];
#pragma unroll
            for (int h = 0; h < 4; ++h) {
                const float4 n0 = *reinterpret_cast<const float4 *>(sh.xn + 16 * k16 + 4 * h);
                const float4 a0 = ok ? ld4(row + 16 * k16 + 4 * h) : n0;
                const float e[4] = {a0.x - n0.x, a0.y - n0.y, a0.z - n0.z, a0.w - n0.w};
                uint32_t word = 0;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const __nv_fp8_storage_t qv = __nv_cvt_float_to_fp8(e[i] / scale, __NV_SATFINITE, __NV_E4M3);
                    const double y = (double)__half2float(__half(__nv_cvt_fp8_to_halfraw(qv, __NV_E4M3))) * (double)scale;
                    const double df = (double)e[i] - y;
                    err2 += df * df;
                    word |= (uint32_t)qv << (8 * i);
                }
                wv[h] = word;
            }
            *reinterpret_cast<uint4 *>(sh.buf + tc::kmajor_off8(rl, 16 * k16, Dp)) = make_uint4(wv[0], wv[1], wv[2], wv[3]);
        }
        err2 += __shfl_xor_sync(FULL, err2, 8);
        err2 += __shfl_xor_sync(FULL, err2, 16);
        if (lane < 8 && valid) {
            filter_terms(s.D.metric, 0.5f * hs, cs, nrm, qn, gam, rd, id, sh.tA[u], sh.tC[u]);
            // relative to ||v|| (hs carries an FP32 rounding: one more relative step of slack)
            const float rel = hs > 0.f ? __double2float_ru(sqrt(err2) / sqrt((double)hs) * (1.0 + 1e-5)) : 0.f;
            sh.tF[u] = make_float2(scale, 1.f + rel);
        }
    }
    tc::fence_async_shared();   // make the generic-proxy stores visible to the MMA
}

template <>
__device__ void stage_rows<0>(const BuildState &s, const TcShared &sh, const TileRows &tr, float qn, float gam,
                              int warp, int lane) {
    const uint32_t Dp = s.D.ld, nk8 = Dp >> 3;
    // Rows past nb and nr are left as they are: the MMA reads them, but their
    // products land only in masked rows / columns of the accumulator.
    for (uint32_t g = warp; g < tr.groups(); g += TC_THREADS / 32) {
        uint32_t rl, u;
        const bool valid = tr.at(g, lane & 7, rl, u);
        const uint32_t id = valid ? __float_as_uint(sh.tA[u].w) : NO_ID;
        const bool ok = id != NO_ID;
        float nrm = 0.f, rd = -FLT_MAX;
        if (ok && lane < 8) {   // issued ahead of the row loads
            nrm = s.D.norms[id];
            rd = *reinterpret_cast<volatile const float *>(s.radius + id);
        }
        const float *row = s.D.X + (size_t)(ok ? id : 0u) * Dp;
        float hs = 0.f, cs = 0.f;
#pragma unroll 4
        for (uint32_t k8 = lane >> 3; k8 < nk8; k8 += 4) {
            float e[8], xv[8];
            const float4 n0 = *reinterpret_cast<const float4 *>(sh.xn + 8 * k8);
            const float4 n1 = *reinterpret_cast<const float4 *>(sh.xn + 8 * k8 + 4);
            xv[0] = n0.x; xv[1] = n0.y; xv[2] = n0.z; xv[3] = n0.w;
            xv[4] = n1.x; xv[5] = n1.y; xv[6] = n1.z; xv[7] = n1.w;
            if (ok) {
                const float4 a0 = ld4(row + 8 * k8), a1 = ld4(row + 8 * k8 + 4);
                e[0] = a0.x - xv[0]; e[1] = a0.y - xv[1]; e[2] = a0.z - xv[2]; e[3] = a0.w - xv[3];
                e[4] = a1.x - xv[4]; e[5] = a1.y - xv[5]; e[6] = a1.z - xv[6]; e[7] = a1.w - xv[7];
            } else {
#pragma unroll
                for (int i = 0; i < 8; ++i) e[i] = 0.f;
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) { hs += e[i] * e[i]; cs += e[i] * xv[i]; }
            uint4 pk;
            pk.x = pack_bf16(e[0], e[1]); pk.y = pack_bf16(e[2], e[3]);
            pk.z = pack_bf16(e[4], e[5]); pk.w = pack_bf16(e[6], e[7]);
            *reinterpret_cast<uint4 *>(sh.buf + tc::kmajor_off(rl, 8 * k8, Dp)) = pk;
        }
        hs += __shfl_xor_sync(FULL, hs, 8);
        hs += __shfl_xor_sync(FULL, hs, 16);
        cs += __shfl_xor_sync(FULL, cs, 8);
        cs += __shfl_xor_sync(FULL, cs, 16);
        if (lane < 8 && valid) {
            filter_terms(s.D.metric, 0.5f * hs, cs, nrm, qn, gam, rd, id, sh.tA[u], sh.tC[u]);
        }
    }
    tc::fence_async_shared();   // make the generic-proxy stores visible to the MMA
}

template <int PREC>
__global__ void __launch_bounds__(TC_THREADS, JOIN_TC_MAX_CTAS_PER_SM)
    join_tc_kernel(const __grid_constant__ BuildState s, uint32_t Umax, JoinQueue jq, uint32_t round) {
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ __align__(8) uint64_t mbar;
    __shared__ uint32_t tmem_base, s_cnt;
    __shared__ uint32_t s_list[TC_CLAIM], s_la[TC_CLAIM], s_lb[TC_CLAIM];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t Dp = s.D.ld, N = s.D.n;
    const uint32_t n_begin = jq.bounds[round], n_end = jq.bounds[round + 1];
    const uint32_t tile_bytes = TC_M * Dp * (PREC ? 1 : 2);
    TcShared sh;
    sh.buf = smem;
    sh.xn = reinterpret_cast<float *>(smem + tile_bytes);
    sh.tA = reinterpret_cast<float4 *>(sh.xn + Dp);   // 16-byte aligned: Dp is a multiple of 16
    sh.tC = reinterpret_cast<float2 *>(sh.tA + Umax + TC_PAD);
    sh.tF = sh.tC + Umax + TC_PAD;

    if (warp == 0) tc::tmem_alloc(&tmem_base, TC_TMEM_COLS);
    if (tid == 0) tc::mbar_init(&mbar, 1);
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = tmem_base;
    const float et = 0.00390625f + 7.63e-6f + (float)(s.D.d + 4) * 1.1921e-7f;   // 2^-8 + 2^-17 + (D+4) 2^-23
    // E4M3 tiles: the products' FP32 accumulation, allowed 2^-20 per add, and the two scale multiplies
    const float g8 = (float)(s.D.d + 4) * 9.5367e-7f + 8.f * 5.9605e-8f;
    const float gam = (float)(s.D.d + 4) * 5.9605e-8f;                             // (D+4) 2^-24
    const int metric = s.D.metric;
    uint32_t phase = 0;
    bool aborted = false;
    unsigned long long comps = 0, passed = 0;

    uint32_t next = 0;
    if (tid == 0) next = n_begin + atomicAdd(jq.work, TC_CLAIM);
    for (;;) {
        // claim TC_CLAIM nodes of this round's range; keep those with new entries
        if (warp == 0) {
            const uint32_t base = __shfl_sync(FULL, next, 0), nn = base + lane;
            bool act = false;
            uint32_t ca = 0, cb = 0;
            if (lane < (int)TC_CLAIM && nn < n_end) {
                s.found[nn] = 0;   // set again by the insert phase (kgraph.cpp:808-810)
                ca = s.cnt_new[nn];
                cb = s.cnt_old[nn];
                act = ca > 0;
            }
            const unsigned am = __ballot_sync(FULL, act);
            if (act) {
                const int slot = __popc(am & ((1u << lane) - 1u));
                if (ca > s.NEWCAP || cb > s.OLDCAP) raise_error(s.err, ERR_CAPACITY);
                s_list[slot] = nn;
                s_la[slot] = min(ca, s.NEWCAP);
                s_lb[slot] = min(cb, s.OLDCAP);
            }
            if (lane == 0) {
                s_cnt = base < n_end ? __popc(am) : NO_ID;
                if (base < n_end) next = n_begin + atomicAdd(jq.work, TC_CLAIM);   // needed when this run is done
            }
        }
        __syncthreads();
        const uint32_t cnt = s_cnt;
        if (cnt == NO_ID) break;
        // a node's list and row are read one node ahead: the first two entries a
        // thread takes of it, and this thread's column of x_n
        uint32_t pid[2] = {0u, 0u};
        float px = 0.f;
        auto entry = [&](uint32_t n, uint32_t a, uint32_t u) {
            return u < a ? s.nn_new[(size_t)n * s.NEWCAP + u] : s.nn_old[(size_t)n * s.OLDCAP + u - a];
        };
        auto fetch = [&](uint32_t li) {
            if (li >= cnt) return;
            const uint32_t n = s_list[li], a = s_la[li], U = a + s_lb[li];
#pragma unroll
            for (uint32_t k = 0; k < 2; ++k)
                if (tid + k * TC_THREADS < U) pid[k] = entry(n, a, tid + k * TC_THREADS);
            if (tid < Dp) px = s.D.X[(size_t)n * Dp + tid];
        };
        fetch(0);
        for (uint32_t li = 0; li < cnt && !aborted; ++li) {
        const uint32_t n = s_list[li], a = s_la[li], b = s_lb[li];
        const uint32_t U = a + b;
        auto put = [&](uint32_t u, uint32_t id) {
            if (id >= N) { raise_error(s.err, ERR_BAD_ID); id = NO_ID; }
            sh.tA[u].w = __uint_as_float(id);
        };
#pragma unroll
        for (uint32_t k = 0; k < 2; ++k)
            if (tid + k * TC_THREADS < U) put(tid + k * TC_THREADS, pid[k]);
        for (uint32_t u = tid + 2 * TC_THREADS; u < U; u += TC_THREADS) put(u, entry(n, a, u));
        if (tid < Dp) sh.xn[tid] = px;
        for (uint32_t k = tid + TC_THREADS; k < Dp; k += TC_THREADS) sh.xn[k] = s.D.X[(size_t)n * Dp + k];
        __syncthreads();
        fetch(li + 1);
        float qn = 0.f;   // |x_n|^2, in every warp
        for (uint32_t k = lane; k < Dp; k += 32) qn += sh.xn[k] * sh.xn[k];
        for (int o = 16; o; o >>= 1) qn += __shfl_xor_sync(FULL, qn, o);
        const bool samp = sampled_node(n);
        for (uint32_t j0 = 0; j0 < a && !aborted; j0 += TC_N) {
            const uint32_t nb = min(TC_N, a - j0);   // new columns [j0, j0 + nb), also the tile's rows 0 .. nb - 1
            bool first = true;
            // their partners: the block itself, then the entries after it, TC_REST at a time
            for (uint32_t us = j0 + nb; first || us < U; us += TC_REST, first = false) {
                const uint32_t nr = us < U ? min(TC_REST, U - us) : 0u;
                stage_rows<PREC>(s, sh, TileRows{j0, first ? nb : 0u, us, nr}, qn, gam, warp, lane);
                tc::fence_before_sync();
                __syncthreads();
                if (warp == 0 && tc::elect_one()) {
                    tc::fence_after_sync();
                    const uint32_t aa = tc::smem_addr(sh.buf);
                    if constexpr (PREC == 1) {   // K = 32 bytes per step, rows of Dp bytes
                        const uint32_t idesc = tc::idesc_e4m3_f32(TC_M, TC_N);
                        for (uint32_t kk = 0; kk < Dp / 32; ++kk) {
                            const uint64_t de = tc::smem_desc(aa + kk * 256, 128, Dp * 8);
                            tc::mma_e4m3(tmem, de, de, idesc, kk > 0);
                        }
                    } else {
                        const uint32_t idesc = tc::idesc_bf16_f32(TC_M, TC_N);
                        for (uint32_t kk = 0; kk < Dp / 16; ++kk) {
                            const uint64_t de = tc::smem_desc(aa + kk * 256, 128, Dp * 16);
                            tc::mma_bf16(tmem, de, de, idesc, kk > 0);
                        }
                    }
                    tc::mma_commit(&mbar);
                }
                const bool ok = __all_sync(FULL, tc::mbar_wait(&mbar, phase, TC_WAIT_CYCLES));
                tc::fence_after_sync();

                // ---- epilogue: this thread's row against the columns
                const uint32_t u = warp == 0 ? j0 + lane : us + 32 * (warp - 1) + lane;
                const bool in = warp == 0 ? first && (uint32_t)lane < nb : u < us + nr;
                const float4 ua = in ? sh.tA[u] : make_float4(0.f, 0.f, 0.f, __uint_as_float(NO_ID));
                const bool uval = __float_as_uint(ua.w) != NO_ID;
                const uint32_t idu = uval ? __float_as_uint(ua.w) : 0u;
                const bool unew = u < a;
                const float2 uc = uval ? sh.tC[u] : make_float2(0.f, 0.f);
                const float2 uf = (PREC == 1 && uval) ? sh.tF[u] : make_float2(1.f, 1.f);
                const float k2 = 2.f * et * ua.y;
                const bool work = ok && __any_sync(FULL, in);
                unsigned pmask[2] = {0u, 0u};
#pragma unroll
                for (int part = 0; part < 2; ++part) {
                    const uint32_t cb = 16 * part;
                    if (!work || cb >= nb) break;   // warp-uniform
                    float v[16];
                    tc::tmem_ld16(tmem + ((uint32_t)(32 * warp) << 16) + cb, v);
                    // the pairs of this row: every column, in the block's own rows those after the row
                    const uint32_t cols = min(16u, nb - cb);
                    unsigned need = uval ? (1u << cols) - 1u : 0u;
                    if (warp == 0 && (uint32_t)lane >= cb) need &= lane - cb >= 15 ? 0u : ~0u << (lane - cb + 1);
                    unsigned pm = 0;
                    // the test of the pair with new entry j, the columns' entry c
                    auto test = [&](uint32_t j, float gram, float &g, float &etp, float4 &ja) {
                        ja = sh.tA[j];   // rows up to Umax: past j1 masked below
                        g = gram;
                        etp = et;
                        float t2 = k2 * ja.y;
                        if constexpr (PREC == 1) {   // the scales, and this pair's relative error
                            const float2 jf = sh.tF[j];
                            g = g * uf.x * jf.x;
                            etp = filter_et8(uf.y, jf.y, g8);
                            t2 = 2.f * etp * ua.y * ja.y;
                        }
                        const float2 jc = metric == METRIC_ANGULAR ? sh.tC[j] : make_float2(0.f, 0.f);
                        return filter_pair((FilterMetric)metric, g, t2, gam, ua.x, ja.x, ua.z, ja.z, uc.x, jc.x, uc.y, jc.y);
                    };
#pragma unroll
                    for (int c = 0; c < 16; ++c) {
                        float4 ja;
                        float g, etp;
                        const FilterTest ft = test(j0 + cb + c, v[c], g, etp, ja);
                        if (!(ft.lhs > ft.rhs)) pm |= 1u << c;
                        const uint32_t idj = __float_as_uint(ja.w);
                        if (idj == NO_ID || (unew && idj == idu)) need &= ~(1u << c);
                    }
                    pm &= need;
                    comps += __popc(need);
                    pmask[part] = pm;
                    if (samp) {   // this node's pairs to the FP64 check
                        const uint32_t have = __popc(need);
                        uint32_t end = have;
                        for (int o = 1; o < 32; o <<= 1) {
                            const uint32_t t = __shfl_up_sync(FULL, end, o);
                            if (lane >= o) end += t;
                        }
                        uint32_t at = 0;
                        if (lane == 31 && end) at = atomicAdd(jq.stail, end);
                        at = __shfl_sync(FULL, at, 31) + end - have;
#pragma unroll 1   // (one copy: rarely run)
                        for (int c = 0; c < (int)cols; ++c) {
                            const bool mine = (need >> c) & 1u;
                            if (!__any_sync(FULL, mine)) continue;
                            float gram = 0.f;
#pragma unroll
                            for (int k = 0; k < 16; ++k)
                                if (k == c) gram = v[k];
                            float4 ja;
                            float g, etp;
                            const FilterTest ft = test(j0 + cb + c, gram, g, etp, ja);
                            const uint4 e = make_uint4(n, idu, __float_as_uint(ja.w), __float_as_uint(g));
                            const float4 f = make_float4(etp, ft.lhs, fmaxf(ua.z, ja.z), (pm >> c) & 1u ? 0.f : 1.f);
                            if (mine && at < JOIN_TC_SAMPLES) { jq.sample[at] = e; jq.filter[at] = f; }
                            unsigned over = __ballot_sync(FULL, mine && at >= JOIN_TC_SAMPLES);
                            for (; over; over &= over - 1) {   // past the record's end: here
                                const int src = __ffs(over) - 1;
                                SampleTally t{};
                                sample_pair(s, __shfl_sync(FULL, e.x, src), __shfl_sync(FULL, e.y, src),
                                            __shfl_sync(FULL, e.z, src), __uint_as_float(__shfl_sync(FULL, e.w, src)),
                                            make_float4(__shfl_sync(FULL, f.x, src), __shfl_sync(FULL, f.y, src),
                                                        __shfl_sync(FULL, f.z, src), __shfl_sync(FULL, f.w, src)),
                                            lane, t);
                                if (lane == 0) t.add(s.tc);
                            }
                            at += mine;
                        }
                    }
                }
                // append the survivors: one queue atomic per warp
                const uint32_t mine = __popc(pmask[0]) + __popc(pmask[1]);
                uint32_t incl = mine;
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t t = __shfl_up_sync(FULL, incl, o);
                    if (lane >= o) incl += t;
                }
                unsigned long long pos = 0;
                if (lane == 31 && incl) pos = atomicAdd(jq.tail, (unsigned long long)incl);
                pos = __shfl_sync(FULL, pos, 31) + incl - mine;
                passed += mine;
#pragma unroll
                for (int part = 0; part < 2; ++part) {
                    unsigned pm = pmask[part];
                    const uint32_t cb = 16 * part;
                    while (pm) {
                        const int c = __ffs(pm) - 1;
                        pm &= pm - 1;
                        const uint32_t idj = __float_as_uint(sh.tA[j0 + cb + c].w);
                        jq.x[pos] = unew ? min(idu, idj) : idj;
                        jq.y[pos] = unew ? max(idu, idj) : idu;
                        jq.n[pos] = n;
                        ++pos;
                    }
                }
                tc::fence_before_sync();
                if (__syncthreads_or(!ok)) {   // TMEM and the tile are free again
                    if (tid == 0) raise_error(s.err, ERR_TC_TIMEOUT);
                    aborted = true;
                    break;
                }
                phase ^= 1;
            }
        }
        }
        if (aborted) break;
        __syncthreads();   // the claimed list is free again
    }

    if (aborted) tc::mbar_wait(&mbar, phase, TC_WAIT_CYCLES);   // the MMA still in flight, bounded
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    if (warp == 0) tc::tmem_free(tmem, TC_TMEM_COLS);

    for (int o = 16; o; o >>= 1) {
        comps += __shfl_xor_sync(FULL, comps, o);
        passed += __shfl_xor_sync(FULL, passed, o);
    }
    if (lane == 0) {
        if (comps) { atomicAdd(s.n_comps, comps); atomicAdd(&s.tc->pairs, comps); }
        if (passed) atomicAdd(&s.tc->rechecked, passed);
    }
}

// The sampled nodes' pairs, a warp each.  Evaluated where they were found, by the
// node's own warps, the pairs of one node took about 1 ms: the tail of every
// launch, in which the other SMs waited (200k x 96 whole build 153 -> 126 ms).
__global__ void __launch_bounds__(256) join_sample_kernel(const __grid_constant__ BuildState s, JoinQueue jq) {
    const int lane = threadIdx.x & 31;
    const uint32_t total = min(*jq.stail, JOIN_TC_SAMPLES), nw = gridDim.x * 8;
    SampleTally t{};
    for (uint32_t e = blockIdx.x * 8 + (threadIdx.x >> 5); e < total; e += nw) {
        const uint4 p = jq.sample[e];
        sample_pair(s, p.x, p.y, p.z, __uint_as_float(p.w), jq.filter[e], lane, t);
    }
    if (lane == 0 && t.sampled) t.add(s.tc);
}

// Phase 2: the queued pairs, 8 per warp pass: canonical FP32 distance by
// 4-lane groups, the unlocked radius pre-test of both endpoints, then the
// inserts, recorded or locked (Nhood::parallel_try_insert, kgraph.cpp:723-736) -- the
// CUDA-core join's inner loop, at full occupancy.
__global__ void __launch_bounds__(256) join_insert_kernel(BuildState s, JoinQueue jq) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const unsigned long long total = *jq.tail;
    const unsigned long long w0 = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const unsigned long long nw = (gridDim.x * blockDim.x) >> 5;
    InsertTally tally;
    // one contiguous run of entries per warp: a node's pairs share rows
    const unsigned long long chunk = ((total + nw - 1) / nw + 7) & ~7ull;
    const unsigned long long end = min(total, (w0 + 1) * chunk);
    for (unsigned long long base = w0 * chunk; base < end; base += 8) {
        const unsigned long long e = base + g;
        const bool valid = e < end;
        const uint32_t x = valid ? jq.x[e] : 0u, y = valid ? jq.y[e] : 0u, nn = valid ? jq.n[e] : 0u;
        const float dd = pair_dist(s.D, x, y, t, FULL);
        // deferred (the offers to the grouped merge) or locked inserts; the pairs were counted by the filter
        unsigned long long comps = 0;
        bool uu = false;
        settle_pass(s, lane, t, valid, x, y, dd, nn, comps, uu, tally, true);
    }
    if (lane == 0 && tally.attempts) {
        atomicAdd(s.inserts, (unsigned long long)tally.attempts);
        atomicAdd(s.inserts + 1, (unsigned long long)tally.landed);
    }
}

// Upper bound of the pairs node n's join produces: a(a-1)/2 + a*b.
__global__ void join_worst_kernel(BuildState s, uint64_t *worst) {
    for (uint32_t n = blockIdx.x * blockDim.x + threadIdx.x; n <= s.D.n; n += gridDim.x * blockDim.x) {
        uint64_t w = 0;
        if (n < s.D.n) {
            const uint64_t a = min(s.cnt_new[n], s.NEWCAP), b = min(s.cnt_old[n], s.OLDCAP);
            w = a * (a > 0 ? a - 1 : 0) / 2 + a * b;
        }
        worst[n] = w;
    }
}

// Round boundaries: bounds[k] = first node whose exclusive prefix of worst-case
// pairs reaches k * slab (bounds[0] = 0, bounds[R] = N).  A round's pairs are
// then below slab + one node's worst case, which the queue holds.
__global__ void join_bounds_kernel(const uint64_t *pre, uint32_t N, uint64_t slab, uint32_t R, uint32_t *bounds) {
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k <= R; k += gridDim.x * blockDim.x) {
        uint32_t r;
        if (k == 0) r = 0;
        else if (k == R) r = N;
        else {
            const uint64_t key = (uint64_t)k * slab;
            uint32_t lo = 0, hi = N;
            while (lo < hi) {
                const uint32_t mid = (lo + hi) >> 1;
                if (pre[mid] < key) lo = mid + 1; else hi = mid;
            }
            r = lo;
        }
        bounds[k] = r;
    }
}

size_t join_tc_tile(const BuildState &s, int prec) { return (size_t)TC_M * s.D.ld * (prec ? 1 : 2); }
size_t join_tc_smem(const BuildState &s, int prec) {
    const size_t Umax = (size_t)s.NEWCAP + s.OLDCAP;
    return join_tc_tile(s, prec) + (size_t)s.D.ld * 4 + (Umax + TC_PAD) * (prec ? 32 : 24);
}

}  // namespace

// The rows and lists the join takes, else kg_build refuses: two tiles, a row and
// 28 bytes per list entry within 200 KB.  (Of them every one fits the 227 KB of a
// CTA as join_tc_smem lays it out: the longest lists go with the narrowest rows,
// E4M3 rows of 32, 7,017 entries, 229,280 bytes.)
bool join_tc_supported(const BuildState &s, int prec) {
    const size_t Umax = (size_t)s.NEWCAP + s.OLDCAP;
    return s.D.ld % (prec ? 32 : 16) == 0 && 2 * join_tc_tile(s, prec) + (size_t)s.D.ld * 4 + Umax * 28 <= 200 * 1024;
}

uint64_t join_tc_node_max(const BuildState &s) {
    return (uint64_t)s.NEWCAP * (s.NEWCAP - 1) / 2 + (uint64_t)s.NEWCAP * s.OLDCAP;
}

cudaError_t join_tc_worst(cudaStream_t st, const BuildState &s, uint64_t *worst) {
    join_worst_kernel<<<(s.D.n + 256) / 256, 256, 0, st>>>(s, worst);
    return cudaGetLastError();
}

cudaError_t join_tc_bounds(cudaStream_t st, const uint64_t *pre, uint32_t N, uint64_t slab, uint32_t R,
                           uint32_t *bounds) {
    join_bounds_kernel<<<(R + 128) / 128, 128, 0, st>>>(pre, N, slab, R, bounds);
    return cudaGetLastError();
}

cudaError_t launch_join_tc(int num_sms, int grid_insert, cudaStream_t st, const BuildState &s, JoinQueue jq,
                           uint32_t round, int prec) {
    auto kern = prec ? join_tc_kernel<1> : join_tc_kernel<0>;
    const size_t smem = join_tc_smem(s, prec);
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout,
                             (int)cudaSharedmemCarveoutMaxShared);
    if (e != cudaSuccess) return e;
    // CTAs per SM from the kernel's registers and shared memory (at most
    // JOIN_TC_MAX_CTAS_PER_SM, which bounds the TMEM columns in use per SM).
    cudaFuncAttributes fa{};
    if ((e = cudaFuncGetAttributes(&fa, kern)) != cudaSuccess) return e;
    int dev = 0, smem_sm = 0, smem_rsv = 0, regs_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
    cudaDeviceGetAttribute(&smem_rsv, cudaDevAttrReservedSharedMemoryPerBlock, dev);
    cudaDeviceGetAttribute(&regs_sm, cudaDevAttrMaxRegistersPerMultiprocessor, dev);
    const size_t per_cta_smem = smem + fa.sharedSizeBytes + (size_t)smem_rsv;
    const int regs_cta = ((fa.numRegs + 7) / 8 * 8) * TC_THREADS;
    int occ = JOIN_TC_MAX_CTAS_PER_SM;
    occ = std::min<int>(occ, (int)((size_t)smem_sm / per_cta_smem));
    occ = std::min<int>(occ, regs_cta ? regs_sm / regs_cta : occ);
    if (occ < 1) return cudaErrorInvalidConfiguration;
    cudaMemsetAsync(jq.tail, 0, 16, st);   // tail, work, stail
    kern<<<num_sms * occ, TC_THREADS, smem, st>>>(s, s.NEWCAP + s.OLDCAP, jq, round);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    join_sample_kernel<<<num_sms * 8, 256, 0, st>>>(s, jq);
    cudaFuncSetAttribute(join_insert_kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                         (int)cudaSharedmemCarveoutMaxL1);
    join_insert_kernel<<<grid_insert, 256, 0, st>>>(s, jq);
    return cudaGetLastError();
}

}  // namespace kgb
