// Exact brute-force k-NN on the fifth-generation tensor cores:
// SearchOracle::search (kgraph.cpp:231-252) for a whole batch of queries, the
// path of every query with P >= N (kgraph.cpp:427-433), of searches without an
// index (python-api.cpp:303-314) and of the Python module's blas=True
// (python-api.cpp:131-205, whose OpenBLAS product it replaces).
//
// The result must be the reference's bit for bit: the K rows with the smallest
// canonical FP32 distance (kg_common.cuh), ties by id (the reference scans in
// id order and inserts after equal distances), distances above epsilon left
// out.  The tensor cores only choose which rows are worth the canonical FP32
// evaluation:
//
//   1. rows and queries are rounded to BF16 -- centred on the dataset mean
//      first (euclidean, l2sqr) unless BF16 holds the rows exactly; per row the
//      exact ||x~||^2 and a rigorous bound e_x >= ||(x - mu) - x~|| are kept
//      (FP64, rounded outward), per query the same.  The rows are stored in a
//      spread order (position p holds row p * A mod n, A coprime to n near
//      0.618 n), so that any prefix is an even sample of the dataset;
//   2. sample sweep: the products of the queries with the first 1/4 to 1/16 of
//      the rows (tcgen05.mma kind::f16, FP32 in TMEM).  With u = q~.x~ -
//      ||x~||^2/2 (euclidean, l2sqr) or q~.x~ (angular, whose rows are divided
//      by their norms first), larger is nearer; the largest u of every 32 rows
//      is kept, and the K-th largest of these maxima, u_K, is met by at least K
//      rows.  The ||x~||^2/2 comes out of the product itself: three more
//      columns hold it (BF16 parts of 8 bits each, 24 together) against ones;
//   3. per query a rigorous margin M >= |canonical - d~| for every row (from the
//      BF16 errors, the FP32 accumulation bound of the products, and the
//      canonical distance's own rounding bound; dataset-wide maxima of the row
//      terms).  K rows have d~ <= d~(u_K), so every row of the exact top K has
//      d~ <= d~(u_K) + 2M;
//   4. full sweep: the rows within that bound are the candidates, about K over
//      the sampled share;
//   5. one warp per query evaluates its candidates with the canonical FP32
//      distance and keeps the K smallest by (distance, id) within epsilon --
//      the reference's list;
//   6. a query with more candidates than its room goes through 2 to 5 once more,
//      now with all rows as the sample, which leaves about K candidates instead
//      of K over the share, and with twice the room.  Only where the margin alone
//      admits more rows than that is it scanned in full on the CUDA cores
//      (counted in the statistics), which takes a warp 37 ms for 200k rows of
//      128: 1,000 queries, K = 10, on a float mixture of that size with centres
//      twice the spread, 605 of them with too many candidates from the sample,
//      34 ms without this step, 0.96 ms with it.
//
// All tensor-core waits are bounded: a wait that runs out raises
// ERR_TC_TIMEOUT, waits (bounded) for what is in flight, frees the CTA's TMEM
// and returns; the host turns the error bit into KG_E_DEVICE.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstring>
#include <numeric>
#include <cuda_bf16.h>
#include "kg_ctx.h"
#include "kg_bruteforce.h"
#include "kg_gemm.h"
#include "kg_tc.cuh"
#include "kg_warp.cuh"

namespace kgb {
namespace {

constexpr long long BF_WAIT_CYCLES = 2000000000ll;
constexpr float U24 = 5.9604645e-8f;      // 2^-24
constexpr float U23 = 1.1920929e-7f;      // 2^-23

__device__ __forceinline__ unsigned long long ordered_u64(double v) {
    unsigned long long u = (unsigned long long)__double_as_longlong(v);
    return (u & 0x8000000000000000ull) ? ~u : (u | 0x8000000000000000ull);
}

// Column sums of the dataset in FP64 (the mean for centring).
__global__ void colsum_kernel(DataView D, double *sum) {
    const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= D.d) return;
    const uint32_t parts = gridDim.y, part = blockIdx.y;
    const uint32_t chunk = (D.n + parts - 1) / parts;
    double s = 0.0;
    for (uint32_t r = part * chunk; r < min(D.n, (part + 1) * chunk); ++r) s += (double)D.X[(size_t)r * D.ld + c];
    atomicAdd(sum + c, s);
}

__global__ void mean_kernel(const double *sum, uint32_t d, uint32_t ld, uint32_t n, int centre, float *mu) {
    const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c < ld) mu[c] = (centre && c < d) ? (float)(sum[c] / (double)n) : 0.f;
}

// One warp per row: v = bf16(x - mu) (FP32 subtraction, then rounding; angular:
// bf16(x / n_x), zero for a zero row), the exact ||v||^2 and e >= ||(x - mu) - v||
// (angular: ||x / n_x - v||; FP64, rounded up), at the row's position in the
// spread order (row * inv mod n); euclidean and l2sqr: also -||v||^2 / 2 as three
// BF16 parts in the row of Xe.  Dataset-wide: max ||v||, max e, max canonical
// norm term and min positive canonical norm (angular); a NaN or infinite row
// leaves an infinite maximum.
__global__ void prep_rows_kernel(DataView D, const float *mu, uint64_t inv, __nv_bfloat16 *Xb, uint4 *Xe,
                                 unsigned long long *ext) {
    const int lane = threadIdx.x & 31;
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
    const bool ang = D.metric == METRIC_ANGULAR;
    double m0 = 0.0, m1 = 0.0, m2 = 0.0, m3 = INFINITY;   // this warp's extremes (lane 0)
    for (uint32_t row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; row < D.n; row += warps) {
        const float *x = D.X + (size_t)row * D.ld;
        const size_t at = (size_t)(row * inv % D.n);
        const float nt = D.norms ? D.norms[row] : 0.f;   // canonical norm term (euclidean / angular)
        double e2 = 0.0, v2 = 0.0;
        for (uint32_t j = lane; j < D.ld; j += 32) {
            float xc = 0.f;
            double xd = 0.0;
            if (j < D.d) {
                xc = ang ? (nt > 0.f ? x[j] / nt : 0.f) : __fsub_rn(x[j], mu[j]);
                xd = ang ? (nt > 0.f ? (double)x[j] / (double)nt : (double)x[j]) : (double)x[j] - (double)mu[j];
            }
            const __nv_bfloat16 b = __float2bfloat16_rn(xc);
            Xb[at * D.ld + j] = b;
            const double vb = (double)__bfloat162float(b), ex = xd - vb;
            e2 += ex * ex;
            v2 += vb * vb;
        }
        for (int o = 16; o; o >>= 1) {
            e2 += __shfl_xor_sync(FULL, e2, o);
            v2 += __shfl_xor_sync(FULL, v2, o);
        }
        if (lane == 0) {
            const float e = e2 > 0.0 ? __double2float_ru(sqrt(e2) * (1.0 + 1e-12)) : 0.f;
            if (!ang) {   // v2 is exact: BF16 squares sum exactly in FP64 for d <= 2^20
                const float h = -0.5f * (float)v2;
                const __nv_bfloat16 h0 = __float2bfloat16_rn(h);
                const float r1 = h - __bfloat162float(h0);
                const __nv_bfloat16 h1 = __float2bfloat16_rn(r1), h2 = __float2bfloat16_rn(r1 - __bfloat162float(h1));
                Xe[at] = make_uint4((uint32_t)__bfloat16_as_ushort(h0) | (uint32_t)__bfloat16_as_ushort(h1) << 16,
                                    (uint32_t)__bfloat16_as_ushort(h2), 0u, 0u);
            }
            m0 = fmax(m0, v2 < INFINITY ? sqrt(v2) : INFINITY);
            m1 = fmax(m1, e2 < INFINITY ? (double)e : INFINITY);
            m2 = fmax(m2, nt < INFINITY ? (double)nt : INFINITY);
            if (ang && nt > 0.f) m3 = fmin(m3, (double)nt);
        }
    }
    if (lane == 0) {
        atomicMax(ext + 0, ordered_u64(m0));
        atomicMax(ext + 1, ordered_u64(m1));
        atomicMax(ext + 2, ordered_u64(m2));
        if (m3 < INFINITY) atomicMin(ext + 3, ordered_u64(m3));
    }
}

// One warp per query: the same centring and rounding, and the canonical norm
// term of the query (the search kernel's computation: python-api.cpp:98-101).
// `map`, if given, holds the queries' rows.
__global__ void prep_queries_kernel(DataView D, const float *mu, const float *Q, uint32_t q_ld, const uint32_t *map,
                                    uint32_t nq, __nv_bfloat16 *Qb, float4 *qmeta) {
    const int lane = threadIdx.x & 31;
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t qi = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; qi < nq; qi += warps) {
        const float *q = Q + (size_t)(map ? map[qi] : qi) * q_ld;
        double e2 = 0.0, v2 = 0.0;
        for (uint32_t j = lane; j < D.ld; j += 32) {
            const float xc = j < D.d ? __fsub_rn(q[j], mu[j]) : 0.f;
            const __nv_bfloat16 b = __float2bfloat16_rn(xc);
            Qb[(size_t)qi * D.ld + j] = b;
            const double vb = (double)__bfloat162float(b);
            const double ex = j < D.d ? ((double)q[j] - (double)mu[j]) - vb : 0.0;
            e2 += ex * ex;
            v2 += vb * vb;
        }
        for (int o = 16; o; o >>= 1) {
            e2 += __shfl_xor_sync(FULL, e2, o);
            v2 += __shfl_xor_sync(FULL, v2, o);
        }
        float qn = 0.f;
        if (D.metric != METRIC_L2SQR) {
            // the canonical order needs the query's padding columns at zero: read through a masked copy
            float n2;
            {
                float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
                const int t = lane & 3;
                const uint32_t chunks = D.d >> 4;
                for (uint32_t c = 0; c < chunks; ++c) lane_acc(acc, ld4(q + 16 * c + 4 * t), ld4(q + 16 * c + 4 * t), METRIC_EUCLIDEAN);
                n2 = group4_reduce(acc, FULL);
                uint32_t i = chunks << 4;
                if (D.d - i >= 8)
                    for (uint32_t e = i + 8; i < e; ++i) n2 = __fadd_rn(n2, __fmul_rn(q[i], q[i]));
                for (; i < D.d; ++i) n2 = __fmaf_rn(q[i], q[i], n2);
            }
            qn = norm_term(n2, D.metric);
        }
        if (lane == 0) {
            const float e = e2 > 0.0 ? __double2float_ru(sqrt(e2) * (1.0 + 1e-12)) : 0.f;
            qmeta[qi] = make_float4((float)v2, e, qn, 0.f);
        }
    }
}

// ---------------------------------------------------------------- the sweeps
// A CTA multiplies 128 or 256 queries (one or two M = 128 tiles, resident in
// shared memory) with tiles of 256 rows that TMA brings through a ring of
// 64-column boxes.  Two TMEM accumulators of 256 columns take turns, so the
// epilogue of one product runs under the MMAs of the next; with two query
// tiles each row tile serves both, which halves the rows' traffic from L2
// (6.4 TB/s at the tensor cores' full rate instead of 12.8).
// Warps 0-7: epilogue (TMEM lanes 32 (w % 4), columns 128 (w / 4)), warp 8: TMA
// producer, warp 9: MMA issuer.
// Schedule: the row tiles go in chunks that stay in L2; within a chunk the
// (query tile, row tile) pairs, query tile slowest, are cut into equal runs,
// one per CTA, the same in every chunk, so a CTA meets the same few query
// tiles in every chunk and no wave is left half empty.
// With the rows' norms folded into the product the epilogue only takes maxima:
// adding them from shared memory there cost the MMAs their operand bandwidth
// (a 16-byte broadcast read is four shared-memory cycles).
// Bound: the MMAs and, behind them, the wait for row boxes (four fit beside two
// query tiles).  10k queries x 1M x 128, K = 10, whole call: 105 ms with 128 x
// 128 tiles that one warp group staged, multiplied and folded in turn, two sweeps
// over all rows and a sorted insert per row; 3.3 ms now (2.56 TFLOP: 770
// TFLOP/s), of which the sample sweep 0.2, threshold 0.15, recheck 0.15 ms.
constexpr int BF_THREADS = 320;
constexpr int BF_EPI = 8;                     // epilogue warps
constexpr uint32_t BF_Q = 128;                // queries per M tile (TMEM lanes)
constexpr uint32_t BF_R = 256;                // rows per tile (TMEM columns per accumulator)
constexpr uint32_t BF_QBOX = BF_Q * 128, BF_RBOX = BF_R * 128;   // bytes of a 64-column box
constexpr uint32_t BF_QEXT = BF_Q * 32, BF_REXT = BF_R * 32;     // bytes of the norm columns (16)
constexpr uint32_t BF_MAX_ST = 6;
constexpr size_t BF_CHUNK_BYTES = 48u << 20;
constexpr size_t BF_SMEM = 222 * 1024;       // with the static part, within the 227 KB of a CTA
// Queries per pass over the rows: as many as have their group maxima and candidates within
// BF_WORK_BYTES (of a group's 4 bytes a query has up to n / 32), at most BF_BATCH.
constexpr size_t BF_BATCH = 32768;
constexpr size_t BF_WORK_BYTES = (size_t)512 << 20;
constexpr uint32_t BF_MAX_GROUPS32 = 16384;   // above it groups are 128 rows

struct SweepArgs {
    uint32_t n, ld, nq, nsub;
    uint32_t stages, estages;   // boxes in the ring; norm-column tiles beside it (0: angular)
    uint32_t qt, rt, rtc;    // query tiles (of nsub x 128), row tiles, row tiles per chunk
    // sample sweep: the largest u of every `width` rows (128, 32, 4 or 1), [group][nqp]
    float *gmax;
    uint32_t nqp, width;
    // full sweep: per query and segment (2 per CTA that meets the query's tile) up to scap positions
    const float *thresh;
    uint32_t *cand, *cand_n, nseg, scap;
    uint32_t *err;
};

// The tiles of one CTA, in order.
struct SweepWalk {
    uint32_t lo, hi, chunk, i;
    __device__ SweepWalk(const SweepArgs &a) : chunk(0) {
        const uint64_t T = (uint64_t)a.qt * a.rtc;
        lo = (uint32_t)(T * blockIdx.x / gridDim.x);
        hi = (uint32_t)(T * (blockIdx.x + 1) / gridDim.x);
        i = lo;
    }
    __device__ bool next(const SweepArgs &a, uint32_t &q, uint32_t &r) {
        while (lo < hi) {
            if (i == hi) { i = lo; ++chunk; }
            if ((uint64_t)chunk * a.rtc >= a.rt) return false;
            q = i / a.rtc;
            r = chunk * a.rtc + i % a.rtc;
            ++i;
            if (r < a.rt) return true;
        }
        return false;
    }
};
// The first CTA whose run meets query tile q.
__host__ __device__ inline uint32_t sweep_first_cta(uint32_t q, uint32_t qt, uint32_t rtc, uint32_t grid) {
    const uint64_t T = (uint64_t)qt * rtc, t = (uint64_t)q * rtc;
    uint32_t b = (uint32_t)(t * grid / T);
    while (T * (b + 1) / grid <= t) ++b;
    return b;
}

template <int MODE>
__global__ void __launch_bounds__(BF_THREADS, 1)
    bf_sweep_kernel(const __grid_constant__ CUtensorMap tQ, const __grid_constant__ CUtensorMap tX,
                    const __grid_constant__ CUtensorMap tE, SweepArgs a) {
    extern __shared__ uint8_t bf_raw[];
    uint8_t *sm = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(bf_raw) + 1023) & ~(uintptr_t)1023);
    __shared__ __align__(8) uint64_t full[BF_MAX_ST], empty[BF_MAX_ST], acc_full[2], acc_empty[2], q_full, q_empty, done;
    __shared__ uint32_t tmem_base;
    __shared__ volatile uint32_t fail;
    __shared__ uint32_t issued, q_issued;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t nb = (a.ld + 63) / 64, ksteps = a.ld / 16, ST = a.stages, nsub = a.nsub;
    const uint32_t EST = a.estages;
    uint8_t *sQ = sm, *sR = sm + nsub * nb * BF_QBOX, *sE = sR + ST * BF_RBOX, *sOne = sE + EST * BF_REXT;
    if (EST && tid < (int)BF_Q) {   // the queries' side of the norm columns: three ones (32-byte swizzle)
        uint4 *o = reinterpret_cast<uint4 *>(sOne + tid * 32);
        const uint32_t hi = (tid >> 2) & 1;
        o[hi] = make_uint4(0x3F803F80u, 0x3F80u, 0u, 0u);
        o[hi ^ 1u] = make_uint4(0u, 0u, 0u, 0u);
    }
    tc::fence_async_shared();
    if (warp == 9) tc::tmem_alloc(&tmem_base, 2 * BF_R);
    if (tid == 0) {
        for (uint32_t s = 0; s < BF_MAX_ST; ++s) { tc::mbar_init(&full[s], 1); tc::mbar_init(&empty[s], 1); }
        for (int s = 0; s < 2; ++s) { tc::mbar_init(&acc_full[s], 1); tc::mbar_init(&acc_empty[s], BF_EPI); }
        tc::mbar_init(&q_full, 1);
        tc::mbar_init(&q_empty, 1);
        tc::mbar_init(&done, 1);
        fail = 0;
        issued = 0;
        q_issued = 0;
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = tmem_base;
    uint32_t q, r;
    if (warp == 8 && lane == 0) {
        SweepWalk w(a);
        uint32_t cur = 0xFFFFFFFFu, visits = 0, c = 0, tile = 0;   // c: boxes issued
        while (!fail && w.next(a, q, r)) {
            if (q != cur) {   // the query tiles of this visit, once the last visit's MMAs have read theirs
                if (visits && !tc::mbar_wait(&q_empty, (visits - 1) & 1u, BF_WAIT_CYCLES)) { fail = 1; break; }
                tc::mbar_expect_tx(&q_full, nsub * nb * BF_QBOX);
                for (uint32_t s = 0; s < nsub; ++s)
                    for (uint32_t j = 0; j < nb; ++j)
                        tc::tma_load_2d(sQ + (s * nb + j) * BF_QBOX, &tQ, 64 * j, (q * nsub + s) * BF_Q, &q_full);
                cur = q;
                ++visits;
            }
            for (uint32_t j = 0; j < nb; ++j, ++c) {
                const uint32_t s = c % ST;
                if (c >= ST && !tc::mbar_wait(&empty[s], ((c / ST) & 1u) ^ 1u, BF_WAIT_CYCLES)) { fail = 1; break; }
                // a tile's norm columns come with its last box; their slot's previous tile is done by then
                // (estages x nb >= stages)
                const bool ext = EST && j == nb - 1;
                tc::mbar_expect_tx(&full[s], BF_RBOX + (ext ? BF_REXT : 0u));
                tc::tma_load_2d(sR + s * BF_RBOX, &tX, 64 * j, r * BF_R, &full[s]);
                if (ext) tc::tma_load_2d(sE + tile % EST * BF_REXT, &tE, 0, r * BF_R, &full[s]);
            }
            ++tile;
        }
        issued = c;
        q_issued = visits;
    } else if (warp == 9) {   // the whole warp, so that the operands stay uniform; one lane issues
        SweepWalk w(a);
        const uint32_t idesc = tc::idesc_bf16_f32(BF_Q, BF_R);
        const uint64_t qd = tc::smem_desc_sw128(tc::smem_addr(sQ), 16, 1024);
        const uint64_t rd = tc::smem_desc_sw128(tc::smem_addr(sR), 16, 1024);
        const uint32_t tm = __reduce_or_sync(FULL, tmem);
        const bool one = tc::elect_one();
        const uint64_t ed = tc::smem_desc_sw32(tc::smem_addr(sE), 16, 256);
        const uint64_t od = tc::smem_desc_sw32(tc::smem_addr(sOne), 16, 256);
        uint32_t cur = 0xFFFFFFFFu, visits = 0, slot0 = 0, ph0 = 0, es = 0, jobs = 0;   // the tile's first box and its phase
        bool go = true;
        while (go && w.next(a, q, r)) {
            if (q != cur) {
                if (visits && one) tc::mma_commit(&q_empty);
                if (fail || !tc::mbar_wait(&q_full, visits & 1u, BF_WAIT_CYCLES)) { fail = 1; break; }
                cur = q;
                ++visits;
            }
            for (uint32_t s = 0; s < nsub && go; ++s, ++jobs) {
                const uint32_t acc = jobs & 1u;
                if (fail || (jobs >= 2 && !tc::mbar_wait(&acc_empty[acc], ((jobs >> 1) & 1u) ^ 1u, BF_WAIT_CYCLES))) {
                    fail = 1;
                    go = false;
                    break;
                }
                uint32_t slot = slot0, ph = ph0;
                for (uint32_t j = 0; j < nb; ++j) {
                    if (s == 0 && (fail || !tc::mbar_wait(&full[slot], ph, BF_WAIT_CYCLES))) {
                        fail = 1;
                        go = false;
                        break;
                    }
                    tc::fence_after_sync();
                    const uint64_t ad = qd + ((s * nb + j) * BF_QBOX >> 4), bd = rd + (slot * BF_RBOX >> 4);
                    const uint32_t kn = min(ksteps - 4 * j, 4u);
                    if (one) {
#pragma unroll
                        for (uint32_t kk = 0; kk < 4; ++kk)
                            if (kk < kn) tc::mma_bf16(tm + acc * BF_R, ad + 2 * kk, bd + 2 * kk, idesc, (j | kk) ? 1u : 0u);
                        if (EST && j == nb - 1) tc::mma_bf16(tm + acc * BF_R, od, ed + (es * BF_REXT >> 4), idesc, 1u);
                        if (s == nsub - 1) tc::mma_commit(&empty[slot]);
                    }
                    if (++slot == ST) { slot = 0; ph ^= 1u; }
                }
                if (go && one) tc::mma_commit(&acc_full[acc]);
                if (s == nsub - 1) { slot0 = slot; ph0 = ph; }
            }
            if (++es == EST) es = 0;
        }
        if (one) tc::mma_commit(&done);   // arrives when every MMA issued above has completed
    } else if (warp < BF_EPI) {
        SweepWalk w(a);
        const uint32_t half = warp >> 2, row32 = 32 * (warp & 3) + lane;
        uint32_t cur = 0xFFFFFFFFu, seg = 0, jobs = 0;
        uint32_t cnt[2] = {0, 0};
        float thr[2] = {INFINITY, INFINITY};
        auto put_counts = [&]() {
            if (MODE == 1 && cur != 0xFFFFFFFFu)
                for (uint32_t s = 0; s < nsub; ++s) {
                    const uint32_t qi = (cur * nsub + s) * BF_Q + row32;
                    if (qi < a.nq) a.cand_n[(size_t)qi * a.nseg + seg] = s ? cnt[1] : cnt[0];
                }
        };
        bool go = true, have = w.next(a, q, r);
        while (go && have) {
            if (MODE == 1 && q != cur) {
                put_counts();
                cur = q;
                seg = 2 * (blockIdx.x - sweep_first_cta(q, a.qt, a.rtc, gridDim.x)) + half;
                for (uint32_t s = 0; s < nsub; ++s) {
                    const uint32_t qi = (q * nsub + s) * BF_Q + row32;
                    const float t = qi < a.nq ? a.thresh[qi] : INFINITY;
                    const uint32_t k = qi < a.nq ? a.cand_n[(size_t)qi * a.nseg + seg] : 0u;
                    if (s) { thr[1] = t; cnt[1] = k; } else { thr[0] = t; cnt[0] = k; }
                }
            }
            const uint32_t tq = q, tr = r;
            have = w.next(a, q, r);
            for (uint32_t s = 0; s < nsub; ++s, ++jobs) {
                const uint32_t acc = jobs & 1u;
                // bounded in slices, so that an MMA issuer that gave up (it sets `fail`) is noticed early
                bool got = false;
                for (long long spent = 0; !got && !fail && spent < BF_WAIT_CYCLES; spent += 1000000)
                    got = tc::mbar_wait(&acc_full[acc], (jobs >> 1) & 1u, 1000000);
                got = __all_sync(FULL, got);
                if (!got) { fail = 1; go = false; break; }
                tc::fence_after_sync();
                const uint32_t base = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + acc * BF_R + 128 * half;
                const uint32_t qi = (tq * nsub + s) * BF_Q + row32;
                uint32_t buf[2][32];
                float m128 = -INFINITY;   // sample sweep: over this warp's columns of the tile
                tc::tmem_ld32_issue(base, buf[0]);
#pragma unroll
                for (int part = 0; part < 4; ++part) {
                    uint32_t *v = buf[part & 1];
                    tc::tmem_ld32_wait(v);
                    if (part < 3) tc::tmem_ld32_issue(base + 32 * (part + 1), buf[(part + 1) & 1]);
                    const uint32_t p0 = tr * BF_R + 128 * half + 32 * part;   // the first column's row position
                    float u[32];
#pragma unroll
                    for (int k = 0; k < 32; ++k) u[k] = __uint_as_float(v[k]);
                    if (MODE == 0 && p0 + 32 > a.n) {   // rows past the sample (TMA fills zeros)
#pragma unroll
                        for (int k = 0; k < 32; ++k)
                            if (p0 + k >= a.n) u[k] = -INFINITY;
                    }
                    if (MODE == 0) {
                        if (qi < a.nq) {
                            const uint32_t wd = a.width;
                            float *o = a.gmax + (size_t)(p0 / wd) * a.nqp + qi;
                            if (wd == 1) {
#pragma unroll
                                for (int k = 0; k < 32; ++k) o[(size_t)k * a.nqp] = u[k];
                            } else {
                                float m = -INFINITY;
#pragma unroll
                                for (int k = 0; k < 32; k += 4) {
                                    const float f = fmaxf(fmaxf(u[k], u[k + 1]), fmaxf(u[k + 2], u[k + 3]));
                                    if (wd == 4) o[(size_t)(k / 4) * a.nqp] = f;
                                    m = fmaxf(m, f);
                                }
                                m128 = fmaxf(m128, m);
                                if (wd == 32 || (wd == 128 && part == 3)) *o = m128;
                                if (wd == 32) m128 = -INFINITY;
                            }
                        }
                    } else {
                        const float th = s ? thr[1] : thr[0];
                        float m[4];   // the largest of each 8 columns
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            m[k] = fmaxf(fmaxf(fmaxf(u[8 * k], u[8 * k + 1]), fmaxf(u[8 * k + 2], u[8 * k + 3])),
                                         fmaxf(fmaxf(u[8 * k + 4], u[8 * k + 5]), fmaxf(u[8 * k + 6], u[8 * k + 7])));
                        const bool any = fmaxf(fmaxf(m[0], m[1]), fmaxf(m[2], m[3])) >= th;
                        if (__any_sync(FULL, any)) {   // one 32-row piece in six: the columns that reached th
                            uint32_t hits = 0;
#pragma unroll
                            for (int k = 0; k < 4; ++k)
                                if (__any_sync(FULL, m[k] >= th)) {
#pragma unroll
                                    for (int c = 8 * k; c < 8 * k + 8; ++c) hits |= u[c] >= th ? 1u << c : 0u;
                                }
                            uint32_t k1 = s ? cnt[1] : cnt[0];
                            uint32_t *o = a.cand + ((size_t)qi * a.nseg + seg) * a.scap;
                            while (hits) {
                                const uint32_t pos = p0 + __ffs(hits) - 1;
                                hits &= hits - 1;
                                if (pos < a.n) {
                                    if (k1 < a.scap) o[k1] = pos;
                                    ++k1;
                                }
                            }
                            if (s) cnt[1] = k1; else cnt[0] = k1;
                        }
                    }
                }
                tc::fence_before_sync();
                __syncwarp();
                if (lane == 0) tc::mbar_arrive(&acc_empty[acc]);
            }
        }
        put_counts();
    }
    __syncthreads();
    const bool mma_done = tc::mbar_wait(&done, 0, BF_WAIT_CYCLES);
    tc::fence_after_sync();
    if (tid == 0 && (!mma_done || fail)) raise_error(a.err, ERR_TC_TIMEOUT);
    if (fail && warp == 8 && lane == 0) {   // the loads in flight land before the CTA leaves its shared memory
        if (q_issued) tc::mbar_wait(&q_full, (q_issued - 1) & 1u, BF_WAIT_CYCLES);
        for (uint32_t s = 0; s < ST && s < issued; ++s) {
            const uint32_t last = s + (issued - 1 - s) / ST * ST;
            tc::mbar_wait(&full[s], (last / ST) & 1u, BF_WAIT_CYCLES);
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 9) tc::tmem_free(tmem, 2 * BF_R);
}

struct Extents {   // dataset-wide row terms (prep_rows_kernel)
    float vmax, emax, ntmax, ntmin;
};

// Order-preserving map of a float's bits to an unsigned key, and back (NaN: the lowest).
__device__ __forceinline__ uint32_t u_key(float f) {
    const uint32_t u = __float_as_uint(f);
    if (f != f) return 0u;
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float u_val(uint32_t k) {
    return __uint_as_float((k & 0x80000000u) ? (k & 0x7FFFFFFFu) : ~k);
}

// Per query: u_K, the K-th largest of its group maxima (a bitwise search over
// the key bits), the margin M, and the u every candidate reaches.  Eight
// queries per block; gmax is [groups][nqp], so a block reads 32-byte pieces of
// its rows; runs of `fold` groups are folded into one (at most BF_GROUPS).
constexpr uint32_t BF_GROUPS = 2048;
__global__ void __launch_bounds__(256) bf_threshold_kernel(const float *gmax, uint32_t nqp, uint32_t groups,
                                                           uint32_t fold, const float4 *qmeta, uint32_t nq, uint32_t K,
                                                           uint32_t d, uint32_t metric, Extents ex, float *thresh,
                                                           uint32_t *cand_n, uint32_t nseg, uint32_t scap) {
    extern __shared__ uint32_t bf_keys[];   // [8][G]
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t q0 = blockIdx.x * 8, G = (groups + fold - 1) / fold;
    {
        const uint32_t ql = threadIdx.x & 7;
        for (uint32_t g = threadIdx.x >> 3; g < G; g += 32) {
            uint32_t m = 0;
            for (uint32_t k = g * fold; k < min(groups, (g + 1) * fold); ++k)
                if (q0 + ql < nq) m = max(m, u_key(gmax[(size_t)k * nqp + q0 + ql]));
            bf_keys[ql * G + g] = m;
        }
    }
    __syncthreads();
    const uint32_t qi = q0 + w;
    if (qi >= nq) return;   // whole warps
    const uint32_t *keys = bf_keys + w * G;
    uint32_t v = 0;
    if (G >= K)
        for (uint32_t bit = 0x80000000u; bit; bit >>= 1) {   // the largest v that K keys reach
            const uint32_t t = v | bit;
            uint32_t c = 0;
            for (uint32_t g = lane; g < G; g += 32) c += keys[g] >= t ? 1u : 0u;
            c = __reduce_add_sync(FULL, c);
            if (c >= K) v = t;
            if (c == K) break;   // K keys reach v: any such v is a bound
        }
    if (lane != 0) return;
    const float4 qm = qmeta[qi];
    const float qv = sqrtf(qm.x) * (1.f + 4.f * U24);     // ||q~||, rounded up
    const float eq = qm.y, qn = qm.z;
    const float gc = (float)(d / 16 + 24) * U24 * 1.01f;   // canonical distance's relative rounding bound
    float slack;   // d~ of a candidate is at most d~(u_K) + 2M: in u, slack below u_K
    if (metric == METRIC_ANGULAR) {   // d~ = -u / n_q
        const float rq = eq / qn, rx = ex.emax;
        const float core = (1.f + 2.f * gc) * (gc + (float)d * U23 * (1.f + rq) * (1.f + rx) + rq * (1.f + rx) + rx);
        const float M = 1.25f * (core + (1.f + rq) * (1.f + rx) * (FLT_EPSILON / (qn * ex.ntmin) + 8.f * U23)) + 1e-30f;
        slack = (qn > 0.f && ex.ntmin > 0.f) ? 2.f * M * qn : INFINITY;
    } else {
        const float X = ex.vmax, e = eq + ex.emax;
        const float s = qv + X;
        const float EA = (2.f * (float)d + 4.f) * U23 * s * s;   // |A~ - ||q~ - x~||^2|
        const float E2 = EA + 2.f * e * s + e * e;                 // |A~ - ||q - x||^2|
        if (metric == METRIC_L2SQR) slack = 1.25f * (E2 + gc * (s + e) * (s + e)) + 1e-30f;   // d~ = ||q~||^2 - 2u
        else slack = 2.f * (1.25f * (0.5f * E2 + 2.5f * gc * (qn + ex.ntmax)) + 1e-30f);       // d~ = ||q~||^2/2 - u
    }
    float t = -INFINITY;
    bool scan = !(slack < INFINITY);   // no usable margin (a NaN or infinite query, a zero norm): scan the query in full
    if (G >= K) {
        const float uk = u_val(v);
        t = __fsub_rd(uk, __fmul_ru(slack, 1.f + 1e-6f));
        scan = scan || !(fabsf(uk) < INFINITY);
    }
    thresh[qi] = scan ? INFINITY : t;
    if (scan) cand_n[(size_t)qi * nseg] = scap + 1;
}

// Orderable 64-bit key: (distance, id) ascending; -0 and +0 compare equal, as in the reference.
__device__ __forceinline__ unsigned long long dist_key(float d, uint32_t id) {
    uint32_t u = __float_as_uint(d == 0.f ? 0.f : d);
    u = (u & 0x80000000u) ? ~u : (u | 0x80000000u);
    return ((unsigned long long)u << 32) | id;
}
__device__ __forceinline__ float key_dist(unsigned long long k) {
    uint32_t u = (uint32_t)(k >> 32);
    u = (u & 0x80000000u) ? (u & 0x7FFFFFFFu) : ~u;
    return __uint_as_float(u);
}

// One warp per query: canonical FP32 distances of the candidates, then the K
// smallest by (distance, id) within epsilon.  A query whose candidates
// overflowed is noted in `again` (its row; the count in stats[2]) or, without
// one, scanned in full; one without a margin is scanned in full.  The queries'
// rows are map[0 .. nq) or, without a map, q0 .. q0 + nq - 1.
__global__ void __launch_bounds__(256) bf_recheck_kernel(DataView D, const float *Q, uint32_t q_ld, uint32_t q0,
                                                         const uint32_t *map, uint32_t nq, uint32_t K, float epsilon,
                                                         const float *thresh, uint32_t *again, const uint32_t *cand,
                                                         const uint32_t *cand_n, uint32_t nseg, uint32_t scap,
                                                         uint64_t mult, uint32_t cap, uint32_t *out_ids,
                                                         float *out_d, uint32_t *out_cnt, float *out_cost,
                                                         uint32_t out_ld, unsigned long long *stats,
                                                         unsigned long long *work) {
    extern __shared__ __align__(16) unsigned char rsm[];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t qi = blockIdx.x * (blockDim.x >> 5) + w;
    if (qi >= nq) return;   // whole warps
    const size_t row = map ? map[qi] : q0 + qi;
    float *q = reinterpret_cast<float *>(rsm) + (size_t)w * D.ld;
    unsigned long long *keys = reinterpret_cast<unsigned long long *>(rsm + (size_t)(blockDim.x >> 5) * D.ld * 4) +
                               (size_t)w * cap;
    for (uint32_t x = lane; x < D.ld; x += 32) q[x] = x < D.d ? Q[row * q_ld + x] : 0.f;
    __syncwarp();
    float qn = 0.f;
    if (D.metric != METRIC_L2SQR) qn = norm_term(group4_raw(q, q, D.d, METRIC_EUCLIDEAN, lane & 3, FULL), D.metric);
    // The candidates lie in nseg segments: gathered behind the room for their keys -- the ids of
    // candidate i at 4 cap + 4 i, its key later at 8 i, so that a pass of 8 writes no key over an id
    // not yet read.
    uint32_t *ids = reinterpret_cast<uint32_t *>(keys) + cap;
    uint32_t nc = 0;
    bool full = false;
    for (uint32_t s0 = 0; s0 < nseg && !full; s0 += 32) {
        const uint32_t k = s0 + lane < nseg ? cand_n[(size_t)qi * nseg + s0 + lane] : 0u;
        uint32_t end = k;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(FULL, end, o);
            if (lane >= o) end += v;
        }
        const uint32_t sum = __shfl_sync(FULL, end, 31);
        full = __any_sync(FULL, k > scap) || nc + sum > cap;
        if (full) break;
        const uint32_t *src = cand + ((size_t)qi * nseg + s0 + lane) * scap;
        for (uint32_t i = 0; i < k; ++i) ids[nc + end - k + i] = (uint32_t)(src[i] * mult % D.n);   // position p holds row p * mult mod n
        nc += sum;
    }
    if (full && again && thresh[qi] < INFINITY) {
        if (lane == 0) again[atomicAdd(stats + 2, 1ull)] = (uint32_t)row;
        return;
    }
    __syncwarp();
    const uint32_t total = full ? D.n : nc;
    const int g = lane >> 2, t = lane & 3;
    // the K smallest keys so far live in keys[0..have) when scanning in full; else all candidates' keys
    uint32_t nkeys = 0;
    unsigned long long worst = ~0ull;   // full scan: the K-th smallest key so far
    for (uint32_t base = 0; base < total; base += 8) {
        const uint32_t i = base + g;
        const uint32_t id = i < total ? (full ? i : ids[i]) : 0u;
        const float dd = query_dist(D, q, qn, id, t, FULL);
        const bool keep = i < total && t == 0 && !(dd > epsilon);
        const unsigned long long key = dist_key(dd, id);
        unsigned km = __ballot_sync(FULL, keep && (!full || key < worst));
        if (!full) {
            if (keep) keys[nkeys + __popc(km & ((1u << lane) - 1u))] = key;
            nkeys += __popc(km);
            __syncwarp();
            continue;
        }
        while (km) {
            const int src = __ffs(km) - 1;
            km &= km - 1;
            const unsigned long long kk = __shfl_sync(FULL, key, src);
            if (kk < worst) {   // keep the K smallest keys, unsorted; evict the largest
                if (nkeys < K) {
                    if (lane == 0) keys[nkeys] = kk;
                    ++nkeys;
                } else {
                    // replace the largest key
                    unsigned long long mx = 0;
                    uint32_t at = 0;
                    for (uint32_t j = lane; j < nkeys; j += 32)
                        if (keys[j] >= mx) { mx = keys[j]; at = j; }
                    for (int o = 16; o; o >>= 1) {
                        const unsigned long long om = __shfl_xor_sync(FULL, mx, o);
                        const uint32_t oa = __shfl_xor_sync(FULL, at, o);
                        if (om > mx || (om == mx && oa > at)) { mx = om; at = oa; }
                    }
                    __syncwarp();
                    if (lane == 0) keys[at] = kk;
                }
                __syncwarp();
                if (nkeys == K) {   // the new K-th smallest
                    unsigned long long mx = 0;
                    for (uint32_t j = lane; j < nkeys; j += 32) mx = max(mx, keys[j]);
                    for (int o = 16; o; o >>= 1) mx = max(mx, __shfl_xor_sync(FULL, mx, o));
                    worst = mx;
                }
            }
            __syncwarp();
        }
    }
    __syncwarp();
    // K rounds of the warp's smallest remaining key
    const uint32_t cnt = min(K, nkeys);
    uint32_t *oi = out_ids + row * out_ld;
    float *od = out_d ? out_d + row * out_ld : nullptr;
    for (uint32_t k = 0; k < cnt; ++k) {
        unsigned long long mn = ~0ull;
        uint32_t at = 0;
        for (uint32_t j = lane; j < nkeys; j += 32)
            if (keys[j] < mn) { mn = keys[j]; at = j; }
        for (int o = 16; o; o >>= 1) {
            const unsigned long long om = __shfl_xor_sync(FULL, mn, o);
            const uint32_t oa = __shfl_xor_sync(FULL, at, o);
            if (om < mn) { mn = om; at = oa; }
        }
        float dk = key_dist(mn);
        if (dk == 0.f) dk = query_dist(D, q, qn, (uint32_t)mn, t, FULL);   // the key does not hold a zero's sign
        if (lane == 0) {
            oi[k] = (uint32_t)(mn & 0xFFFFFFFFu);
            if (od) od[k] = dk;
            keys[at] = ~0ull;
        }
        __syncwarp();
    }
    if (lane == 0) {
        out_cnt[row] = cnt;
        if (out_cost) out_cost[row] = 1.0f;   // kgraph.cpp:428-431
        atomicAdd(stats + 0, (unsigned long long)(full ? 0u : nc));
        if (full) atomicAdd(stats + 1, 1ull);
        if (work) atomicAdd(work, (unsigned long long)total);
    }
}

}  // namespace

bool bruteforce_tc_supported(const kg_ctx *ctx, uint32_t K) {
    return K > 0 && K <= BF_MAX_K && ctx->ld <= 256;
}

// Rows of the dataset prepared for the sweeps (once per dataset version).
// First uncentred: a dataset whose values BF16 holds exactly (small integers,
// as in the benchmark's mixtures) keeps e_x = 0 and needs no centring.  Any
// other euclidean / l2sqr dataset is prepared again centred on its mean, which
// makes the BF16 error scale with the spread of the data instead of its offset.
// Data with a NaN or an infinity have no margin (bf_usable false: the scan).
int bruteforce_prepare(kg_ctx *ctx) {
    if (ctx->bf_data_version == ctx->data_version) return KG_OK;
    const uint32_t n = ctx->n, ld = ctx->ld;
    // the spread order: position p holds row p * mult mod n, mult coprime to n
    uint64_t mult = std::max<uint64_t>(1, (uint64_t)(0.6180339887 * n)), inv = 1;
    while (std::gcd(mult, (uint64_t)n) != 1) ++mult;
    {   // extended Euclid: inv * mult = 1 mod n
        int64_t r0 = n, r1 = (int64_t)mult, t0 = 0, t1 = 1;
        while (r1) {
            const int64_t k = r0 / r1;
            std::swap(r0, r1); r1 -= k * r0;
            std::swap(t0, t1); t1 -= k * t0;
        }
        inv = (uint64_t)(t0 < 0 ? t0 + n : t0);
    }
    cudaError_t e;
    if ((e = ctx->bf_rows.reserve((size_t)n * ld * 2)) != cudaSuccess ||
        (e = ctx->bf_meta.reserve(ctx->metric == METRIC_ANGULAR ? 0 : (size_t)n * 16)) != cudaSuccess ||
        (e = ctx->bf_aux.reserve((size_t)ld * 12 + 64 + 64)) != cudaSuccess)
        return cuda_fail(ctx, e, "alloc brute-force rows");
    cudaStream_t st = ctx->stream;
    double *sum = ctx->bf_aux.as<double>();
    float *mu = reinterpret_cast<float *>(sum + ld);
    unsigned long long *ext = reinterpret_cast<unsigned long long *>(mu + ld);
    const DataView D{ctx->X.as<float>(), ctx->norms.as<float>(), n, ctx->d, ld, ctx->metric};
    auto dec = [](unsigned long long o) {
        unsigned long long u = (o & 0x8000000000000000ull) ? (o & ~0x8000000000000000ull) : ~o;
        double v;
        std::memcpy(&v, &u, 8);
        return v;
    };
    unsigned long long h[4];
    for (int centre = 0; centre < 2; ++centre) {
        if (centre) {
            cudaMemsetAsync(sum, 0, ld * 8, st);
            dim3 grid((ctx->d + 127) / 128, std::min<uint32_t>(1024, (n + 255) / 256));
            colsum_kernel<<<grid, 128, 0, st>>>(D, sum);
        }
        mean_kernel<<<(ld + 127) / 128, 128, 0, st>>>(sum, ctx->d, ld, n, centre, mu);
        const unsigned long long init[4] = {0, 0, 0, ~0ull};
        cudaMemcpyAsync(ext, init, sizeof(init), cudaMemcpyHostToDevice, st);
        prep_rows_kernel<<<ctx->num_sms * 8, 256, 0, st>>>(D, mu, inv, ctx->bf_rows.as<__nv_bfloat16>(),
                                                           ctx->bf_meta.as<uint4>(), ext);
        if ((e = cudaGetLastError()) != cudaSuccess) return cuda_fail(ctx, e, "brute-force prep");
        cudaMemcpyAsync(h, ext, sizeof(h), cudaMemcpyDeviceToHost, st);
        if ((e = cudaStreamSynchronize(st)) != cudaSuccess) return cuda_fail(ctx, e, "brute-force prep");
        if (ctx->metric == METRIC_ANGULAR || dec(h[1]) == 0.0) break;   // uncentred: exact, or angular
    }
    // dataset maxima, rounded up (the minimum rounded down)
    ctx->bf_ext[0] = (float)(dec(h[0]) * (1 + 1e-6));
    ctx->bf_ext[1] = (float)(dec(h[1]) * (1 + 1e-6));
    ctx->bf_ext[2] = (float)(dec(h[2]) * (1 + 1e-6));
    ctx->bf_ext[3] = h[3] != ~0ull ? (float)(dec(h[3]) * (1 - 1e-6)) : 0.f;
    ctx->bf_mult = mult;
    ctx->bf_usable = ctx->bf_ext[0] < 1e18f && ctx->bf_ext[1] < 1e18f && ctx->bf_ext[2] < INFINITY;
    ctx->bf_data_version = ctx->data_version;
    return KG_OK;
}

// The sample sweep's rows and groups, the candidates a query has room for, and
// how many queries take one pass.  `all`: for queries that come a second time,
// all rows are the sample.
struct SweepPlan {
    uint32_t cap, ns, width;
    size_t batch;
    SweepPlan(uint32_t n, uint32_t K, bool all) : cap((all ? 2 : 1) * std::max<uint32_t>(1024, 8 * K)) {
        // A share of the rows that leaves about K / share candidates per query, at most half of `cap`;
        // groups of 32 rows where that makes at least 8 K of them, else smaller ones, so that few of the
        // K nearest sampled rows share a group.
        const uint32_t share = all ? 1 : K <= 2 ? 8 : K <= 24 ? 16 : K <= 64 ? 8 : 4;
        ns = n / share / BF_R * BF_R;
        if (ns < 4096 || share == 1) ns = n;
        width = ns / 32 >= 8 * K ? 32 : ns / 4 >= 8 * K ? 4 : 1;
        if (ns / 32 > BF_MAX_GROUPS32) width = 128;
        const size_t per = (size_t)(ns / width + BF_R) * 4 + (size_t)(all ? 24 : 8) * cap;
        batch = std::min(BF_BATCH, std::max<size_t>(BF_WORK_BYTES / per, 32));
        const size_t tile = batch >= 2 * BF_Q ? 2 * BF_Q : 32;   // whole tiles of queries where there are some
        batch = batch / tile * tile;
    }
};

// One pass over the rows for at most p.batch queries: rows q0 .. q0 + nq - 1, or map[0 .. nq).
static int bruteforce_batch(kg_ctx *ctx, const SweepPlan &p, const float *Q, uint32_t q_ld, uint32_t q0,
                            const uint32_t *map, uint32_t nq, uint32_t K, float epsilon, uint32_t *again,
                            uint32_t *out_ids, float *out_d, uint32_t *out_cnt, float *out_cost, uint32_t out_ld,
                            unsigned long long *stats, unsigned long long *work) {
    const uint32_t n = ctx->n, ld = ctx->ld;
    cudaStream_t st = ctx->stream;
    // Two M tiles per CTA where the queries fill them (else half the MMAs would multiply padding) and
    // the ring beside them holds more than one row tile (its boxes are released by the second product).
    const uint32_t nb = (ld + 63) / 64;
    const bool ext = ctx->metric != METRIC_ANGULAR;   // norm columns
    auto ring = [&](uint32_t subs) {   // boxes that fit, with enough norm-column tiles for them
        uint32_t k = BF_MAX_ST;
        auto bytes = [&] { return subs * nb * BF_QBOX + k * BF_RBOX + (ext ? (k + nb - 1) / nb * BF_REXT + BF_QEXT : 0u); };
        while (k > 1 && bytes() > BF_SMEM - 1024) --k;
        return k;
    };
    const uint32_t nsub = nq > BF_Q && ring(2) > nb ? 2 : 1;
    const uint32_t qt = (nq + nsub * BF_Q - 1) / (nsub * BF_Q), rt = (n + BF_R - 1) / BF_R;
    const uint32_t chunks = (uint32_t)(((size_t)n * ld * 2 + BF_CHUNK_BYTES - 1) / BF_CHUNK_BYTES);
    const uint32_t rtc = (rt + chunks - 1) / chunks;
    const uint32_t cap = p.cap, ns = p.ns, width = p.width;
    const uint32_t srt = (ns + BF_R - 1) / BF_R, groups = (ns + width - 1) / width;
    const uint32_t fold = (groups + BF_GROUPS - 1) / BF_GROUPS, G = (groups + fold - 1) / fold;
    const uint32_t nqp = (nq + 31) / 32 * 32;
    const uint32_t grid1 = (uint32_t)std::min<uint64_t>(ctx->num_sms, (uint64_t)qt * rtc);
    const uint32_t grid0 = (uint32_t)std::min<uint64_t>(ctx->num_sms, (uint64_t)qt * srt);
    // segments of candidates: two (column halves) per CTA that meets a query tile, each with room for
    // twice its even share (the spread order deals the candidates out evenly); the queries that come a
    // second time get twice the share of the CTA that meets most of their tile
    uint32_t nseg = 1;
    for (uint32_t q = 0; q < qt; ++q) {
        const uint32_t b0 = sweep_first_cta(q, qt, rtc, grid1);
        const uint64_t T = (uint64_t)qt * rtc, end = (uint64_t)(q + 1) * rtc;
        uint32_t b1 = b0;
        while (b1 + 1 < grid1 && T * (b1 + 1) / grid1 < end) ++b1;
        nseg = std::max(nseg, b1 - b0 + 1);
    }
    nseg *= 2;
    uint32_t even = 2 * cap / nseg;
    if (!again) even = (uint32_t)std::min<uint64_t>(cap, (uint64_t)cap * ((uint64_t)qt * rtc / grid1 + 1) / rtc);
    const uint32_t scap = std::min<uint32_t>(cap, std::max<uint32_t>(128, even));
    cudaError_t e;
    auto pad = [](size_t b) { return (b + 255) / 256 * 256; };
    const size_t need = pad((size_t)nq * ld * 2) + pad((size_t)nq * 16) + pad((size_t)srt * (BF_R / width) * nqp * 4) +
                        pad((size_t)nq * 4) + pad((size_t)nq * nseg * scap * 4) + pad((size_t)nq * nseg * 4);
    if ((e = ctx->bf_work.reserve(need)) != cudaSuccess) return cuda_fail(ctx, e, "alloc brute force");
    char *at = ctx->bf_work.as<char>();
    auto carve = [&](size_t bytes) { char *q = at; at += pad(bytes); return q; };
    __nv_bfloat16 *Qb = reinterpret_cast<__nv_bfloat16 *>(carve((size_t)nq * ld * 2));
    float4 *qmeta = reinterpret_cast<float4 *>(carve((size_t)nq * 16));
    float *gmax = reinterpret_cast<float *>(carve((size_t)srt * (BF_R / width) * nqp * 4));
    float *thresh = reinterpret_cast<float *>(carve((size_t)nq * 4));
    uint32_t *cand = reinterpret_cast<uint32_t *>(carve((size_t)nq * nseg * scap * 4));
    uint32_t *cand_n = reinterpret_cast<uint32_t *>(carve((size_t)nq * nseg * 4));
    cudaMemsetAsync(cand_n, 0, (size_t)nq * nseg * 4, st);
    const DataView D{ctx->X.as<float>(), ctx->norms.as<float>(), n, ctx->d, ld, ctx->metric};
    const float *mu = reinterpret_cast<const float *>(ctx->bf_aux.as<double>() + ld);
    prep_queries_kernel<<<std::max<uint32_t>(1, std::min<uint32_t>((nq + 7) / 8, ctx->num_sms * 8)), 256, 0, st>>>(
        D, mu, map ? Q : Q + (size_t)q0 * q_ld, q_ld, map, nq, Qb, qmeta);
    CUtensorMap mQ, mX, mE;
    if (!tc_bf16_map(&mQ, Qb, ld, nq, ld, 64, BF_Q) || !tc_bf16_map(&mX, ctx->bf_rows.p, ld, n, ld, 64, BF_R))
        return set_error(ctx, KG_E_CUDA, "brute force: tensor map");
    mE = mX;
    // (rows of 8 in memory, 16 in the box: TMA fills the rest with zeros)
    if (ext && !tc_bf16_map(&mE, ctx->bf_meta.p, 8, n, 8, 16, BF_R, CU_TENSOR_MAP_SWIZZLE_32B))
        return set_error(ctx, KG_E_CUDA, "brute force: tensor map");
    SweepArgs a{};
    a.ld = ld; a.nq = nq; a.nsub = nsub;
    a.stages = ring(nsub);
    a.estages = ext ? (a.stages + nb - 1) / nb : 0u;
    a.qt = qt;
    a.gmax = gmax; a.nqp = nqp; a.width = width;
    a.thresh = thresh;
    a.cand = cand; a.cand_n = cand_n; a.nseg = nseg; a.scap = scap;
    a.err = ctx->errw.as<uint32_t>();
    const size_t tsmem = (size_t)8 * G * 4;
    if ((e = cudaFuncSetAttribute(bf_sweep_kernel<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)BF_SMEM)) !=
            cudaSuccess ||
        (e = cudaFuncSetAttribute(bf_sweep_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)BF_SMEM)) !=
            cudaSuccess ||
        (e = cudaFuncSetAttribute(bf_threshold_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)(8 * BF_GROUPS * 4))) != cudaSuccess)
        return cuda_fail(ctx, e, "brute-force sweep attributes");
    a.n = ns; a.rt = srt; a.rtc = srt;
    bf_sweep_kernel<0><<<grid0, BF_THREADS, BF_SMEM, st>>>(mQ, mX, mE, a);
    const Extents ex{ctx->bf_ext[0], ctx->bf_ext[1], ctx->bf_ext[2], ctx->bf_ext[3]};
    bf_threshold_kernel<<<(nq + 7) / 8, 256, tsmem, st>>>(gmax, nqp, groups, fold, qmeta, nq, K, ctx->d, ctx->metric, ex,
                                                          thresh, cand_n, nseg, scap);
    a.n = n; a.rt = rt; a.rtc = rtc;
    bf_sweep_kernel<1><<<grid1, BF_THREADS, BF_SMEM, st>>>(mQ, mX, mE, a);
    const uint32_t wpb = 4;
    const size_t rsmem = (size_t)wpb * (ld * 4 + (size_t)cap * 8);
    if ((e = cudaFuncSetAttribute(bf_recheck_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)rsmem)) !=
        cudaSuccess)
        return cuda_fail(ctx, e, "brute-force recheck attributes");
    bf_recheck_kernel<<<(nq + wpb - 1) / wpb, wpb * 32, rsmem, st>>>(D, Q, q_ld, q0, map, nq, K, epsilon, thresh, again,
                                                                     cand, cand_n, nseg, scap, ctx->bf_mult, cap, out_ids,
                                                                     out_d, out_cnt, out_cost, out_ld, stats, work);
    if ((e = cudaGetLastError()) != cudaSuccess) return cuda_fail(ctx, e, "brute-force launch");
    return KG_OK;
}

int bruteforce_tc(kg_ctx *ctx, const float *Q, uint32_t q_ld, uint32_t nq, uint32_t K, float epsilon, uint32_t *out_ids,
                  float *out_d, uint32_t *out_cnt, float *out_cost, uint32_t out_ld, unsigned long long *work) {
    cudaError_t e;
    if ((e = ctx->bf_again.reserve((size_t)nq * 4)) != cudaSuccess) return cuda_fail(ctx, e, "alloc brute force");
    // candidates rechecked, queries scanned in full, queries to come again (read by the caller after its
    // sync); behind the mean
    unsigned long long *stats = reinterpret_cast<unsigned long long *>(ctx->bf_aux.as<char>() + (size_t)ctx->ld * 12 + 64);
    cudaMemsetAsync(stats, 0, 24, ctx->stream);
    ctx->bf_stats_dev = stats;
    const SweepPlan p(ctx->n, K, false);
    for (size_t q0 = 0; q0 < nq; q0 += p.batch) {
        const int r = bruteforce_batch(ctx, p, Q, q_ld, (uint32_t)q0, nullptr, (uint32_t)std::min<size_t>(p.batch, nq - q0),
                                       K, epsilon, ctx->bf_again.as<uint32_t>(), out_ids, out_d, out_cnt, out_cost,
                                       out_ld, stats, work);
        if (r != KG_OK) return r;
    }
    return KG_OK;
}

int bruteforce_again(kg_ctx *ctx, const float *Q, uint32_t q_ld, uint32_t count, uint32_t K, float epsilon,
                     uint32_t *out_ids, float *out_d, uint32_t *out_cnt, float *out_cost, uint32_t out_ld,
                     unsigned long long *work) {
    const SweepPlan p(ctx->n, K, true);
    for (size_t i = 0; i < count; i += p.batch) {
        const int r = bruteforce_batch(ctx, p, Q, q_ld, 0, ctx->bf_again.as<uint32_t>() + i,
                                       (uint32_t)std::min<size_t>(p.batch, count - i), K, epsilon, nullptr, out_ids,
                                       out_d, out_cnt, out_cost, out_ld, ctx->bf_stats_dev, work);
        if (r != KG_OK) return r;
    }
    return KG_OK;
}

}  // namespace kgb
