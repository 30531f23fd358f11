// Graph post-processing on the GPU: reverse-edge completion
// (KGraphImpl::reverse, kgraph.cpp:667-702) and pruning (kgraph.cpp:584-665).
//
// reverse.  The reference appends, for every node i in increasing order and
// every kept forward edge j, the edge to ng[i] and its reverse to ng[e.id],
// then std::sort's each list by distance and drops ADJACENT duplicate ids.
// std::sort is not stable, so the final order of equal distances -- and which
// duplicates end up adjacent -- depends on the list's push order and on the
// GNU introsort.  Here the push order is rebuilt exactly (reverse edges,
// source and distance, grouped by target with a stable radix sort of (target)
// over edges numbered in (i, j) order, the node's own forward edges spliced in
// at i == x), and each list is sorted by the same introsort (kg_sort.h), one
// warp per node.  The result is the reference's graph bit for bit.
#include <cub/cub.cuh>
#include <iostream>
#include <vector>
#include "kg_ctx.h"
#include "kg_sort.h"

namespace kgb {

cudaError_t scan_counts64(kg_ctx *ctx, const uint64_t *in, uint64_t *out, uint32_t n);

namespace {

__global__ void rev_count_kernel(uint32_t N, const uint64_t *off, const uint32_t *M, int rev_k, uint64_t *kcnt) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < N; i += gridDim.x * blockDim.x) {
        uint32_t deg = (uint32_t)(off[i + 1] - off[i]);
        uint32_t k = rev_k > 0 ? min((uint32_t)rev_k, deg) : min(M[i], deg);
        kcnt[i] = k;
    }
}

// One entry per kept forward edge, in (i, j) order: its target, and its source and distance.
__global__ void rev_edges_kernel(uint32_t N, const uint64_t *off, const uint32_t *nbr, const float *nbr_d,
                                 const uint64_t *koff, uint32_t *key, unsigned long long *val, uint32_t *err) {
    const int lane = threadIdx.x & 31;
    const uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t i = w; i < N; i += nw) {
        const uint64_t b = koff[i], o = off[i];
        const uint32_t k = (uint32_t)(koff[i + 1] - b);
        for (uint32_t j = lane; j < k; j += 32) {
            uint32_t t = nbr[o + j];
            if (t >= N) { atomicOr(err, 4u); t = i; }
            key[b + j] = t;
            val[b + j] = (unsigned long long)__float_as_uint(nbr_d[o + j]) << 32 | i;
        }
    }
}

// toff[t]: the first sorted edge whose target is t or above; toff[N] = E.
__global__ void rev_offsets_kernel(uint32_t N, uint64_t E, const uint32_t *skey, uint64_t *toff) {
    for (uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; e <= E; e += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t hi = e < E ? skey[e] : N;
        for (uint32_t t = e ? skey[e - 1] + 1 : 0u; t <= hi; ++t) toff[t] = e;
    }
}

// Rebuilds node x's list in the reference's push order, sorts it with the
// GNU introsort, removes adjacent duplicate ids; writes its final length.  The
// list has room at koff[x] + toff[x] of the output (every forward edge and every
// reverse edge before it); it is sorted in shared memory up to REV_CAP entries,
// in place beyond.  Bound: the sort's dependent steps, one warp per list.  1M
// nodes x 40 edges, the whole call: 29.4 ms with one thread per list sorting in
// global memory and searching each reverse edge's source; 10.1 ms now (both
// with the import and export of the graph).
constexpr uint32_t REV_CAP = 480;
constexpr int REV_WARPS = 8;
__global__ void __launch_bounds__(REV_WARPS * 32) rev_assemble_kernel(uint32_t N, const uint64_t *off, const uint32_t *nbr,
                                                                      const float *nbr_d, const uint64_t *koff,
                                                                      const uint64_t *toff,
                                                                      const unsigned long long *sval, uint32_t *out_i,
                                                                      float *out_d, uint64_t *fdeg) {
    __shared__ float s_d[REV_WARPS][REV_CAP];
    __shared__ uint32_t s_i[REV_WARPS][REV_CAP], s_tmp[REV_WARPS][WARP_SORT_TMP];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const unsigned ALL = 0xFFFFFFFFu, below = (1u << lane) - 1u;
    const uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t x = w; x < N; x += nw) {
        const uint64_t k0 = koff[x], q0 = toff[x], o0 = off[x];
        const uint32_t kx = (uint32_t)(koff[x + 1] - k0), rx = (uint32_t)(toff[x + 1] - q0), p = kx + rx;
        uint32_t *gi = out_i + k0 + q0;
        float *gd = out_d + k0 + q0;
        const bool in_smem = p <= REV_CAP;
        uint32_t *li = in_smem ? s_i[wib] : gi;
        float *ld = in_smem ? s_d[wib] : gd;
        // reverse edges from sources below x, then (behind the node's own) from sources above it
        uint32_t nb = 0;
        bool nan = false;   // among the distances this lane stored
        for (uint32_t b = 0; b < rx; b += 32) {
            const uint32_t j = b + lane;
            const unsigned long long v = j < rx ? sval[q0 + j] : 0ull;
            const uint32_t src = (uint32_t)v;
            if (j < rx && src != x) {
                const uint32_t at = src < x ? j : j + kx;
                const float dd = __uint_as_float((uint32_t)(v >> 32));
                li[at] = src;
                ld[at] = dd;
                nan |= dd != dd;
            }
            nb += __popc(__ballot_sync(ALL, j < rx && src < x));
        }
        // own forward edges; a self loop's reverse edge follows its forward edge
        uint32_t ns = 0;
        for (uint32_t b = 0; b < kx; b += 32) {
            const uint32_t j = b + lane;
            const uint32_t id = j < kx ? nbr[o0 + j] : 0u;
            const unsigned self = __ballot_sync(ALL, j < kx && (id == x || id >= N));   // an id out of range was keyed to x
            if (j < kx) {
                const uint32_t at = nb + j + ns + __popc(self & below);
                const float dd = nbr_d[o0 + j];
                li[at] = id;
                ld[at] = dd;
                nan |= dd != dd;
                if ((self >> lane) & 1u) { li[at + 1] = x; ld[at + 1] = dd; }
            }
            ns += __popc(self);
        }
        __syncwarp();
        if (p <= (uint32_t)WARP_SORT_MAX) {
            warp_gnu_sort(ld, li, nullptr, (int)p, s_tmp[wib], nan, lane);   // kgraph.cpp:697
        } else {
            if (lane == 0) { WarpSortAcc acc{ld, li, nullptr}; gnu_sort(acc, 0, (int)p); }
            __syncwarp();
        }
        uint32_t m = 0;   // std::unique by id (kgraph.cpp:698): entries equal to the one before go
        uint32_t last = 0;
        for (uint32_t b = 0; b < p; b += 32) {
            const uint32_t r = b + lane;
            const uint32_t id = r < p ? li[r] : 0u;
            const float dd = r < p ? ld[r] : 0.f;
            uint32_t prev = __shfl_up_sync(ALL, id, 1);
            if (lane == 0) prev = last;
            last = __shfl_sync(ALL, id, 31);
            const bool keep = r < p && (r == 0 || id != prev);
            const unsigned km = __ballot_sync(ALL, keep);
            if (keep) {   // at or before r, and every lane has read its entry
                const uint32_t at = m + __popc(km & below);
                gi[at] = id;
                gd[at] = dd;
            }
            m += __popc(km);
        }
        if (lane == 0) fdeg[x] = m;
        __syncwarp();
    }
}

// Like koff, the lists' places in the assembled graph: room for every edge.
__global__ void rev_places_kernel(uint32_t N, const uint64_t *koff, const uint64_t *toff, uint64_t *noff) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i <= N; i += gridDim.x * blockDim.x) noff[i] = koff[i] + toff[i];
}

__global__ void compact_kernel(uint32_t N, const uint64_t *src_off, const uint64_t *dst_off, const uint32_t *si,
                               const float *sd, uint32_t *di, float *dd, uint32_t *M, int set_M) {
    const int lane = threadIdx.x & 31;
    const uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t x = w; x < N; x += nw) {
        const uint64_t a = src_off[x], b = dst_off[x];
        const uint32_t c = (uint32_t)(dst_off[x + 1] - b);
        for (uint32_t r = lane; r < c; r += 32) {
            di[b + r] = si[a + r];
            if (sd) dd[b + r] = sd[a + r];
        }
        if (set_M && lane == 0) M[x] = c;
    }
}

__global__ void prune1_count_kernel(uint32_t N, const uint64_t *off, const uint32_t *M, uint64_t *cnt) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < N; i += gridDim.x * blockDim.x) {
        uint32_t deg = (uint32_t)(off[i + 1] - off[i]);
        cnt[i] = deg > M[i] ? M[i] : deg;
    }
}

}  // namespace

// Installs (off, ids, dists) of n nodes as the context's graph, taking ownership
// of the three scratch buffers by swapping them in.
static void swap_graph(kg_ctx *ctx, DevBuf &off, DevBuf &ids, DevBuf &dists) {
    std::swap(ctx->offsets, off);
    std::swap(ctx->nbr, ids);
    std::swap(ctx->nbr_d, dists);
}

int graph_reverse(kg_ctx *ctx, int rev_k) {
    if (rev_k == 0) return KG_OK;
    if (!ctx->has_graph) return set_error(ctx, KG_E_RUNTIME, "no index");
    if (ctx->no_dist) return set_error(ctx, KG_E_RUNTIME, "Need distance information to reverse graph");
    std::cerr << "Graph completion with reverse edges..." << std::endl;
    const uint32_t N = ctx->gn;
    const size_t n = N;
    cudaStream_t st = ctx->stream;
    cudaError_t e;
    // Work space kept in the context between calls: a build reverses once per call, and freeing and
    // re-allocating ~2 GB (1M nodes) each time costs device-synchronising cudaFree / cudaMalloc calls whose
    // time varied from build to build.  Buffers grow with 1/8 slack.
    DevBuf *R = ctx->rev_scratch;
    DevBuf &kcnt = R[0], &koff = R[1], &toff = R[2], &noff = R[3], &fdeg = R[4], &foff = R[5], &key = R[6], &val = R[7],
           &skey = R[8], &sval = R[9], &tmp = R[10], &ad = R[11], &fi = R[12], &fd = R[13];
    auto grow = [](DevBuf &b, size_t bytes) { return b.reserve(bytes <= b.bytes ? bytes : bytes + bytes / 8); };
    auto fail = [&](const char *w) { return cuda_fail(ctx, e, w); };
    if ((e = grow(kcnt, (n + 1) * 8)) != cudaSuccess || (e = grow(koff, (n + 1) * 8)) != cudaSuccess ||
        (e = grow(toff, (n + 1) * 8)) != cudaSuccess || (e = grow(noff, (n + 1) * 8)) != cudaSuccess ||
        (e = grow(fdeg, (n + 1) * 8)) != cudaSuccess || (e = grow(foff, (n + 1) * 8)) != cudaSuccess)
        return fail("alloc reverse");
    cudaMemsetAsync(kcnt.as<uint64_t>() + n, 0, 8, st);   // the scans take one extra zero
    cudaMemsetAsync(fdeg.as<uint64_t>() + n, 0, 8, st);
    const int grid = ctx->num_sms * 4;
    rev_count_kernel<<<grid, 256, 0, st>>>(N, ctx->offsets.as<uint64_t>(), ctx->Mnode.as<uint32_t>(), rev_k,
                                           kcnt.as<uint64_t>());
    if ((e = scan_counts64(ctx, kcnt.as<uint64_t>(), koff.as<uint64_t>(), N)) != cudaSuccess) return fail("scan");
    uint64_t Ef = 0;
    cudaMemcpyAsync(&Ef, koff.as<uint64_t>() + N, 8, cudaMemcpyDeviceToHost, st);
    cudaStreamSynchronize(st);
    if (Ef >= 0xFFFFFFFFull) { e = cudaErrorInvalidValue; return fail("graph too large to reverse"); }
    if ((e = grow(key, Ef * 4 + 4)) != cudaSuccess || (e = grow(val, Ef * 8 + 8)) != cudaSuccess ||
        (e = grow(skey, Ef * 4 + 4)) != cudaSuccess || (e = grow(sval, Ef * 8 + 8)) != cudaSuccess)
        return fail("alloc reverse");
    rev_edges_kernel<<<grid * 2, 256, 0, st>>>(N, ctx->offsets.as<uint64_t>(), ctx->nbr.as<uint32_t>(),
                                               ctx->nbr_d.as<float>(), koff.as<uint64_t>(), key.as<uint32_t>(),
                                               val.as<unsigned long long>(), ctx->errw.as<uint32_t>());
    // stable radix sort by target keeps the (i, j) order within each target
    int end_bit = 1;
    while (end_bit < 32 && (1ull << end_bit) < n) ++end_bit;
    size_t tb = 0;
    cub::DoubleBuffer<uint32_t> keys(key.as<uint32_t>(), skey.as<uint32_t>());
    cub::DoubleBuffer<unsigned long long> vals(val.as<unsigned long long>(), sval.as<unsigned long long>());
    cub::DeviceRadixSort::SortPairs(nullptr, tb, keys, vals, (int64_t)Ef, 0, end_bit, st);
    if ((e = grow(tmp, tb)) != cudaSuccess) return fail("alloc sort");
    if ((e = cub::DeviceRadixSort::SortPairs(tmp.p, tb, keys, vals, (int64_t)Ef, 0, end_bit, st)) != cudaSuccess)
        return fail("sort");
    rev_offsets_kernel<<<grid * 2, 256, 0, st>>>(N, Ef, keys.Current(), toff.as<uint64_t>());
    rev_places_kernel<<<grid, 256, 0, st>>>(N, koff.as<uint64_t>(), toff.as<uint64_t>(), noff.as<uint64_t>());
    const uint64_t E2 = 2 * Ef;
    if ((e = grow(ad, E2 * 4 + 4)) != cudaSuccess) return fail("alloc reverse");
    uint32_t *ai = reinterpret_cast<uint32_t *>(vals.Alternate());   // the assembled ids: room for 2 Ef of them
    std::cerr << "Reranking edges..." << std::endl;
    rev_assemble_kernel<<<ctx->num_sms * 6, REV_WARPS * 32, 0, st>>>(
        N, ctx->offsets.as<uint64_t>(), ctx->nbr.as<uint32_t>(), ctx->nbr_d.as<float>(), koff.as<uint64_t>(),
        toff.as<uint64_t>(), vals.Current(), ai, ad.as<float>(), fdeg.as<uint64_t>());
    if ((e = cudaGetLastError()) != cudaSuccess) return fail("reverse");
    if ((e = scan_counts64(ctx, fdeg.as<uint64_t>(), foff.as<uint64_t>(), N)) != cudaSuccess) return fail("scan");
    uint64_t Efin = 0;
    cudaMemcpyAsync(&Efin, foff.as<uint64_t>() + N, 8, cudaMemcpyDeviceToHost, st);
    cudaStreamSynchronize(st);
    if ((e = grow(fi, Efin * 4 + 4)) != cudaSuccess || (e = grow(fd, Efin * 4 + 4)) != cudaSuccess)
        return fail("alloc reverse");
    compact_kernel<<<grid * 2, 256, 0, st>>>(N, noff.as<uint64_t>(), foff.as<uint64_t>(), ai, ad.as<float>(),
                                             fi.as<uint32_t>(), fd.as<float>(),
                                             ctx->Mnode.as<uint32_t>(), 1);
    if ((e = cudaGetLastError()) != cudaSuccess) return fail("reverse");
    if ((e = cudaStreamSynchronize(st)) != cudaSuccess) return fail("reverse");
    swap_graph(ctx, foff, fi, fd);
    ctx->E = Efin;
    ++ctx->graph_version;
    return check_device_error(ctx, "reverse");
}

// prune1 (kgraph.cpp:584-590) on the GPU.
static int prune1(kg_ctx *ctx) {
    const uint32_t N = ctx->gn;
    const size_t n = N;
    cudaStream_t st = ctx->stream;
    cudaError_t e;
    DevBuf cnt, noff, ni, nd;
    if ((e = cnt.reserve((n + 1) * 8)) != cudaSuccess || (e = noff.reserve((n + 1) * 8)) != cudaSuccess)
        return cuda_fail(ctx, e, "alloc prune");
    cudaMemsetAsync(cnt.p, 0, (n + 1) * 8, st);
    prune1_count_kernel<<<ctx->num_sms * 4, 256, 0, st>>>(N, ctx->offsets.as<uint64_t>(), ctx->Mnode.as<uint32_t>(),
                                                           cnt.as<uint64_t>());
    if ((e = scan_counts64(ctx, cnt.as<uint64_t>(), noff.as<uint64_t>(), N)) != cudaSuccess) return cuda_fail(ctx, e, "scan");
    uint64_t E = 0;
    cudaMemcpyAsync(&E, noff.as<uint64_t>() + N, 8, cudaMemcpyDeviceToHost, st);
    cudaStreamSynchronize(st);
    if ((e = ni.reserve(E * 4 + 4)) != cudaSuccess || (e = nd.reserve(E * 4 + 4)) != cudaSuccess)
        return cuda_fail(ctx, e, "alloc prune");
    compact_kernel<<<ctx->num_sms * 8, 256, 0, st>>>(N, ctx->offsets.as<uint64_t>(), noff.as<uint64_t>(),
                                                     ctx->nbr.as<uint32_t>(), ctx->no_dist ? nullptr : ctx->nbr_d.as<float>(),
                                                     ni.as<uint32_t>(), nd.as<float>(), nullptr, 0);
    if ((e = cudaStreamSynchronize(st)) != cudaSuccess) return cuda_fail(ctx, e, "prune");
    swap_graph(ctx, noff, ni, nd);
    ctx->E = E;
    ++ctx->graph_version;
    return KG_OK;
}

// prune2 (kgraph.cpp:593-656): a sequential level-by-level pass whose every
// step reads the edits of the steps before it (reverse lists and flags of
// other nodes), so it runs on the host, in the reference's order, on the
// graph copied out of HBM; the result goes back to HBM.  It is maintenance
// of a finished index, not part of build or search.
static int prune2(kg_ctx *ctx) {
    const uint32_t N = ctx->gn;
    std::vector<uint64_t> off(N + 1);
    std::vector<uint32_t> ids(ctx->E), M(N);
    std::vector<float> ds(ctx->no_dist ? 0 : ctx->E);
    cudaMemcpy(off.data(), ctx->offsets.p, (N + 1) * 8, cudaMemcpyDeviceToHost);
    cudaMemcpy(ids.data(), ctx->nbr.p, ctx->E * 4, cudaMemcpyDeviceToHost);
    if (!ctx->no_dist) cudaMemcpy(ds.data(), ctx->nbr_d.p, ctx->E * 4, cudaMemcpyDeviceToHost);
    cudaMemcpy(M.data(), ctx->Mnode.p, N * 4, cudaMemcpyDeviceToHost);
    std::vector<uint8_t> flag(ctx->E, 0);
    std::vector<std::vector<uint32_t>> rev(N);
    std::vector<uint32_t> newL(N, 0), todo(N), next;
    for (uint32_t i = 0; i < N; ++i) todo[i] = i;
    auto at = [&](uint32_t node, uint32_t k) { return off[node] + k; };
    for (uint32_t l = 0; !todo.empty(); ++l) {
        next.clear();
        for (uint32_t i : todo) {
            if (l >= M[i]) continue;
            next.push_back(i);
            if (l >= off[i + 1] - off[i]) return set_error(ctx, KG_E_RUNTIME, "M larger than the list");
            if (flag[at(i, l)]) continue;
            flag[at(i, l)] = 1;
            uint32_t T;
            {
                uint32_t &nl = newL[i];
                T = ids[at(i, nl)] = ids[at(i, l)];
                if (!ds.empty()) ds[at(i, nl)] = ds[at(i, l)];
                ++nl;
            }
            rev[T].push_back(i);
            for (uint32_t ll = l + 1; ll < M[i]; ++ll) {
                if (flag[at(i, ll)]) continue;
                for (uint32_t j = 0; j < newL[T]; ++j)
                    if (ids[at(i, ll)] == ids[at(T, j)]) { flag[at(i, ll)] = 1; break; }
            }
            for (uint32_t r : rev[i])
                for (uint32_t ll = l; ll < M[r]; ++ll)
                    if (ids[at(r, ll)] == T) flag[at(r, ll)] = 1;
        }
        todo.swap(next);
    }
    cudaMemcpy(ctx->nbr.p, ids.data(), ctx->E * 4, cudaMemcpyHostToDevice);
    if (!ctx->no_dist) cudaMemcpy(ctx->nbr_d.p, ds.data(), ctx->E * 4, cudaMemcpyHostToDevice);
    cudaMemcpy(ctx->Mnode.p, newL.data(), N * 4, cudaMemcpyHostToDevice);
    ++ctx->graph_version;
    return prune1(ctx);
}

int graph_prune(kg_ctx *ctx, unsigned level) {
    if (!ctx->has_graph) return set_error(ctx, KG_E_RUNTIME, "no index");
    if (level & 1) {
        int r = prune1(ctx);
        if (r != KG_OK) return r;
    }
    if (level & 2) {
        int r = prune2(ctx);
        if (r != KG_OK) return r;
    }
    return KG_OK;
}

}  // namespace kgb

extern "C" int kg_reverse(kg_ctx *ctx, int rev_k) {
    if (!ctx) return KG_E_INVALID;
    std::lock_guard<std::mutex> g(ctx->mu);
    cudaSetDevice(ctx->device);
    return kgb::graph_reverse(ctx, rev_k);
}

extern "C" int kg_prune(kg_ctx *ctx, unsigned level) {
    if (!ctx) return KG_E_INVALID;
    std::lock_guard<std::mutex> g(ctx->mu);
    cudaSetDevice(ctx->device);
    return kgb::graph_prune(ctx, level);
}
