// gx_cluster_scan.cuh -- an exclusive scan in one launch, by one cluster of blocks.
//
// The plan and the tree build scan dozens of arrays of a few thousand to a few hundred
// thousand entries, between kernels that make the entries and kernels that spread them out
// again.  As sums, scan of the sums and a second pass that was three launches of 3 us each
// around 2 us of work.  Here the blocks of a cluster sum a contiguous share each, exchange
// the sums through distributed shared memory at a cluster barrier, and scan their shares;
// the caller's load and store functions make the entries and use their offsets in the same
// pass.  Beyond CS_MAX_N entries the three launches over the whole GPU are faster: at 331k one
// cluster takes 27 us, and the plan of 2,000,000 leaves spent 3.6 of its 44 ms in scans by one
// cluster.  cs_scan takes the one form or the other.
#pragma once
#include <cooperative_groups.h>

#include "gx_internal.cuh"

constexpr int CS_THREADS = 1024;
constexpr int CS_ITEMS = 4;
constexpr int CS_MAX_BLOCKS = 16;
constexpr int64_t CS_MAX_N = (int64_t)1 << 17;

// K running totals scanned together
template <int K>
struct CsVec {
    int64_t v[K];
};

template <int K>
__device__ __forceinline__ CsVec<K> cs_shfl_up_add(CsVec<K> a, int o) {
    const bool take = (int)(threadIdx.x & 31) >= o;
#pragma unroll
    for (int k = 0; k < K; k++) {
        const int64_t u = __shfl_up_sync(0xffffffffu, a.v[k], o);
        if (take) a.v[k] += u;
    }
    return a;
}

// Exclusive prefix of a over the block; total: the block's sum, to every thread.  sh: 33
// values, free again when the call returns.
template <int K>
__device__ __forceinline__ CsVec<K> cs_block_scan(const CsVec<K> a, CsVec<K> *sh, CsVec<K> &total) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    CsVec<K> inc = a;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) inc = cs_shfl_up_add<K>(inc, o);
    if (lane == 31) sh[w] = inc;
    __syncthreads();
    if (w == 0) {
        CsVec<K> x = sh[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) x = cs_shfl_up_add<K>(x, o);
        sh[lane] = x;
    }
    __syncthreads();
    total = sh[31];
#pragma unroll
    for (int k = 0; k < K; k++) inc.v[k] += (w > 0 ? sh[w - 1].v[k] : 0) - a.v[k];
    __syncthreads();
    return inc;
}

// All threads of a cluster of CS_THREADS-thread blocks call it: store(i, prefix, value) for
// every i < n with value = load(i) (a CsVec<K>; called twice for an entry) and prefix the sum
// of those before it, by the thread that stores.  Returns the sum over all entries.  Ends
// with a cluster barrier: what store wrote is visible to the cluster.
template <int K, class Load, class Store>
__device__ CsVec<K> cluster_scan(int64_t n, const Load &load, const Store &store) {
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    __shared__ CsVec<K> sh[33], mine;
    const int nb = (int)cl.num_blocks(), rank = (int)cl.block_rank(), t = threadIdx.x;
    const int64_t share = max((int64_t)CS_THREADS, (n + nb - 1) / nb);
    const int64_t s0 = min(n, rank * share), s1 = min(n, s0 + share);
    CsVec<K> sum{};
    for (int64_t i = s0 + t; i < s1; i += CS_THREADS) {
        const CsVec<K> x = load(i);
#pragma unroll
        for (int k = 0; k < K; k++) sum.v[k] += x.v[k];
    }
    CsVec<K> total;
    cs_block_scan<K>(sum, sh, total);
    if (t == 0) mine = total;
    cl.sync();
    CsVec<K> run{}, all{};
    for (int r = 0; r < nb; r++) {
        const CsVec<K> x = *cl.map_shared_rank(&mine, r);
#pragma unroll
        for (int k = 0; k < K; k++) {
            if (r < rank) run.v[k] += x.v[k];
            all.v[k] += x.v[k];
        }
    }
    for (int64_t base = s0; base < s1; base += CS_THREADS * CS_ITEMS) {
        CsVec<K> v[CS_ITEMS], s{};
#pragma unroll
        for (int q = 0; q < CS_ITEMS; q++) {
            const int64_t i = base + (int64_t)t * CS_ITEMS + q;
            v[q] = i < s1 ? load(i) : CsVec<K>{};
#pragma unroll
            for (int k = 0; k < K; k++) s.v[k] += v[q].v[k];
        }
        CsVec<K> p = cs_block_scan<K>(s, sh, total);
#pragma unroll
        for (int k = 0; k < K; k++) p.v[k] += run.v[k];
#pragma unroll
        for (int q = 0; q < CS_ITEMS; q++) {
            const int64_t i = base + (int64_t)t * CS_ITEMS + q;
            if (i < s1) store(i, p, v[q]);
#pragma unroll
            for (int k = 0; k < K; k++) p.v[k] += v[q].v[k];
        }
#pragma unroll
        for (int k = 0; k < K; k++) run.v[k] += total.v[k];
    }
    cl.sync();
    return all;
}

// Launches kernel as one cluster for about n entries (one block for a few thousand, else 16
// where the device takes them, else the portable 8).
template <class... Params, class... Args>
int cs_launch(gx_ctx *ctx, int64_t n, void (*kernel)(Params...), Args... args) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at = {};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.blockDim = dim3(CS_THREADS);
    cfg.stream = ctx->stream;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    unsigned blocks = n <= CS_THREADS * CS_ITEMS ? 1 : 8;
    if (blocks > 1) {
        int fit = 0;
        at.val.clusterDim.x = CS_MAX_BLOCKS;
        cfg.gridDim = dim3(CS_MAX_BLOCKS);
        if (ctx->cluster16 == 0) {
            ctx->cluster16 = -1;
            if (cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
                cudaOccupancyMaxActiveClusters(&fit, kernel, &cfg) == cudaSuccess && fit > 0)
                ctx->cluster16 = 1;
            cudaGetLastError();  // a device without the larger cluster is no error
        }
        if (ctx->cluster16 > 0 &&
            cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess)
            blocks = CS_MAX_BLOCKS;
    }
    at.val.clusterDim.x = blocks;
    cfg.gridDim = dim3(blocks);
    GX_CUDA(ctx, cudaLaunchKernelEx(&cfg, kernel, Params(args)...));
    ctx->launches++;
    return GX_OK;
}

// ---- one scan in either form ----
// F describes it: off() (true: nothing is to be done), count() entries, load(i), store(i,
// prefix, value) as above, and total(sum of all), called by one thread.
template <int K, class F>
__global__ void __launch_bounds__(CS_THREADS) k_scan_one_cluster(F f) {
    if (f.off()) return;
    const CsVec<K> all = cluster_scan<K>(
        f.count(), [&](int64_t i) { return f.load(i); },
        [&](int64_t i, const CsVec<K> &p, const CsVec<K> &v) { f.store(i, p, v); });
    if (blockIdx.x == 0 && threadIdx.x == 0) f.total(all);
}

constexpr int64_t CS_TILE = CS_THREADS * CS_ITEMS;

template <int K, class F>
__global__ void __launch_bounds__(CS_THREADS) k_scan_tile_sums(F f, CsVec<K> *sums) {
    __shared__ CsVec<K> sh[33];
    if (f.off()) return;
    const int64_t n = f.count(), base = blockIdx.x * CS_TILE;
    if (base >= n) return;
    CsVec<K> sum{}, total;
    for (int q = 0; q < CS_ITEMS; q++) {
        const int64_t i = base + q * CS_THREADS + threadIdx.x;
        if (i >= n) break;
        const CsVec<K> x = f.load(i);
#pragma unroll
        for (int k = 0; k < K; k++) sum.v[k] += x.v[k];
    }
    cs_block_scan<K>(sum, sh, total);
    if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

template <int K, class F>
__global__ void __launch_bounds__(CS_THREADS) k_scan_tile_tops(F f, CsVec<K> *sums) {
    __shared__ CsVec<K> sh[33];
    if (f.off()) return;
    const int64_t nb = (f.count() + CS_TILE - 1) / CS_TILE;
    CsVec<K> run{}, total;
    for (int64_t base = 0; base < nb; base += CS_THREADS) {
        const int64_t i = base + threadIdx.x;
        CsVec<K> p = cs_block_scan<K>(i < nb ? sums[i] : CsVec<K>{}, sh, total);
#pragma unroll
        for (int k = 0; k < K; k++) {
            p.v[k] += run.v[k];
            run.v[k] += total.v[k];
        }
        if (i < nb) sums[i] = p;
    }
    __syncthreads();  // off() has been read: total may change it
    if (threadIdx.x == 0) f.total(run);
}

template <int K, class F>
__global__ void __launch_bounds__(CS_THREADS) k_scan_tile_stores(F f, const CsVec<K> *sums) {
    __shared__ CsVec<K> sh[33];
    if (f.off()) return;
    const int64_t n = f.count(), base = blockIdx.x * CS_TILE + (int64_t)threadIdx.x * CS_ITEMS;
    if (blockIdx.x * CS_TILE >= n) return;
    CsVec<K> v[CS_ITEMS], s{}, total;
#pragma unroll
    for (int q = 0; q < CS_ITEMS; q++) {
        v[q] = base + q < n ? f.load(base + q) : CsVec<K>{};
#pragma unroll
        for (int k = 0; k < K; k++) s.v[k] += v[q].v[k];
    }
    CsVec<K> p = cs_block_scan<K>(s, sh, total);
    const CsVec<K> before = sums[blockIdx.x];
#pragma unroll
    for (int k = 0; k < K; k++) p.v[k] += before.v[k];
#pragma unroll
    for (int q = 0; q < CS_ITEMS; q++) {
        if (base + q < n) f.store(base + q, p, v[q]);
#pragma unroll
        for (int k = 0; k < K; k++) p.v[k] += v[q].v[k];
    }
}

// About n entries, n_cap at most.
template <int K, class F>
int cs_scan(gx_ctx *ctx, int64_t n, int64_t n_cap, const F &f) {
    if (n <= CS_MAX_N) return cs_launch(ctx, n, k_scan_one_cluster<K, F>, f);
    const int64_t nb = (n_cap + CS_TILE - 1) / CS_TILE;
    GX_TRY(gx_ensure(ctx, ctx->scratch_g, sizeof(CsVec<K>) * (size_t)nb));
    CsVec<K> *sums = dptr<CsVec<K>>(ctx->scratch_g);
    k_scan_tile_sums<K, F><<<(unsigned)nb, CS_THREADS, 0, ctx->stream>>>(f, sums);
    k_scan_tile_tops<K, F><<<1, CS_THREADS, 0, ctx->stream>>>(f, sums);
    k_scan_tile_stores<K, F><<<(unsigned)nb, CS_THREADS, 0, ctx->stream>>>(f, sums);
    ctx->launches += 3;
    GX_CUDA(ctx, cudaGetLastError());
    return GX_OK;
}
