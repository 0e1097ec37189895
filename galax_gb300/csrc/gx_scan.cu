// gx_scan.cu -- device-wide exclusive scan and a stable LSD radix sort.
//
// Up to 131,072 entries a scan is one launch (gx_cluster_scan.cuh), above that
// reduce-then-scan in three.  The radix sort replaces the stable `indices.sort_by_key(|&i| keys[i])` of
// Tree::build (galax-core/src/lib.rs:192).  It is a three-kernel
// reduce-then-scan design: no kernel waits on another CTA, so there is no
// inter-block spin anywhere.  Stability: within a tile each warp owns a
// contiguous run of 256 items and ranks them in index order with
// __match_any_sync; warps and tiles are ordered by the digit-major offset scan.
#include "gx_cluster_scan.cuh"
#include "gx_internal.cuh"

namespace {

constexpr int SCAN_THREADS = 256;
constexpr int SCAN_ITEMS = 4;
constexpr int SCAN_TILE = SCAN_THREADS * SCAN_ITEMS;  // 1024

template <class T>
__device__ T block_exclusive_scan(T v, T *total) {
    __shared__ T warp_tot[SCAN_THREADS / 32];
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    T inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        T t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
    }
    if (lane == 31) warp_tot[w] = inc;
    __syncthreads();
    if (w == 0) {
        T s = (lane < SCAN_THREADS / 32) ? warp_tot[lane] : T(0);
        T si = s;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            T t = __shfl_up_sync(0xffffffffu, si, o);
            if (lane >= o) si += t;
        }
        if (lane < SCAN_THREADS / 32) warp_tot[lane] = si - s;
        if (lane == SCAN_THREADS / 32 - 1) *total = si;
    }
    __syncthreads();
    T r = warp_tot[w] + inc - v;
    __syncthreads();
    return r;
}

template <class T>
__global__ void k_scan_sums(const T *in, int64_t n, T *sums) {
    __shared__ T tot;
    int64_t base = (int64_t)blockIdx.x * SCAN_TILE;
    T s = 0;
    for (int k = 0; k < SCAN_ITEMS; k++) {
        int64_t i = base + (int64_t)threadIdx.x * SCAN_ITEMS + k;
        if (i < n) s += in[i];
    }
    block_exclusive_scan<T>(s, &tot);
    if (threadIdx.x == 0) sums[blockIdx.x] = tot;
}

// In-place exclusive scan of `sums` (nb entries) by one block; writes the grand total.
template <class T>
__device__ void scan_single_block(T *sums, int64_t nb, T *total) {
    __shared__ T tot;
    T carry = 0;
    for (int64_t base = 0; base < nb; base += SCAN_TILE) {
        T v[SCAN_ITEMS];
        T s = 0;
        for (int k = 0; k < SCAN_ITEMS; k++) {
            int64_t i = base + (int64_t)threadIdx.x * SCAN_ITEMS + k;
            v[k] = (i < nb) ? sums[i] : T(0);
            s += v[k];
        }
        T ex = block_exclusive_scan<T>(s, &tot);
        T run = carry + ex;
        for (int k = 0; k < SCAN_ITEMS; k++) {
            int64_t i = base + (int64_t)threadIdx.x * SCAN_ITEMS + k;
            if (i < nb) sums[i] = run;
            run += v[k];
        }
        carry += tot;
        __syncthreads();
    }
    if (threadIdx.x == 0 && total) *total = carry;
}

template <class T>
__global__ void k_scan_single(T *sums, int64_t nb, T *total) {
    scan_single_block<T>(sums, nb, total);
}

template <class T>
__global__ void k_scan_apply(const T *in, T *out, int64_t n, const T *sums) {
    __shared__ T tot;
    int64_t base = (int64_t)blockIdx.x * SCAN_TILE;
    T v[SCAN_ITEMS];
    T s = 0;
    for (int k = 0; k < SCAN_ITEMS; k++) {
        int64_t i = base + (int64_t)threadIdx.x * SCAN_ITEMS + k;
        v[k] = (i < n) ? in[i] : T(0);
        s += v[k];
    }
    T run = sums[blockIdx.x] + block_exclusive_scan<T>(s, &tot);
    for (int k = 0; k < SCAN_ITEMS; k++) {
        int64_t i = base + (int64_t)threadIdx.x * SCAN_ITEMS + k;
        if (i < n) out[i] = run;
        run += v[k];
    }
}

// Device-length forms: the length is *n_dev + n_add (at most n_cap), read on the
// device, so a scan over a count produced by an earlier kernel needs no host round
// trip.  Grids are sized for n_cap; blocks past the length do no work.
__device__ __forceinline__ int64_t dev_len(const int64_t *n_dev, int64_t n_add, int64_t n_cap) {
    int64_t n = *n_dev + n_add;
    return n < n_cap ? n : n_cap;
}

__global__ void k_scan_sums_dn(const int64_t *in, const int64_t *n_dev, int64_t n_add, int64_t n_cap,
                               int64_t *sums) {
    __shared__ int64_t tot;
    const int64_t n = dev_len(n_dev, n_add, n_cap);
    int64_t base = (int64_t)blockIdx.x * SCAN_TILE;
    int64_t s = 0;
    if (base < n)
        for (int k = 0; k < SCAN_ITEMS; k++) {
            int64_t i = base + (int64_t)threadIdx.x * SCAN_ITEMS + k;
            if (i < n) s += in[i];
        }
    block_exclusive_scan<int64_t>(s, &tot);
    if (threadIdx.x == 0) sums[blockIdx.x] = tot;
}

__global__ void k_scan_apply_dn(const int64_t *in, int64_t *out, const int64_t *n_dev, int64_t n_add, int64_t n_cap,
                                const int64_t *sums) {
    __shared__ int64_t tot;
    const int64_t n = dev_len(n_dev, n_add, n_cap);
    int64_t base = (int64_t)blockIdx.x * SCAN_TILE;
    if (base >= n) return;  // uniform per block
    int64_t v[SCAN_ITEMS];
    int64_t s = 0;
    for (int k = 0; k < SCAN_ITEMS; k++) {
        int64_t i = base + (int64_t)threadIdx.x * SCAN_ITEMS + k;
        v[k] = (i < n) ? in[i] : 0;
        s += v[k];
    }
    int64_t run = sums[blockIdx.x] + block_exclusive_scan<int64_t>(s, &tot);
    for (int k = 0; k < SCAN_ITEMS; k++) {
        int64_t i = base + (int64_t)threadIdx.x * SCAN_ITEMS + k;
        if (i < n) out[i] = run;
        run += v[k];
    }
}

// one array of n entries, or of min(*n_dev + n_add, n)
template <class T>
__global__ void __launch_bounds__(CS_THREADS) k_scan_cluster(const T *in, T *out, int64_t n, const int64_t *n_dev,
                                                             int64_t n_add, T *total) {
    const int64_t len = n_dev ? dev_len(n_dev, n_add, n) : n;
    const CsVec<1> all = cluster_scan<1>(
        len, [&](int64_t i) { return CsVec<1>{{(int64_t)in[i]}}; },
        [&](int64_t i, const CsVec<1> &p, const CsVec<1> &) { out[i] = (T)p.v[0]; });
    if (total && blockIdx.x == 0 && threadIdx.x == 0) *total = (T)all.v[0];
}

template <class T>
int scan_impl(gx_ctx *ctx, const T *in, T *out, int64_t n, T *total_host) {
    if (n <= 0) {
        if (total_host) *total_host = 0;
        return GX_OK;
    }
    int64_t nb = (n + SCAN_TILE - 1) / SCAN_TILE;
    GX_TRY(gx_ensure(ctx, ctx->scratch_g, sizeof(T) * (nb + 1)));
    T *sums = dptr<T>(ctx->scratch_g);
    if (n <= CS_MAX_N) {
        GX_TRY(cs_launch(ctx, n, k_scan_cluster<T>, in, out, n, nullptr, 0, sums + nb));
        if (total_host) {
            GX_CUDA(ctx, cudaMemcpyAsync(total_host, sums + nb, sizeof(T), cudaMemcpyDeviceToHost, ctx->stream));
            GX_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
        }
        return GX_OK;
    }
    k_scan_sums<T><<<(unsigned)nb, SCAN_THREADS, 0, ctx->stream>>>(in, n, sums);
    k_scan_single<T><<<1, SCAN_THREADS, 0, ctx->stream>>>(sums, nb, sums + nb);
    k_scan_apply<T><<<(unsigned)nb, SCAN_THREADS, 0, ctx->stream>>>(in, out, n, sums);
    ctx->launches += 3;
    GX_CUDA(ctx, cudaGetLastError());
    if (total_host) {
        GX_CUDA(ctx, cudaMemcpyAsync(total_host, sums + nb, sizeof(T), cudaMemcpyDeviceToHost, ctx->stream));
        GX_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    }
    return GX_OK;
}

// ------------------------------------------------------------------ radix sort
constexpr int RS_WARPS = 8;
constexpr int RS_ROUNDS = 8;
constexpr int RS_WARP_ITEMS = 32 * RS_ROUNDS;          // 256
constexpr int RS_TILE = RS_WARPS * RS_WARP_ITEMS;      // 2048
constexpr int RS_BINS = 256;

// digit counts of a tile, digit-major: hist[d * nb + tile]
__global__ void k_rs_hist(const uint64_t *__restrict__ keys, int64_t n, int shift, int bins, unsigned *hist,
                          int64_t nb) {
    __shared__ unsigned h[RS_BINS];
    for (int i = threadIdx.x; i < bins; i += blockDim.x) h[i] = 0;
    __syncthreads();
    const int64_t base = (int64_t)blockIdx.x * RS_TILE;
    uint64_t k[RS_TILE / 256];
#pragma unroll
    for (int r = 0; r < RS_TILE / 256; r++) {
        const int64_t i = base + r * 256 + threadIdx.x;
        k[r] = i < n ? keys[i] : 0;
    }
#pragma unroll
    for (int r = 0; r < RS_TILE / 256; r++)
        if (base + r * 256 + threadIdx.x < n) atomicAdd(&h[(unsigned)(k[r] >> shift) & (unsigned)(bins - 1)], 1u);
    __syncthreads();
    for (int d = threadIdx.x; d < bins; d += blockDim.x) hist[(int64_t)d * nb + blockIdx.x] = h[d];
}

// One block per digit: its tiles' counts become their exclusive scan, tot[d] the digit's
// count.  The scan over the digits themselves (256 values) is left to the scatter's blocks,
// so a pass is three launches and no scan of the whole count matrix.
__global__ void __launch_bounds__(SCAN_THREADS) k_rs_rows(unsigned *hist, int64_t nb, unsigned *tot) {
    scan_single_block<unsigned>(hist + blockIdx.x * nb, nb, tot + blockIdx.x);
}

__global__ void __launch_bounds__(RS_WARPS * 32) k_rs_scatter(const uint64_t *__restrict__ kin,
                                                             const uint32_t *__restrict__ vin, uint64_t *kout,
                                                             uint32_t *vout, int64_t n, int shift, int bins,
                                                             const unsigned *__restrict__ offs, int64_t nb,
                                                             const unsigned *__restrict__ tot) {
    static_assert(RS_WARPS * 32 == RS_BINS && RS_BINS == SCAN_THREADS, "a thread per digit");
    const unsigned mask = (unsigned)(bins - 1);
    __shared__ unsigned first[RS_BINS], sum;  // where this tile's items of a digit begin
    const unsigned mine = (int)threadIdx.x < bins ? tot[threadIdx.x] : 0u;
    const unsigned before = block_exclusive_scan<unsigned>(mine, &sum);
    if ((int)threadIdx.x < bins) first[threadIdx.x] = before + offs[(int64_t)threadIdx.x * nb + blockIdx.x];
    if (__syncthreads_or(mine == (unsigned)n)) {  // every key has the same digit: the stable order is the present one
        for (int64_t i = (int64_t)blockIdx.x * RS_TILE + threadIdx.x; i < n && i < (int64_t)(blockIdx.x + 1) * RS_TILE;
             i += blockDim.x) {
            kout[i] = kin[i];
            vout[i] = vin[i];
        }
        return;
    }
    __shared__ unsigned cnt[RS_WARPS][RS_BINS];
    for (int i = threadIdx.x; i < RS_WARPS * RS_BINS; i += blockDim.x) (&cnt[0][0])[i] = 0u;
    __syncthreads();
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    unsigned lt = (1u << lane) - 1u;
    int64_t base = (int64_t)blockIdx.x * RS_TILE + (int64_t)w * RS_WARP_ITEMS;
    uint64_t k[RS_ROUNDS];
    uint32_t v[RS_ROUNDS];
    unsigned d[RS_ROUNDS], rk[RS_ROUNDS];
#pragma unroll
    for (int r = 0; r < RS_ROUNDS; r++) {
        int64_t i = base + r * 32 + lane;
        bool ok = i < n;
        k[r] = ok ? kin[i] : 0ull;
        v[r] = ok ? vin[i] : 0u;
        d[r] = ok ? ((unsigned)(k[r] >> shift) & mask) : 0xFFFFFFFFu;
        unsigned peers = __match_any_sync(0xffffffffu, d[r]);
        int leader = __ffs(peers) - 1;
        unsigned c = ok ? cnt[w][d[r]] : 0u;
        __syncwarp();
        if (ok && lane == leader) cnt[w][d[r]] = c + __popc(peers);
        __syncwarp();
        rk[r] = c + __popc(peers & lt);
    }
    __syncthreads();
    for (int dd = threadIdx.x; dd < bins; dd += blockDim.x) {
        unsigned run = first[dd];
        for (int ww = 0; ww < RS_WARPS; ww++) {
            unsigned t = cnt[ww][dd];
            cnt[ww][dd] = run;
            run += t;
        }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < RS_ROUNDS; r++) {
        if (d[r] == 0xFFFFFFFFu) continue;
        const unsigned pos = cnt[w][d[r]] + rk[r];
        kout[pos] = k[r];
        vout[pos] = v[r];
    }
}

}  // namespace

int gx_exclusive_scan_i64(gx_ctx *ctx, const int64_t *in, int64_t *out, int64_t n) {
    return scan_impl<int64_t>(ctx, in, out, n, nullptr);
}

int gx_exclusive_scan_i64_devn(gx_ctx *ctx, const int64_t *in, int64_t *out, const int64_t *n_dev, int64_t n_add,
                               int64_t n_cap, int64_t *total_dev) {
    if (n_cap <= 0) return GX_OK;
    if (n_cap <= CS_MAX_N) return cs_launch(ctx, n_cap, k_scan_cluster<int64_t>, in, out, n_cap, n_dev, n_add, total_dev);
    int64_t nb = (n_cap + SCAN_TILE - 1) / SCAN_TILE;
    GX_TRY(gx_ensure(ctx, ctx->scratch_g, sizeof(int64_t) * (size_t)(nb + 1)));
    int64_t *sums = dptr<int64_t>(ctx->scratch_g);
    k_scan_sums_dn<<<(unsigned)nb, SCAN_THREADS, 0, ctx->stream>>>(in, n_dev, n_add, n_cap, sums);
    k_scan_single<int64_t><<<1, SCAN_THREADS, 0, ctx->stream>>>(sums, nb, total_dev ? total_dev : sums + nb);
    k_scan_apply_dn<<<(unsigned)nb, SCAN_THREADS, 0, ctx->stream>>>(in, out, n_dev, n_add, n_cap, sums);
    ctx->launches += 3;
    GX_CUDA(ctx, cudaGetLastError());
    return GX_OK;
}

int gx_exclusive_scan_i32(gx_ctx *ctx, const int32_t *in, int32_t *out, int64_t n, int32_t *total_host) {
    return scan_impl<int32_t>(ctx, in, out, n, total_host);
}

// Stable sort of (keys, vals) by key bits [begin_bit, end_bit).  Ping-pongs with the
// *_alt buffers; *result_in_alt tells where the sorted data ended up.
int gx_radix_sort_u64(gx_ctx *ctx, uint64_t *keys, uint32_t *vals, int64_t n, int begin_bit, int end_bit,
                      uint64_t *keys_alt, uint32_t *vals_alt, bool *result_in_alt) {
    *result_in_alt = false;
    if (n <= 1) return GX_OK;
    int64_t nb = (n + RS_TILE - 1) / RS_TILE;
    if (nb * RS_BINS > 0x7fffffffLL) return gx_fail(ctx, GX_ERR_CAP_EXCEEDED, "radix sort: too many items");
    GX_TRY(gx_ensure(ctx, ctx->scratch_e, sizeof(unsigned) * (size_t)(nb * RS_BINS + 1)));
    GX_TRY(gx_ensure(ctx, ctx->scratch_f, sizeof(unsigned) * RS_BINS));
    unsigned *hist = dptr<unsigned>(ctx->scratch_e);
    unsigned *tot = dptr<unsigned>(ctx->scratch_f);
    uint64_t *ki = keys, *ko = keys_alt;
    uint32_t *vi = vals, *vo = vals_alt;
    // passes of at most 8 bits, as even as the key allows (42 bits: six of 7, whose runs in
    // the scatter are twice as long as those of 8)
    const int passes = (end_bit - begin_bit + 7) / 8;
    for (int q = 0, shift = begin_bit; q < passes; q++) {
        const int bits = (end_bit - shift + passes - q - 1) / (passes - q), bins = 1 << bits;
        k_rs_hist<<<(unsigned)nb, 256, 0, ctx->stream>>>(ki, n, shift, bins, hist, nb);
        k_rs_rows<<<(unsigned)bins, SCAN_THREADS, 0, ctx->stream>>>(hist, nb, tot);
        k_rs_scatter<<<(unsigned)nb, RS_WARPS * 32, 0, ctx->stream>>>(ki, vi, ko, vo, n, shift, bins, hist, nb, tot);
        ctx->launches += 3;
        GX_CUDA(ctx, cudaGetLastError());
        shift += bits;
        uint64_t *tk = ki; ki = ko; ko = tk;
        uint32_t *tv = vi; vi = vo; vo = tv;
    }
    *result_in_alt = (ki == keys_alt);
    return GX_OK;
}
