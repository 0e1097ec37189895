// gx_kdk.cu -- device-resident leapfrog, diagnostics and the sampled exact sum.
//
//  * leapfrog_kdk (galax-integrate/src/lib.rs:158-189): kick dt/2, drift dt,
//    force (static tree), kick dt/2 -- FP64 state, separately rounded mul/add;
//  * diagnostics (galax-core/src/lib.rs:1638-1683): KE, FMM PE, momentum, Lz as
//    deterministic two-stage block reductions (fixed grid, fixed tree order);
//  * validate_fmm's exact sum (lib.rs:1537-1553) for sampled targets.
#include <cooperative_groups.h>

#include <mutex>

#include "gx_internal.cuh"
#include "gx_mass_r3.cuh"

namespace {

constexpr int RED_THREADS = 256;
constexpr int RED_BLOCKS = 304;  // 2 x 152 SMs

__global__ void k_kick_drift(int64_t n, double h, double dt, double *x, double *y, double *vx, double *vy,
                             const double *ax, const double *ay) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double u = __dadd_rn(vx[i], __dmul_rn(ax[i], h));
    double v = __dadd_rn(vy[i], __dmul_rn(ay[i], h));
    vx[i] = u;
    vy[i] = v;
    x[i] = __dadd_rn(x[i], __dmul_rn(u, dt));
    y[i] = __dadd_rn(y[i], __dmul_rn(v, dt));
}

__global__ void k_kick(int64_t n, double h, double *vx, double *vy, const double *ax, const double *ay) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    vx[i] = __dadd_rn(vx[i], __dmul_rn(ax[i], h));
    vy[i] = __dadd_rn(vy[i], __dmul_rn(ay[i], h));
}

// k_kick of one step and k_kick_drift of the next: the same operations in the same order, the
// velocities and accelerations read once
__global__ void k_kick_kick_drift(int64_t n, double h, double dt, double *x, double *y, double *vx, double *vy,
                                  const double *ax, const double *ay) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double kx = __dmul_rn(ax[i], h), ky = __dmul_rn(ay[i], h);
    const double u = __dadd_rn(__dadd_rn(vx[i], kx), kx);
    const double v = __dadd_rn(__dadd_rn(vy[i], ky), ky);
    vx[i] = u;
    vy[i] = v;
    x[i] = __dadd_rn(x[i], __dmul_rn(u, dt));
    y[i] = __dadd_rn(y[i], __dmul_rn(v, dt));
}

__device__ __forceinline__ double block_sum(double v, double *sh) {
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) sh[w] = v;
    __syncthreads();
    double r = 0.0;
    if (threadIdx.x == 0)
        for (int k = 0; k < (int)(blockDim.x >> 5); k++) r += sh[k];
    __syncthreads();
    return r;
}

// per block: {KE, PE, px, py, Lz} over a grid-stride range
__global__ void k_diag_partial(int64_t n, const double *x, const double *y, const double *vx, const double *vy,
                               const double *m, const double *ax, const double *ay, double *part) {
    __shared__ double sh[RED_THREADS / 32];
    double ke = 0, pe = 0, px = 0, py = 0, lz = 0;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        double mi = m[i], u = vx[i], v = vy[i], xi = x[i], yi = y[i];
        double v2 = __dadd_rn(__dmul_rn(u, u), __dmul_rn(v, v));
        ke += __dmul_rn(__dmul_rn(0.5, mi), v2);
        double am = sqrt(__dadd_rn(__dmul_rn(ax[i], ax[i]), __dmul_rn(ay[i], ay[i])));
        double r = fmax(sqrt(__dadd_rn(__dmul_rn(xi, xi), __dmul_rn(yi, yi))), 1.0);
        pe += __dmul_rn(__dmul_rn(mi, am), r);
        px += __dmul_rn(mi, u);
        py += __dmul_rn(mi, v);
        lz += __dmul_rn(mi, __dsub_rn(__dmul_rn(xi, v), __dmul_rn(yi, u)));
    }
    double s[5] = {ke, pe, px, py, lz};
    for (int k = 0; k < 5; k++) {
        double t = block_sum(s[k], sh);
        if (threadIdx.x == 0) part[k * gridDim.x + blockIdx.x] = t;
    }
}

__global__ void k_diag_final(const double *part, int nb, double *out) {
    __shared__ double sh[RED_THREADS / 32];
    for (int k = 0; k < 5; k++) {
        double v = 0.0;
        for (int b = threadIdx.x; b < nb; b += blockDim.x) v += part[k * nb + b];
        double t = block_sum(v, sh);
        if (threadIdx.x == 0) out[k] = (k == 1) ? -0.5 * t : t;
    }
}

// One cluster of blocks per sampled target, the bodies dealt out over its threads; the
// blocks' sums are added in rank order through distributed shared memory, so the result
// does not depend on scheduling and no scratch is needed.  Bound by the FP64 pipe: m r^-3
// comes from the integer pipes (gx_mass_r3), which leaves six FP64 instructions a pair.
__global__ void __launch_bounds__(RED_THREADS) k_n2_sampled(int64_t n, const double *__restrict__ x,
                                                            const double *__restrict__ y,
                                                            const double *__restrict__ m, double eps2,
                                                            const int64_t *__restrict__ idx, double *ax, double *ay) {
    namespace cg = cooperative_groups;
    __shared__ double sh[RED_THREADS / 32];
    __shared__ double2 tot;
    cg::cluster_group cl = cg::this_cluster();
    const unsigned nb = cl.num_blocks(), rank = cl.block_rank();
    const int64_t s = blockIdx.x / nb, i = idx[s];
    const double xi = x[i], yi = y[i];
    double fx = 0.0, fy = 0.0;
#pragma unroll 2
    for (int64_t j = (int64_t)rank * blockDim.x + threadIdx.x; j < n; j += (int64_t)nb * blockDim.x) {
        const double mj = m[j], dx = x[j] - xi, dy = y[j] - yi;
        const double f = gx_mass_r3(fma(dx, dx, fma(dy, dy, eps2)), gx_mass_split(mj), mj);
        if (j != i) {  // the target itself adds nothing, not even where dx = x - x is NaN
            fx = fma(f, dx, fx);
            fy = fma(f, dy, fy);
        }
    }
    const double tx = block_sum(fx, sh);
    const double ty = block_sum(fy, sh);
    if (threadIdx.x == 0) tot = make_double2(tx, ty);
    cl.sync();
    if (rank == 0 && threadIdx.x == 0) {
        double sx = 0.0, sy = 0.0;
        for (unsigned b = 0; b < nb; b++) {
            const double2 v = *cl.map_shared_rank(&tot, b);
            sx += v.x;
            sy += v.y;
        }
        ax[s] = sx;
        ay[s] = sy;
    }
    cl.sync();  // the other blocks' sums stay in place until rank 0 has read them
}

// Blocks of a cluster: enough to fill the GPU (eight blocks an SM) when the samples alone do not.
cudaError_t launch_n2(int64_t n, const double *x, const double *y, const double *m, double eps2, const int64_t *idx,
                      int64_t n_idx, double *ax, double *ay, int sms, cudaStream_t st) {
    unsigned c = 1;
    while (c < 8 && n_idx * c < (int64_t)sms * 8 && (int64_t)c * RED_THREADS < n) c *= 2;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)n_idx * c);
    cfg.blockDim = dim3(RED_THREADS);
    cfg.stream = st;
    cudaLaunchAttribute at = {};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = c;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k_n2_sampled, n, x, y, m, eps2, idx, ax, ay);
}

}  // namespace

int gx_diag_device(gx_ctx *ctx, double out[5]) {
    GX_TRY(gx_ensure(ctx, ctx->red, sizeof(double) * (5 * RED_BLOCKS + 8)));
    double *part = dptr<double>(ctx->red), *res = part + 5 * RED_BLOCKS;
    int64_t n = ctx->n_bodies;
    k_diag_partial<<<RED_BLOCKS, RED_THREADS, 0, ctx->stream>>>(n, dptr<double>(ctx->x), dptr<double>(ctx->y),
                                                                dptr<double>(ctx->vx), dptr<double>(ctx->vy),
                                                                dptr<double>(ctx->m), dptr<double>(ctx->ax),
                                                                dptr<double>(ctx->ay), part);
    k_diag_final<<<1, RED_THREADS, 0, ctx->stream>>>(part, RED_BLOCKS, res);
    ctx->launches += 2;
    GX_CUDA(ctx, cudaGetLastError());
    GX_CUDA(ctx, cudaMemcpyAsync(out, res, sizeof(double) * 5, cudaMemcpyDeviceToHost, ctx->stream));
    GX_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    return GX_OK;
}

int gx_kdk_device(gx_ctx *ctx, int64_t n_steps, double dt, int64_t energy_every, double *diag, int64_t *n_diag,
                  int64_t rebuild_every) {
    int64_t n = ctx->n_bodies, nd = 0;
    double h = 0.5 * dt;
    bool kicked = true;  // the last step's second half kick is done
    for (int64_t step = 0; step < n_steps; step++) {
        (kicked ? k_kick_drift : k_kick_kick_drift)<<<gx_blocks(n, 256), 256, 0, ctx->stream>>>(
            n, h, dt, dptr<double>(ctx->x), dptr<double>(ctx->y), dptr<double>(ctx->vx), dptr<double>(ctx->vy),
            dptr<double>(ctx->ax), dptr<double>(ctx->ay));
        ctx->launches++;
        if (rebuild_every > 0 && (step + 1) % rebuild_every == 0) {
            // the tree of the drifted positions (the bodies, ids and accelerations are permuted with it)
            GX_TRY(gx_rebuild_internal(ctx));
            GX_TRY(gx_ensure_plan_public(ctx));
        }
        GX_TRY(gx_forces_device(ctx, false));
        // left to the next step's first kernel unless the velocities are looked at before
        kicked = step + 1 == n_steps || (energy_every > 0 && (step + 1) % energy_every == 0);
        if (kicked) {
            k_kick<<<gx_blocks(n, 256), 256, 0, ctx->stream>>>(n, h, dptr<double>(ctx->vx), dptr<double>(ctx->vy),
                                                               dptr<double>(ctx->ax), dptr<double>(ctx->ay));
            ctx->launches++;
        }
        GX_CUDA(ctx, cudaGetLastError());
        if (energy_every > 0 && (step + 1) % energy_every == 0) {
            double d[5];
            GX_TRY(gx_diag_device(ctx, d));
            if (diag) {
                double *row = diag + 6 * nd;
                row[0] = (double)(step + 1);
                row[1] = d[0];
                row[2] = d[1];
                row[3] = d[2];
                row[4] = d[3];
                row[5] = d[4];
            }
            nd++;
        }
    }
    GX_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    if (n_diag) *n_diag = nd;
    return GX_OK;
}

int gx_n2_device(gx_ctx *ctx, const int64_t *idx, int64_t n_idx, double *ax, double *ay) {
    if (n_idx <= 0) return GX_OK;
    GX_TRY(gx_ensure(ctx, ctx->scratch_a, sizeof(int64_t) * (size_t)n_idx + sizeof(double) * 2 * (size_t)n_idx));
    int64_t *didx = dptr<int64_t>(ctx->scratch_a);
    double *dax = reinterpret_cast<double *>(didx + n_idx), *day = dax + n_idx;
    for (int64_t k = 0; k < n_idx; k++)
        if (idx[k] < 0 || idx[k] >= ctx->n_bodies) return gx_fail(ctx, GX_ERR_INVALID_ARG, "n2: index out of range");
    GX_CUDA(ctx, cudaMemcpyAsync(didx, idx, sizeof(int64_t) * n_idx, cudaMemcpyHostToDevice, ctx->stream));
    GX_CUDA(ctx, launch_n2(ctx->n_bodies, dptr<double>(ctx->x), dptr<double>(ctx->y), dptr<double>(ctx->m),
                           ctx->eps * ctx->eps, didx, n_idx, dax, day, ctx->sm_count, ctx->stream));
    ctx->launches++;
    GX_CUDA(ctx, cudaGetLastError());
    GX_CUDA(ctx, cudaMemcpyAsync(ax, dax, sizeof(double) * n_idx, cudaMemcpyDeviceToHost, ctx->stream));
    GX_CUDA(ctx, cudaMemcpyAsync(ay, day, sizeof(double) * n_idx, cudaMemcpyDeviceToHost, ctx->stream));
    GX_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    return GX_OK;
}

// ---------------------------------------------------------------- allocation-free variant
// gx_n2_sampled_static: the sampled exact sum without a context and without any
// device allocation.  Some callers cannot allocate device memory at the moment
// they want a force check: a simulation whose device memory is owned by another
// runtime's caching allocator (which may already hold nearly all of HBM, so a
// cudaMalloc would fail or fragment it).  Their device arrays are passed in; the
// per-sample indices and results are staged through the file-scope array below
// instead of context scratch.  The call copies through pageable host memory and
// synchronises its stream, so that stream must not be capturing.
//
// The array is GX_N2_STATIC_MAX_SAMPLES * 24 bytes (96 KiB); every GPU that loads
// this library holds it until the process exits.  All calls on a device share it
// and it keeps the last call's contents: each call overwrites every slot it reads
// (indices, then one result per sample), so nothing has to start at zero, but
// calls that overlap on the GPU (other streams, other host threads) race on it.
namespace {
static __device__ __align__(256) unsigned char g_n2_static_scratch[GX_N2_STATIC_MAX_SAMPLES *
                                                                   (sizeof(int64_t) + 2 * sizeof(double))];
// Device address of the array per device ordinal, found once per device with that
// device current (the host-side symbol is a stand-in, not a device address) and kept
// for the life of the process: it belongs to the device's primary context, so a
// caller's cudaDeviceReset ends the use of this entry point in that process.
constexpr int kMaxDevices = 64;
void *g_n2_static_addr[kMaxDevices] = {};
std::mutex g_n2_static_mu;
}  // namespace

extern "C" int gx_n2_sampled_static(const double *x, const double *y, const double *m, int64_t n, double eps,
                                    const int64_t *idx, int64_t n_idx, double *ax, double *ay, void *stream) {
    if (n < 0 || n_idx < 0 || !(eps >= 0.0)) return GX_ERR_INVALID_ARG;
    if (n_idx > GX_N2_STATIC_MAX_SAMPLES) return GX_ERR_CAP_EXCEEDED;
    if (n_idx == 0) return GX_OK;
    if (!x || !y || !m || !idx || !ax || !ay) return GX_ERR_INVALID_ARG;
    for (int64_t k = 0; k < n_idx; k++)
        if (idx[k] < 0 || idx[k] >= n) return GX_ERR_INVALID_ARG;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return GX_ERR_INIT;
    void *base = nullptr;
    {
        std::lock_guard<std::mutex> lk(g_n2_static_mu);
        if (!g_n2_static_addr[dev]) {
            void *p = nullptr;
            if (cudaGetSymbolAddress(&p, g_n2_static_scratch) != cudaSuccess || !p) {
                cudaGetLastError();
                return GX_ERR_KERNEL_LOAD;
            }
            g_n2_static_addr[dev] = p;
        }
        base = g_n2_static_addr[dev];
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    int64_t *didx = static_cast<int64_t *>(base);
    double *dax = reinterpret_cast<double *>(didx + GX_N2_STATIC_MAX_SAMPLES);
    double *day = dax + GX_N2_STATIC_MAX_SAMPLES;
    if (cudaMemcpyAsync(didx, idx, sizeof(int64_t) * n_idx, cudaMemcpyHostToDevice, st) != cudaSuccess) {
        cudaGetLastError();
        return GX_ERR_CUDA;
    }
    int sms = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        launch_n2(n, x, y, m, eps * eps, didx, n_idx, dax, day, sms, st) != cudaSuccess) {
        cudaGetLastError();
        return GX_ERR_CUDA;
    }
    if (cudaMemcpyAsync(ax, dax, sizeof(double) * n_idx, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaMemcpyAsync(ay, day, sizeof(double) * n_idx, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess) {
        cudaGetLastError();
        return GX_ERR_CUDA;
    }
    return GX_OK;
}
