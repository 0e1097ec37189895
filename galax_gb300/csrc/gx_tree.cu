// gx_tree.cu -- device Tree::build (galax-core/src/lib.rs:163-361) and
// build_constrained (lib.rs:541-694).
//
// Bit-exactness rules: every value that decides topology or feeds a key is
// computed with separately rounded IEEE operations (__dmul_rn / __dadd_rn /
// __dsub_rn, which the compiler never contracts into FMA), in the reference's
// order: Morton normalisation, leaf mass and COM sums (body order), parent sums
// (child slot order), box centres and half-widths.
#include <cooperative_groups.h>

#include <algorithm>

#include "gx_cluster_scan.cuh"
#include "gx_internal.cuh"

namespace {

constexpr double kOneMinus = 1.0 - 1e-15;  // clamp bound of normalize (lib.rs:76)

// normalize (lib.rs:75-78): NaN clamps to NaN and casts to 0, like Rust `as u64`.
__device__ __forceinline__ uint64_t normalize_ref(double x, double lo, double hi) {
    double t = __ddiv_rn(__dsub_rn(x, lo), __dsub_rn(hi, lo));
    if (t < 0.0) t = 0.0;
    if (t > kOneMinus) t = kOneMinus;
    if (!(t > 0.0)) return 0ull;
    return __double2ull_rz(__dmul_rn(t, 2097152.0));
}

// The same cell index without the division.  The key uses t = RN(a / w), a = x - lo,
// w = hi - lo, only through floor(t * 2^21) clamped to [0, 2^21 - 1] (the clamp at
// 1 - 1e-15 and the clamp at 0 land in the end cells; NaN gives 0).  With
// iw = RN(1/w) (w > 0 finite, iw normal, formed once on the host) and |a/w| < 2,
// q = RN(a * iw) is within 1.5 * 2^-52 of a/w and RN(a/w) within 0.5 * 2^-52, so the two
// differ by at most 2^-51; times 2^21 (exact) that is 2^-30.  Hence when s = q * 2^21 lies
// farther than 2^-29 from an integer, floor(s) = floor(RN(a/w) * 2^21) exactly; values
// that near a cell boundary, and non-finite ones, take the correctly rounded division.
// One multiply instead of a correctly rounded FP64 division per coordinate.  iw21 =
// iw * 2^21 (exact), so s = RN(a * iw21) = RN(a * iw) * 2^21 wherever RN(a * iw) is
// normal; where it is not, s < 2^-29 and both take the division.  FP64 throughput on
// this part is a small fraction of FP32, so the tests on s (the window, the end cells,
// floor and the distance to the nearest integer) are integer operations on its bits,
// each equal to the FP64 comparison it replaces: for 1 <= s < 2^22 with exponent e the
// integer part is the significand shifted right by 52 - e and the fraction its low
// 52 - e bits, so "fraction in (2^-29, 1 - 2^-29)" is "low bits in (2^(23-e),
// 2^(52-e) - 2^(23-e))".
__device__ __forceinline__ uint64_t normalize_dev(double x, double lo, double hi, double iw21) {
    if (iw21 > 0.0) {
        const double s = __dmul_rn(__dsub_rn(x, lo), iw21);
        const int64_t b = __double_as_longlong(s);
        const uint64_t mag = (uint64_t)b & 0x7fffffffffffffffull;
        if (b <= 0) {                                            // s <= 0 (or a NaN with the sign bit)
            if (mag < 0x3ff0000000000000ull) return 0ull;        // -1 < s <= 0: the low cell
        } else if (b >= 0x413fffff80000000ll) {                  // s >= 2097151.5 (or +inf, NaN)
            if (b < 0x4150000000000000ll) return 2097151ull;     // s < 2^22: the top cell
        } else if (b < 0x3ff0000000000000ll) {                   // 0 < s < 1: cell 0 away from both ends
            if (b > 0x3e20000000000000ll && b < 0x3fefffffff000000ll) return 0ull;  // 2^-29 < s < 1 - 2^-29
        } else {                                                 // 1 <= s < 2097151.5
            const int sh = 52 - ((int)(b >> 52) - 1023);         // 32 .. 52
            const uint64_t sig = ((uint64_t)b & 0x000fffffffffffffull) | 0x0010000000000000ull;
            const uint64_t fr = sig & ((1ull << sh) - 1ull), eps = 1ull << (sh - 29);
            if (fr > eps && fr < (1ull << sh) - eps) return sig >> sh;
        }
    }
    return normalize_ref(x, lo, hi);
}

// spread_bits (lib.rs:85-93)
__device__ __forceinline__ uint64_t spread_dev(uint64_t v) {
    uint64_t x = v & ((1ull << 21) - 1);
    x = (x | (x << 16)) & 0x0000ffff0000ffffull;
    x = (x | (x << 8)) & 0x00ff00ff00ff00ffull;
    x = (x | (x << 4)) & 0x0f0f0f0f0f0f0f0full;
    x = (x | (x << 2)) & 0x3333333333333333ull;
    x = (x | (x << 1)) & 0x5555555555555555ull;
    return x;
}

__global__ void k_morton(const double *__restrict__ x, const double *__restrict__ y, int64_t n, double x0, double x1,
                         double y0, double y1, double ixw21, double iyw21, uint64_t *__restrict__ keys,
                         uint32_t *__restrict__ idx) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    keys[i] = spread_dev(normalize_dev(x[i], x0, x1, ixw21)) | (spread_dev(normalize_dev(y[i], y0, y1, iyw21)) << 1);
    if (idx) idx[i] = (uint32_t)i;
}

}  // namespace

// RN(1 / (hi - lo)) * 2^21 for the division-free normalisation, or 0 (the division path)
// when the width is not a positive finite number whose reciprocal is a normal number with
// a finite 2^21 multiple
double gx_inv_width21(double lo, double hi) {
    const double w = hi - lo;
    if (!(w > 0.0) || !std::isfinite(w)) return 0.0;
    const double iw = 1.0 / w, iw21 = iw * 2097152.0;
    return (std::isfinite(iw21) && std::fpclassify(iw) == FP_NORMAL) ? iw21 : 0.0;
}

void gx_launch_morton(gx_ctx *ctx, const double *x, const double *y, int64_t n, const double bounds[4], uint64_t *keys,
                      uint32_t *idx) {
    k_morton<<<gx_blocks(n, 256), 256, 0, ctx->stream>>>(x, y, n, bounds[0], bounds[1], bounds[2], bounds[3],
                                                         gx_inv_width21(bounds[0], bounds[1]),
                                                         gx_inv_width21(bounds[2], bounds[3]), keys, idx);
    ctx->launches++;
}

namespace {

// gather of the seven body arrays (Tree::permute, lib.rs:146-161), na of them per
// launch: the index read once per body and a body's loads in flight together.  The
// launch's source arrays are meant to fit the L2 together (a gather from unsorted order
// touches them at random; from the previous step's order, almost in sequence).
struct Arrays7 {
    const double *in[7];
    double *out[7];
};
// perm (or null) takes a copy of idx.
__global__ void k_permute7(const uint32_t *__restrict__ idx, int64_t n, int na, Arrays7 a, uint32_t *perm) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t j = idx[i];
    if (perm) perm[i] = j;
    double v[7];
#pragma unroll
    for (int k = 0; k < 7; k++)
        if (k < na) v[k] = a.in[k][j];
#pragma unroll
    for (int k = 0; k < 7; k++)
        if (k < na) a.out[k][i] = v[k];
}

__device__ __forceinline__ double fmin_rs(double a, double b) { return (a != a) ? b : ((b != b) ? a : (b < a ? b : a)); }
__device__ __forceinline__ double fmax_rs(double a, double b) { return (a != a) ? b : ((b != b) ? a : (b > a ? b : a)); }

// ---- parent rounds (lib.rs:269-354) ----
// The rounds run without host round trips: the level bounds, the shift and the round's
// segment and group counts live in a device state block, every kernel of a round reads
// them there, and the host only waits once per batch of rounds.  A round whose new
// level would not fit the node storage sets the overflow flag; the build is then redone
// with more storage.
enum {
    TS_S = 0, TS_E = 1, TS_C = 2, TS_SHIFT = 3, TS_NSEG = 4, TS_NG = 5, TS_FLAGS = 6, TS_ROUNDS = 7,
    TS_CHAIN_M = 8,  // min over adjacent leaves of the highest bit in which their first keys differ
    TS_CHAIN_L = 9,  // single-child rounds built by k_chain_rounds
    TS_BEFORE = 10,  // rounds built before k_rounds_cluster
    TS_N = 11
};
enum { TS_DONE = 1, TS_OVERFLOW = 2, TS_STUCK = 4 };
constexpr int TS_MAX_ROUNDS = 400;  // level starts kept: TS_MAX_ROUNDS + 2

__device__ __forceinline__ void tree_state_init(int64_t nl, int64_t *st, int64_t *lstart) {
    st[TS_S] = 0;
    st[TS_E] = st[TS_C] = nl;
    st[TS_SHIFT] = 2;
    st[TS_NSEG] = st[TS_NG] = 0;
    st[TS_FLAGS] = nl > 1 ? 0 : TS_DONE;
    st[TS_ROUNDS] = 0;
    st[TS_CHAIN_M] = 64;
    st[TS_CHAIN_L] = st[TS_BEFORE] = 0;
    lstart[0] = 0;
    lstart[1] = nl;
}

// leaf nodes (lib.rs:228-267); one thread per leaf, sums in body order.  The first also sets
// the build's state.
__global__ void k_leaves(const double *__restrict__ x, const double *__restrict__ y, const double *__restrict__ m,
                         const int32_t *__restrict__ rs, const int32_t *__restrict__ re, int64_t nl, double *cx,
                         double *cy, double *hw, double *mass, double *comx, double *comy, int32_t *bs, int32_t *be,
                         int4 *child, int32_t *parent, uint8_t *is_leaf, int64_t *st, int64_t *lstart) {
    int64_t L = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (L >= nl) return;
    if (L == 0) tree_state_init(nl, st, lstart);
    int32_t s = rs[L], e = re[L];
    double ms = 0.0, sx = 0.0, sy = 0.0;
    double bx0 = 1.7976931348623157e308, bx1 = -1.7976931348623157e308;
    double by0 = 1.7976931348623157e308, by1 = -1.7976931348623157e308;
    for (int32_t i = s; i < e; i++) {
        double mm = m[i], xi = x[i], yi = y[i];
        ms = __dadd_rn(ms, mm);
        sx = __dadd_rn(sx, __dmul_rn(xi, mm));
        sy = __dadd_rn(sy, __dmul_rn(yi, mm));
        bx0 = fmin_rs(bx0, xi); bx1 = fmax_rs(bx1, xi);
        by0 = fmin_rs(by0, yi); by1 = fmax_rs(by1, yi);
    }
    double c_x = __dmul_rn(__dadd_rn(bx0, bx1), 0.5), c_y = __dmul_rn(__dadd_rn(by0, by1), 0.5);
    double h = __dadd_rn(__dmul_rn(fmax_rs(__dsub_rn(bx1, bx0), __dsub_rn(by1, by0)), 0.5), 1e-15);
    cx[L] = c_x; cy[L] = c_y; hw[L] = h; mass[L] = ms;
    comx[L] = ms > 0.0 ? __ddiv_rn(sx, ms) : c_x;
    comy[L] = ms > 0.0 ? __ddiv_rn(sy, ms) : c_y;
    bs[L] = s; be[L] = e;
    child[L] = make_int4(-1, -1, -1, -1);
    parent[L] = -1;
    is_leaf[L] = 1;
}

// leaf ranges of Tree::build: chunks of n_max
__global__ void k_chunk_ranges(int64_t n, int64_t n_max, int64_t nl, int32_t *rs, int32_t *re) {
    int64_t L = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (L >= nl) return;
    int64_t s = L * n_max, e = s + n_max < n ? s + n_max : n;
    rs[L] = (int32_t)s;
    re[L] = (int32_t)e;
}


constexpr int TS_CLUSTER = 65536;  // levels of at most this many nodes: k_rounds_cluster
// the multi-block round kernels do nothing once the build is over or the level is small
__device__ __forceinline__ bool round_off(const int64_t *st) { return st[TS_FLAGS] != 0 || st[TS_C] <= TS_CLUSTER; }

__global__ void k_round_heads(const int64_t *st, const uint64_t *__restrict__ keys, const int32_t *__restrict__ bs,
                              int64_t *head) {
    if (round_off(st)) return;
    const int64_t s = st[TS_S], c = st[TS_C];
    const unsigned sh = (unsigned)st[TS_SHIFT] & 63u;
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= c) return;
    uint64_t g = keys[bs[s + i]] >> sh;
    head[i] = (i == 0) ? 1 : (g != (keys[bs[s + i - 1]] >> sh));
}

__global__ void k_seg_start(const int64_t *st, const int64_t *head, const int64_t *segex, int64_t *segstart) {
    if (round_off(st)) return;
    const int64_t c = st[TS_C];
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= c) return;
    if (head[i]) segstart[segex[i]] = i;
}

__global__ void k_seg_groups(const int64_t *st, const int64_t *segstart, int64_t *gcnt) {
    if (round_off(st)) return;
    const int64_t c = st[TS_C], nseg = st[TS_NSEG];
    int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= nseg) return;
    int64_t len = ((k + 1 < nseg) ? segstart[k + 1] : c) - segstart[k];
    gcnt[k] = (len + 3) / 4;
}

// the new level must fit the node storage; its child slots start empty
__global__ void k_round_open(int64_t *st, int64_t cap_nodes, int4 *child) {
    if (round_off(st)) return;
    const int64_t e = st[TS_E], ng = st[TS_NG];
    if (e + ng > cap_nodes) {
        if (blockIdx.x == 0 && threadIdx.x == 0) st[TS_FLAGS] |= TS_OVERFLOW;
        return;
    }
    int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (g < ng) child[e + g] = make_int4(-1, -1, -1, -1);
}

__global__ void k_assign(const int64_t *st, const int64_t *head, const int64_t *segex, const int64_t *segstart,
                         const int64_t *goff, int32_t *parent, int32_t *child) {
    if (round_off(st)) return;
    const int64_t s = st[TS_S], e = st[TS_E], c = st[TS_C];
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= c) return;
    int64_t seg = segex[i] + head[i] - 1;
    int64_t pos = i - segstart[seg];
    int64_t g = goff[seg] + pos / 4;
    parent[s + i] = (int32_t)(e + g);
    child[(e + g) * 4 + (pos & 3)] = (int32_t)(s + i);
}

// after a round: record the new level, move to it, and stop at a single node
__global__ void k_round_close(int64_t *st, int64_t *level_start) {
    if (round_off(st)) return;
    const int64_t e = st[TS_E], ng = st[TS_NG];
    if (st[TS_ROUNDS] >= TS_MAX_ROUNDS) {
        st[TS_FLAGS] |= TS_STUCK;
        return;
    }
    const int64_t r = ++st[TS_ROUNDS];
    level_start[r + 1] = e + ng;
    st[TS_S] = e;
    st[TS_E] = e + ng;
    st[TS_C] = ng;
    st[TS_SHIFT] += 2;
    if (ng <= 1) st[TS_FLAGS] |= TS_DONE;
}

// One parent of a round (lib.rs:298-335): mass, COM from the children's com x mass,
// centre of the union of the children's boxes, hw = 2 x the largest child hw, body range.
__device__ __forceinline__ void parent_fields_one(int64_t q, double *cx, double *cy, double *hw, double *mass,
                                                  double *comx, double *comy, int32_t *bs, int32_t *be,
                                                  const int4 *child, int32_t *parent, uint8_t *is_leaf) {
    int4 c4 = child[q];
    int cc[4] = {c4.x, c4.y, c4.z, c4.w};
    double ms = 0.0, sx = 0.0, sy = 0.0, mh = 0.0;
    double bx0 = 1.7976931348623157e308, bx1 = -1.7976931348623157e308;
    double by0 = 1.7976931348623157e308, by1 = -1.7976931348623157e308;
    int first = cc[0], last = cc[0];
    for (int k = 0; k < 4; k++) {
        int s = cc[k];
        if (s < 0) break;
        last = s;
        double cm = mass[s], h = hw[s], ccx = cx[s], ccy = cy[s];
        ms = __dadd_rn(ms, cm);
        sx = __dadd_rn(sx, __dmul_rn(comx[s], cm));
        sy = __dadd_rn(sy, __dmul_rn(comy[s], cm));
        if (h > mh) mh = h;
        double cl = __dsub_rn(ccx, h), cr = __dadd_rn(ccx, h);
        if (cl < bx0) bx0 = cl;
        if (cr > bx1) bx1 = cr;
        double cb = __dsub_rn(ccy, h), ct = __dadd_rn(ccy, h);
        if (cb < by0) by0 = cb;
        if (ct > by1) by1 = ct;
    }
    double c_x = __dmul_rn(__dadd_rn(bx0, bx1), 0.5), c_y = __dmul_rn(__dadd_rn(by0, by1), 0.5);
    cx[q] = c_x; cy[q] = c_y; hw[q] = __dmul_rn(mh, 2.0); mass[q] = ms;
    comx[q] = ms > 0.0 ? __ddiv_rn(sx, ms) : c_x;
    comy[q] = ms > 0.0 ? __ddiv_rn(sy, ms) : c_y;
    bs[q] = bs[first];
    be[q] = be[last];
    if (parent) parent[q] = -1;  // null: the topology is already there
    is_leaf[q] = 0;
}

__global__ void k_parent_fields(const int64_t *st, double *cx, double *cy, double *hw, double *mass, double *comx,
                                double *comy, int32_t *bs, int32_t *be, const int4 *child, int32_t *parent,
                                uint8_t *is_leaf) {
    if (round_off(st)) return;
    const int64_t e = st[TS_E], ng = st[TS_NG];
    int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= ng) return;
    parent_fields_one(e + g, cx, cy, hw, mass, comx, comy, bs, be, child, parent, is_leaf);
}

// Single-child rounds.  Round r groups consecutive nodes whose first bodies' keys agree
// after >> 2r; while every node of the level is its own group, the round makes one parent
// per node.  Starting from the leaves, that holds for rounds r = 1 .. m/2 exactly, m the
// smallest, over adjacent leaves, highest bit in which their first keys differ (below
// it the prefixes differ for every pair; at 2r > m one pair agrees).  k_chain_depth finds
// m; k_chain_rounds builds those rounds at once, a thread per leaf walking its chain
// (level l node x + l nl is the one parent of x + (l-1) nl, its fields by the same
// parent_fields_one as a round), and moves the round state past them, so the multi-block
// rounds start at the first round that groups.  At 1M Plummer that is the first eight
// rounds: 8 x 13 launches become 2.
__global__ void k_chain_depth(int64_t nl, const uint64_t *__restrict__ keys, const int32_t *__restrict__ bs,
                              int64_t *st) {
    __shared__ int wmin[8];
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    int m = 64;
    if (i >= 1 && i < nl) {
        const uint64_t d = keys[bs[i]] ^ keys[bs[i - 1]];
        m = d ? 63 - __clzll((long long)d) : -1;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = min(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) wmin[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        int b = wmin[0];
        for (int w = 1; w < (int)(blockDim.x >> 5); w++) b = min(b, wmin[w]);
        if (b < 64) atomicMin(reinterpret_cast<long long *>(st + TS_CHAIN_M), (long long)b);
    }
}

__global__ void k_chain_rounds(int64_t *st, int64_t *level_start, int64_t nl, int64_t cap_nodes, double *cx,
                               double *cy, double *hw, double *mass, double *comx, double *comy, int32_t *bs,
                               int32_t *be, int4 *child, int32_t *parent, uint8_t *is_leaf) {
    if (st[TS_FLAGS] != 0) return;
    int64_t L = st[TS_CHAIN_M] >= 2 ? st[TS_CHAIN_M] / 2 : 0;
    L = min(L, cap_nodes / nl - 1);
    L = min(L, (int64_t)TS_MAX_ROUNDS - 2);
    if (L <= 0) return;
    const int64_t x = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (x < nl) {
        for (int64_t l = 1; l <= L; l++) {
            const int64_t q = x + l * nl, c = x + (l - 1) * nl;
            child[q] = make_int4((int)c, -1, -1, -1);
            parent[c] = (int32_t)q;
            parent_fields_one(q, cx, cy, hw, mass, comx, comy, bs, be, child, parent, is_leaf);
        }
    }
    if (x == 0) {
        for (int64_t r = 1; r <= L; r++) level_start[r + 1] = (r + 1) * nl;
        st[TS_S] = L * nl;
        st[TS_E] = (L + 1) * nl;
        st[TS_C] = nl;
        st[TS_SHIFT] = 2 + 2 * L;
        st[TS_ROUNDS] = L;
        st[TS_CHAIN_L] = L;
    }
}

// The rounds of levels of at most TS_CLUSTER nodes: their topology in one launch
// (k_rounds_cluster), then the nodes' fields level by level.
//
// Which nodes a round groups depends on the leaves alone.  Let d be the highest bit in which
// a node's first key differs from the first key of the node before it; the node begins a
// segment of the round with shift sh exactly when d >= sh.  A parent inherits the d of its
// first child: if that child began a segment, the children before it have smaller d, so its
// d is the parents' too, and if not, d < sh and neither it nor its parent begins a segment
// again.  So a thread loads the d of a run of consecutive nodes once (a byte each, in one
// register pair), and every round is two scans over the cluster, of the last segment head
// and of the groups begun, with nothing read from global memory; the thread that holds a
// group's first node keeps the parent.  The groups and their order are those of the
// multi-block rounds: a segment's nodes by fours.
constexpr int RC_THREADS = CS_THREADS;
constexpr int RC_RUN = 8;  // nodes a thread holds at most: TS_CLUSTER nodes on 8 blocks
static_assert(TS_CLUSTER <= 8 * RC_THREADS * RC_RUN, "a level fits the smaller cluster");

// Inclusive scan over the block (op: max or sum) of one int a thread; wt: 33 ints, the last
// one the block's result.
template <class Op>
__device__ __forceinline__ int rc_block_scan(int v, int *wt, Op op, int zero) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v = op(v, u);
    }
    if (lane == 31) wt[w] = v;
    __syncthreads();
    if (w == 0) {
        int x = wt[lane];
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x = op(x, u);
        }
        wt[lane] = x;
        if (lane == 31) wt[32] = x;
    }
    __syncthreads();
    return w > 0 ? op(v, wt[w - 1]) : op(v, zero);
}

__global__ void __launch_bounds__(RC_THREADS) k_rounds_cluster(int64_t *st, int64_t *level_start, int64_t cap_nodes,
                                                               const uint64_t *__restrict__ keys,
                                                               const int32_t *__restrict__ bs, int32_t *child,
                                                               int32_t *parent) {
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    const int nb = (int)cl.num_blocks(), rank = (int)cl.block_rank();
    const int t = threadIdx.x, lane = t & 31;
    __shared__ int wmax[2][33], wsum[2][33];  // by the round's parity: a block reads the others' after one barrier
    __shared__ int prev_last, prev_cnt, all_cnt;
    // the round state, kept by every thread alike and written back at the end
    int64_t s = st[TS_S], e = st[TS_E], flags = st[TS_FLAGS], rounds = st[TS_ROUNDS], shift = st[TS_SHIFT];
    int64_t c = st[TS_C];
    cl.sync();  // all blocks have read the state before one writes it
    if (flags != 0 || c > TS_CLUSTER) return;
    // this thread's nodes i0 .. i0 + n - 1 and their d + 1 (0: equal keys; 255: the first node)
    const int per = (int)((c + nb * RC_THREADS - 1) / (nb * RC_THREADS));
    int i0 = (int)min(c, (int64_t)(rank * RC_THREADS + t) * per), n = (int)min(c, (int64_t)i0 + per) - i0;
    uint64_t dv = 0;
    const auto load_d = [&](const auto &key) {
        dv = 0;
        uint64_t p = n > 0 && i0 > 0 ? key(s + i0 - 1) : 0;
        for (int k = 0; k < n; k++) {
            const uint64_t g = key(s + i0 + k), x = g ^ p;
            const int d1 = i0 + k == 0 ? 255 : (x ? 64 - __clzll((long long)x) : 0);
            dv |= (uint64_t)d1 << (8 * k);
            p = g;
        }
    };
    load_d([&](int64_t q) { return keys[bs[q]]; });
    const auto mx = [](int a, int b) { return max(a, b); };
    const auto sm = [](int a, int b) { return a + b; };
    for (int par = 0; flags == 0; par ^= 1) {
        // The reference's shift is taken modulo 64 (a tree of more than 4^11 leaves in an order
        // without runs gets there): at 0 again, the d of the nodes' own first keys count, which
        // are those of their first leaves.
        const int sh = (int)(shift & 63);
        if (sh == 0) {
            cl.sync();  // the last round's child slots are written
            const int64_t nl = level_start[1];
            const auto key = [&](int64_t q) {
                while (q >= nl) q = child[4 * q];
                return keys[bs[q]];
            };
            load_d(key);
        }
        // the last segment head before this thread's run
        int last = -1;
        for (int k = 0; k < n; k++)
            if ((int)((dv >> (8 * k)) & 255u) > sh) last = i0 + k;
        const int m = rc_block_scan(last, wmax[par], mx, -1);
        int head = __shfl_up_sync(0xffffffffu, m, 1);
        if (lane == 0) head = t > 0 ? wmax[par][(t >> 5) - 1] : -1;
        cl.sync();
        if (t < 32) {
            int v = t < rank ? *cl.map_shared_rank(&wmax[par][32], t) : -1;
            for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
            if (t == 0) prev_last = v;
        }
        __syncthreads();
        head = max(head, prev_last);
        // groups of four within each segment: those that begin in this run
        int cnt = 0, h = head;
        for (int k = 0; k < n; k++) {
            if ((int)((dv >> (8 * k)) & 255u) > sh) h = i0 + k;
            cnt += ((i0 + k - h) & 3) == 0;
        }
        int g = rc_block_scan(cnt, wsum[par], sm, 0) - cnt;
        cl.sync();
        if (t < 32) {
            const int v = t < nb ? *cl.map_shared_rank(&wsum[par][32], t) : 0;
            int before = t < rank ? v : 0, total = v;
            for (int o = 16; o > 0; o >>= 1) {
                before += __shfl_xor_sync(0xffffffffu, before, o);
                total += __shfl_xor_sync(0xffffffffu, total, o);
            }
            if (t == 0) {
                prev_cnt = before;
                all_cnt = total;
            }
        }
        __syncthreads();
        g += prev_cnt;
        const int64_t ng = all_cnt;
        if (e + ng > cap_nodes) {
            flags |= TS_OVERFLOW;
            break;
        }
        if (rounds >= TS_MAX_ROUNDS) {
            flags |= TS_STUCK;
            break;
        }
        // parents and child slots; the parents of the groups begun here are this thread's next run
        int q = g - 1, kept = 0;
        uint64_t nd = 0;
        h = head;
        for (int k = 0; k < n; k++) {
            const int i = i0 + k;
            const uint64_t d = (dv >> (8 * k)) & 255u;
            if ((int)d > sh) h = i;
            const int pos = (i - h) & 3;
            if (pos == 0) {
                q++;
                nd |= d << (8 * kept++);
            }
            parent[s + i] = (int32_t)(e + q);
            child[(e + q) * 4 + pos] = (int32_t)(s + i);
        }
        dv = nd;
        n = kept;
        i0 = g;
        s = e;
        e += ng;
        c = ng;
        shift += 2;
        rounds++;
        if (rank == 0 && t == 0) level_start[rounds + 1] = e;
        if (ng <= 1) flags |= TS_DONE;
    }
    if ((flags & TS_DONE) && rank == 0 && t == 0) parent[s] = -1;  // the root
    cl.sync();  // no block leaves while another may read its shared memory
    if (rank == 0 && t == 0) {
        st[TS_S] = s;
        st[TS_E] = e;
        st[TS_C] = c;
        st[TS_SHIFT] = shift;
        st[TS_FLAGS] = flags;
        st[TS_ROUNDS] = rounds;
    }
}

// every child slot of the new levels starts empty
__global__ void k_slots_clear(const int64_t *st, int64_t cap_nodes, int4 *child) {
    if (st[TS_FLAGS] != 0) return;
    const int64_t q = st[TS_E] + (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (q < cap_nodes) child[q] = make_int4(-1, -1, -1, -1);
}

// The fields of the nodes built by k_rounds_cluster: the levels after the first `from`
// (built before it), the k-th of them by launch k of k_fields_level over the whole GPU
// while it has more than FIELDS_SMALL nodes, the rest in one cluster (k_fields_small).
constexpr int FIELDS_SMALL = 2048;
constexpr int FIELDS_BLOCKS = 8, FIELDS_THREADS = 256;
__global__ void k_fields_level(const int64_t *st, const int64_t *level_start, int64_t lv, double *cx, double *cy,
                               double *hw, double *mass, double *comx, double *comy, int32_t *bs, int32_t *be,
                               const int4 *child, uint8_t *is_leaf) {
    lv += st[TS_BEFORE];
    if (!(st[TS_FLAGS] & TS_DONE) || lv > st[TS_ROUNDS]) return;
    const int64_t s = level_start[lv], c = level_start[lv + 1] - s;
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (c <= FIELDS_SMALL || i >= c) return;
    parent_fields_one(s + i, cx, cy, hw, mass, comx, comy, bs, be, child, nullptr, is_leaf);
}
__global__ void __launch_bounds__(FIELDS_THREADS) k_fields_small(const int64_t *st, const int64_t *level_start,
                                                                int64_t launched, double *cx, double *cy, double *hw,
                                                                double *mass, double *comx, double *comy, int32_t *bs,
                                                                int32_t *be, const int4 *child, uint8_t *is_leaf) {
    cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
    if (!(st[TS_FLAGS] & TS_DONE)) return;
    const int64_t n = st[TS_ROUNDS], from = st[TS_BEFORE] + 1;
    for (int64_t lv = from; lv <= n; lv++) {
        const int64_t s = level_start[lv], c = level_start[lv + 1] - s;
        if (c > FIELDS_SMALL && lv < from + launched) continue;
        for (int64_t i = cl.block_rank() * FIELDS_THREADS + threadIdx.x; i < c; i += FIELDS_BLOCKS * FIELDS_THREADS)
            parent_fields_one(s + i, cx, cy, hw, mass, comx, comy, bs, be, child, nullptr, is_leaf);
        cl.sync();
    }
}

// the rounds built so far: the cluster's levels come after them
__global__ void k_mark_before(int64_t *st) { st[TS_BEFORE] = st[TS_ROUNDS]; }

// ---- build_constrained helpers (lib.rs:541-694) ----
// leaf ranges bounded by n_max and by the sorted split points (lib.rs:603-613):
// computed on the host from the split list, which is small.

}  // namespace

// Node storage with capacity growth (contents preserved).
static int ensure_nodes(gx_ctx *ctx, int64_t need) {
    struct F { DevBuf *b; size_t sz; };
    F f[] = {{&ctx->cx, 8}, {&ctx->cy, 8}, {&ctx->hw, 8}, {&ctx->mass, 8}, {&ctx->comx, 8}, {&ctx->comy, 8},
             {&ctx->bs, 4}, {&ctx->be, 4}, {&ctx->child, 16}, {&ctx->parent, 4}, {&ctx->is_leaf, 1}};
    for (auto &e : f) {
        size_t want = e.sz * (size_t)need;
        if (e.b->bytes >= want) continue;
        size_t nb = std::max(want, e.b->bytes * 2);
        void *p = nullptr;
        if (cudaMalloc(&p, nb) != cudaSuccess) return gx_fail(ctx, GX_ERR_ALLOC, "node storage allocation failed");
        if (e.b->p) {
            cudaMemcpyAsync(p, e.b->p, e.b->bytes, cudaMemcpyDeviceToDevice, ctx->stream);
            cudaStreamSynchronize(ctx->stream);
            cudaFree(e.b->p);
        }
        e.b->p = p;
        e.b->bytes = nb;
    }
    return GX_OK;
}

// Builds nodes from leaf ranges already in scratch (rs, re as int32), using ctx->keys
// (Morton keys of the tree-ordered bodies).
static int build_from_ranges(gx_ctx *ctx, const int32_t *rs, const int32_t *re, int64_t nl) {
    if (nl <= 0) return gx_fail(ctx, GX_ERR_STATE, "tree build: no leaves");
    // node storage: the last build's node count (a rebuild every step keeps it), else a
    // guess (10 to 20 nodes a leaf: the single-child levels); a round that overflows it makes
    // the build start again with more
    int64_t cap = std::max<int64_t>(nl * 12 + 512, ctx->hint_nodes + ctx->hint_nodes / 8 + 64);
    // per-round scratch: head, segex, segstart, gcnt, goff (int64, <= nl each)
    GX_TRY(gx_ensure(ctx, ctx->scratch_a, sizeof(int64_t) * (size_t)(nl + 1) * 5));
    GX_TRY(gx_ensure(ctx, ctx->tree_state, sizeof(int64_t) * (TS_N + TS_MAX_ROUNDS + 2)));
    int64_t *st = dptr<int64_t>(ctx->tree_state);
    int64_t *lstart = st + TS_N;  // level starts
    int64_t *head = dptr<int64_t>(ctx->scratch_a);
    int64_t *segex = head + (nl + 1), *segstart = segex + (nl + 1), *gcnt = segstart + (nl + 1),
            *goff = gcnt + (nl + 1);
    const unsigned gb = gx_blocks(nl, 256);
    int64_t hs[TS_N + TS_MAX_ROUNDS + 2];  // the state and, behind it, the level starts
    for (int attempt = 0;; attempt++) {
        if (attempt == 8) return gx_fail(ctx, GX_ERR_ALLOC, "tree build: node storage keeps overflowing");
        GX_TRY(ensure_nodes(ctx, cap));
        k_leaves<<<gx_blocks(nl, 128), 128, 0, ctx->stream>>>(
            dptr<double>(ctx->x), dptr<double>(ctx->y), dptr<double>(ctx->m), rs, re, nl, dptr<double>(ctx->cx),
            dptr<double>(ctx->cy), dptr<double>(ctx->hw), dptr<double>(ctx->mass), dptr<double>(ctx->comx),
            dptr<double>(ctx->comy), dptr<int32_t>(ctx->bs), dptr<int32_t>(ctx->be), dptr<int4>(ctx->child),
            dptr<int32_t>(ctx->parent), dptr<uint8_t>(ctx->is_leaf), st, lstart);
        ctx->launches++;
        if (nl > 1) {
            k_chain_depth<<<gx_blocks(nl, 256), 256, 0, ctx->stream>>>(nl, dptr<uint64_t>(ctx->keys),
                                                                      dptr<int32_t>(ctx->bs), st);
            k_chain_rounds<<<gx_blocks(nl, 128), 128, 0, ctx->stream>>>(
                st, lstart, nl, cap, dptr<double>(ctx->cx), dptr<double>(ctx->cy), dptr<double>(ctx->hw),
                dptr<double>(ctx->mass), dptr<double>(ctx->comx), dptr<double>(ctx->comy), dptr<int32_t>(ctx->bs),
                dptr<int32_t>(ctx->be), dptr<int4>(ctx->child), dptr<int32_t>(ctx->parent),
                dptr<uint8_t>(ctx->is_leaf));
            ctx->launches += 2;
        }
        // multi-block rounds, if any level may need them, in batches (the last build's count
        // first), each batch followed by the cluster's rounds
        int batch = nl > TS_CLUSTER ? std::max(4, ctx->hint_big_rounds + 1) : 0;
        int issued = 0;
        for (;;) {
            for (int r = 0; r < batch; r++) {
                k_round_heads<<<gb, 256, 0, ctx->stream>>>(st, dptr<uint64_t>(ctx->keys), dptr<int32_t>(ctx->bs), head);
                GX_TRY(gx_exclusive_scan_i64_devn(ctx, head, segex, st + TS_C, 0, nl, st + TS_NSEG));
                k_seg_start<<<gb, 256, 0, ctx->stream>>>(st, head, segex, segstart);
                k_seg_groups<<<gb, 256, 0, ctx->stream>>>(st, segstart, gcnt);
                GX_TRY(gx_exclusive_scan_i64_devn(ctx, gcnt, goff, st + TS_NSEG, 0, nl, st + TS_NG));
                k_round_open<<<gb, 256, 0, ctx->stream>>>(st, cap, dptr<int4>(ctx->child));
                k_assign<<<gb, 256, 0, ctx->stream>>>(st, head, segex, segstart, goff, dptr<int32_t>(ctx->parent),
                                                      dptr<int32_t>(ctx->child));
                k_parent_fields<<<gx_blocks(nl, 128), 128, 0, ctx->stream>>>(
                    st, dptr<double>(ctx->cx), dptr<double>(ctx->cy), dptr<double>(ctx->hw), dptr<double>(ctx->mass),
                    dptr<double>(ctx->comx), dptr<double>(ctx->comy), dptr<int32_t>(ctx->bs), dptr<int32_t>(ctx->be),
                    dptr<int4>(ctx->child), dptr<int32_t>(ctx->parent), dptr<uint8_t>(ctx->is_leaf));
                k_round_close<<<1, 1, 0, ctx->stream>>>(st, lstart);
                ctx->launches += 7;
            }
            // the rest of the topology, then the fields of its levels (the last build's number
            // of large ones, four on a first build)
            k_mark_before<<<1, 1, 0, ctx->stream>>>(st);
            k_slots_clear<<<gx_blocks(cap - nl, 256), 256, 0, ctx->stream>>>(st, cap, dptr<int4>(ctx->child));
            GX_TRY(cs_launch(ctx, nl, k_rounds_cluster, st, lstart, cap, dptr<uint64_t>(ctx->keys),
                             dptr<int32_t>(ctx->bs), dptr<int32_t>(ctx->child), dptr<int32_t>(ctx->parent)));
            const int large = nl > FIELDS_SMALL ? (ctx->hint_field_levels > 0 ? ctx->hint_field_levels : 4) : 0;
            const unsigned gf = gx_blocks(std::min<int64_t>(nl, TS_CLUSTER), 128);
            for (int k = 1; k <= large; k++)
                k_fields_level<<<gf, 128, 0, ctx->stream>>>(
                    st, lstart, k, dptr<double>(ctx->cx), dptr<double>(ctx->cy), dptr<double>(ctx->hw),
                    dptr<double>(ctx->mass), dptr<double>(ctx->comx), dptr<double>(ctx->comy), dptr<int32_t>(ctx->bs),
                    dptr<int32_t>(ctx->be), dptr<int4>(ctx->child), dptr<uint8_t>(ctx->is_leaf));
            cudaLaunchConfig_t cfg = {};
            cudaLaunchAttribute at = {};
            at.id = cudaLaunchAttributeClusterDimension;
            at.val.clusterDim.x = FIELDS_BLOCKS;
            at.val.clusterDim.y = at.val.clusterDim.z = 1;
            cfg.gridDim = dim3(FIELDS_BLOCKS);
            cfg.blockDim = dim3(FIELDS_THREADS);
            cfg.stream = ctx->stream;
            cfg.attrs = &at;
            cfg.numAttrs = 1;
            GX_CUDA(ctx, cudaLaunchKernelEx(&cfg, k_fields_small, (const int64_t *)st, (const int64_t *)lstart,
                                            (int64_t)large, dptr<double>(ctx->cx), dptr<double>(ctx->cy),
                                            dptr<double>(ctx->hw), dptr<double>(ctx->mass), dptr<double>(ctx->comx),
                                            dptr<double>(ctx->comy), dptr<int32_t>(ctx->bs), dptr<int32_t>(ctx->be),
                                            (const int4 *)dptr<int4>(ctx->child), dptr<uint8_t>(ctx->is_leaf)));
            ctx->launches += 3 + large;
            GX_CUDA(ctx, cudaGetLastError());
            issued += batch;
            static_assert(sizeof(hs) <= GX_PIN, "the state and the level starts in one gx_fetch");
            GX_TRY(gx_fetch(ctx, hs, st, sizeof(hs)));
            if (hs[TS_FLAGS] & TS_STUCK) return gx_fail(ctx, GX_ERR_STATE, "tree build did not converge");
            if (hs[TS_FLAGS] != 0) break;
            batch = 8;
        }
        if (!(hs[TS_FLAGS] & TS_OVERFLOW)) break;
        cap *= 2;
    }
    const int64_t rounds = hs[TS_ROUNDS];
    std::vector<int64_t> ls(hs + TS_N, hs + TS_N + rounds + 2);
    ctx->level_start.assign(ls.begin(), ls.end());
    ctx->hint_big_rounds = 0;  // multi-block rounds after the single-child ones
    for (size_t l = 0; l + 2 < ls.size(); l++)
        if (ls[l + 1] - ls[l] > TS_CLUSTER) ctx->hint_big_rounds++;
    ctx->hint_big_rounds = std::max<int64_t>(0, ctx->hint_big_rounds - hs[TS_CHAIN_L]);
    ctx->hint_field_levels = 0;  // levels of k_fields_level
    for (int64_t l = hs[TS_BEFORE] + 1; l <= rounds; l++)
        if (ls[l + 1] - ls[l] > FIELDS_SMALL) ctx->hint_field_levels++;
    const int64_t nn = ls.back();
    ctx->n_nodes = nn;
    ctx->hint_nodes = nn;
    ctx->n_leaves = nl;
    ctx->n_levels = (int32_t)ctx->level_start.size() - 1;
    return GX_OK;
}

// Bodies must already be resident (ctx->x ... in input order).  Sorts them into
// Morton order on the device, then builds the node hierarchy.
int gx_tree_build_device(gx_ctx *ctx, int64_t n, int64_t n_max, const double bounds[4], int flags) {
    ctx->have_tree = false;
    ctx->plan_ref_valid = ctx->plan_acc_valid = ctx->ref_lists_valid = false;
    if (n <= 0) {
        ctx->n_nodes = ctx->n_leaves = 0;
        ctx->n_levels = 0;
        ctx->level_start.assign(1, 0);
        ctx->have_tree = true;
        return GX_OK;
    }
    if (n >= 0x7fffffffLL) return gx_fail(ctx, GX_ERR_CAP_EXCEEDED, "n must be < 2^31");
    // keys + permutation
    GX_TRY(gx_ensure(ctx, ctx->keys, sizeof(uint64_t) * n));
    GX_TRY(gx_ensure(ctx, ctx->scratch_b, sizeof(uint64_t) * n));               // keys alt
    GX_TRY(gx_ensure(ctx, ctx->scratch_c, sizeof(uint32_t) * n * 2));           // idx, idx alt
    uint64_t *keys = dptr<uint64_t>(ctx->keys), *keys_alt = dptr<uint64_t>(ctx->scratch_b);
    uint32_t *idx = dptr<uint32_t>(ctx->scratch_c), *idx_alt = idx + n;
    gx_launch_morton(ctx, dptr<double>(ctx->x), dptr<double>(ctx->y), n, bounds, keys, idx);
    GX_CUDA(ctx, cudaGetLastError());
    if (!(flags & GX_BUILD_BALANCED)) {
        bool alt = false;
        GX_TRY(gx_radix_sort_u64(ctx, keys, idx, n, 0, 42, keys_alt, idx_alt, &alt));
        if (alt) {
            GX_CUDA(ctx, cudaMemcpyAsync(keys, keys_alt, sizeof(uint64_t) * n, cudaMemcpyDeviceToDevice, ctx->stream));
            idx = idx_alt;
        }
        // permute the seven arrays into their spare copies, then swap them in; as many
        // arrays per launch as fit in half of the 129 MB L2 together (all seven at 1M)
        DevBuf *arrs[7] = {&ctx->x, &ctx->y, &ctx->vx, &ctx->vy, &ctx->m, &ctx->ax, &ctx->ay};
        const int per = (int)std::max<int64_t>(1, std::min<int64_t>(7, ((int64_t)64 << 20) / (8 * n)));
        GX_TRY(gx_ensure(ctx, ctx->perm, sizeof(uint32_t) * n));
        for (int k0 = 0; k0 < 7; k0 += per) {
            const int na = std::min(per, 7 - k0);
            Arrays7 a7{};
            for (int k = 0; k < na; k++) {
                GX_TRY(gx_ensure(ctx, ctx->body_alt[k0 + k], sizeof(double) * n));
                a7.in[k] = dptr<double>(*arrs[k0 + k]);
                a7.out[k] = dptr<double>(ctx->body_alt[k0 + k]);
            }
            k_permute7<<<gx_blocks(n, 256), 256, 0, ctx->stream>>>(
                idx, n, na, a7, k0 == 0 ? dptr<uint32_t>(ctx->perm) : nullptr);
            ctx->launches++;
        }
        for (int k = 0; k < 7; k++) std::swap(*arrs[k], ctx->body_alt[k]);
        GX_CUDA(ctx, cudaGetLastError());
    }
    int64_t nl = (n + n_max - 1) / n_max;
    GX_TRY(gx_ensure(ctx, ctx->scratch_f, sizeof(int32_t) * (size_t)(2 * nl + 2) + 64));
    // scratch_f held the sort's digit totals; the sort is finished at this point
    int32_t *rs = dptr<int32_t>(ctx->scratch_f), *re = rs + nl;
    k_chunk_ranges<<<gx_blocks(nl, 256), 256, 0, ctx->stream>>>(n, n_max, nl, rs, re);
    ctx->launches++;
    GX_CUDA(ctx, cudaGetLastError());
    ctx->n_bodies = n;
    GX_TRY(build_from_ranges(ctx, rs, re, nl));
    ctx->have_tree = true;
    return GX_OK;
}

// Rebuild with forced split points (build_with_constraints, lib.rs:592-694): no sort;
// keys from the resident bodies.  Exposed to the balanced builder in gx_lists.cu.
int gx_tree_rebuild_with_splits(gx_ctx *ctx, int64_t n_max, const double bounds[4], const std::vector<int64_t> &splits) {
    int64_t n = ctx->n_bodies;
    GX_TRY(gx_ensure(ctx, ctx->keys, sizeof(uint64_t) * n));
    GX_TRY(gx_ensure(ctx, ctx->scratch_c, sizeof(uint32_t) * n * 2));
    gx_launch_morton(ctx, dptr<double>(ctx->x), dptr<double>(ctx->y), n, bounds, dptr<uint64_t>(ctx->keys),
                     dptr<uint32_t>(ctx->scratch_c));
    std::vector<int32_t> hrs, hre;
    int64_t s = 0;
    size_t k = 0;
    while (s < n) {
        int64_t bound = std::min(s + n_max, n);
        while (k < splits.size() && splits[k] <= s) k++;
        int64_t e = (k < splits.size() && splits[k] < bound) ? splits[k] : bound;
        hrs.push_back((int32_t)s);
        hre.push_back((int32_t)e);
        s = e;
    }
    int64_t nl = (int64_t)hrs.size();
    GX_TRY(gx_ensure(ctx, ctx->scratch_f, sizeof(int32_t) * (size_t)(2 * nl + 2) + 64));
    int32_t *rs = dptr<int32_t>(ctx->scratch_f), *re = rs + nl;
    GX_CUDA(ctx, cudaMemcpyAsync(rs, hrs.data(), sizeof(int32_t) * nl, cudaMemcpyHostToDevice, ctx->stream));
    GX_CUDA(ctx, cudaMemcpyAsync(re, hre.data(), sizeof(int32_t) * nl, cudaMemcpyHostToDevice, ctx->stream));
    GX_TRY(build_from_ranges(ctx, rs, re, nl));
    ctx->have_tree = true;
    return GX_OK;
}
