// groupfilter.cu -- fused collaborative filtering of matched groups.
//
// One CTA filters one group end to end, with everything staged in shared
// memory:
//   1. gather the N patches of the observation (and of the pilot for Wiener)
//      and of the Poisson variance volume V = max(scale * max(x, 0), floor)
//      (src/bmnd/variance.py:556-598);
//   2. forward separable transform, group axis first then the patch axes
//      (transforms.py:209-255); every axis product accumulates with one fused
//      multiply-add per term in k order, which is how NumPy's sgemm evaluates
//      the reference's matrix products;
//   3. noise standard deviation of every coefficient: the approximate
//      propagation through squared transforms (variance.py:613-623,
//      :1647-1653) and, for the first k group planes, the exact
//      overlap-aware variance sum_v V_v (sum_{e in v} E_e)^2 over the union of
//      overlapping patch voxels (variance.py:758-851, :920-975), then the
//      plane limiting rule (variance.py:1572-1631);
//   4. hard thresholding with the tolerance-aware Poisson mask
//      (bmndalgo.py:460-485, poisson.py:30-46) or the variance-scaled Poisson
//      Wiener gain (wiener.py:24-95, bmndalgo.py:878-894);
//   5. per-patch aggregation weights 1 / (sum_g Ginv[o,g]^2 plane_risk[g] +
//      eps) (aggregationweights.py:213-259, :616-653), or one weight per group
//      from its exact windowed-synthesis risk (wiener.py:638-822);
//   6. inverse transform and weighted Kaiser-window scatter: to the members'
//      store rows, summed in a fixed order afterwards, or by atomics into
//      float64 numerator / denominator volumes (patchaggregation.py:170-199).
//
// The union of overlapping voxels comes from one member mask per axis and
// coordinate (N <= 32): a cell's members are the AND of its coordinates' masks,
// so each voxel's entries come out in ascending group order and the float32 sums
// are deterministic.
//
// What bounds it: the instructions issued (78 % of the issue slots at 16 members
// of 8x8), half of them in the exact variance's products; memory stays below 10 %.
#include <cuda_runtime.h>
#include <stdint.h>

#include "bmnd_common.cuh"

namespace bmnd {
namespace {

constexpr int kThreads = 256;      // threads per group (CTA)
constexpr int kMiscWild = 13;      // misc word: the group holds a value of 1e30 or more, an infinity or NaN

// Shared-memory plan.  A fixed part holds the group matrix, the transform
// tables, positions and small per-group arrays.  The union region first holds
// the exact-variance phase's axis masks and union-voxel lists; once that
// phase is done it holds the group buffers: S (noise sigma), X (noisy
// coefficients) and R (pilot coefficients, Wiener) or V (attenuation, hard
// thresholding).  Transforms run in place, so no scratch buffer is needed.
// With exact risk weights the union-voxel lists are still needed after the
// shrinkage, so they get a region of their own after the group buffers.
struct Layout {
    // byte offsets into dynamic shared memory
    int64_t g, gt2, fw, fi, fit, dir, win, mdiag, voff, kron, pos, org0, shf, shl, sg, ex, part, lag, uni, s, x, r, v, grid, lval,
        lstart, lent, scan, plane, wts, misc, risk, total;
    int32_t part_over;  // the exact phase's partial sums overwrite its lists
    int32_t kron_used;  // S^T is copied to `kron`
};

struct FilterArgs {
    BmndStageParams sp;
    Layout L;
    int32_t P;
    int32_t nmax;
    int32_t kmax;
    int32_t counts[BMND_MAX_DIMS];
    int64_t vstride[BMND_MAX_DIMS];
    const float* noisy;
    const float* pilot;
    const int32_t* sel;
    const int32_t* count;
    int64_t n_refs;
    double* num;
    double* den;
    const float* st;  // S^T: st[p * kron_stride(P) + j] = S[j, p], the Kronecker product of the patch transforms
    double* sig_num;  // optional: sigma-map numerator (sum of sigma x weight x window), else null
    // group-mass conservation, second pass: the first pass's denominator
    // (read only); the kernel then re-aggregates the numerator alone
    const double* den_ro;
    int* err;  // 1: a group's mass correction is undefined; 2: a group was skipped (bad members)
    // group probe: per-group intermediate arrays instead of the aggregation
    GroupProbe probe;
    int64_t n_lins;      // patch-grid positions: a member's lin lies in [0, n_lins)
    int64_t ucells_cap;  // union-box cells the layout's lists hold
    AggStore store;      // deterministic aggregation: rows of the entry store, or store.store == null
};

// Whether launch_group_filter takes an instantiation for the patch shape
__host__ inline bool specialised_shape(const BmndStageParams& sp) {
    const int32_t* b = sp.block;
    if (sp.exact_risk_weights) return false;
    if (sp.ndim == 2) return b[0] == 8 && b[1] == 8;
    return sp.ndim == 3 && b[0] == b[1] && b[0] == b[2] && (b[0] == 4 || b[0] == 5);
}
// S^T of patches of 33-64 voxels (16 KB) lies in shared memory for the Haar form
// of the exact phase (exact_haar), which reads it with 32-bit addresses and no L1
// tags; the other forms read the table in global memory, so a copy would only
// take residency (8x8 patches of a 384 x 416 image, 16 exact planes: stage 1 takes
// 8.2 ms without it, 10.6 with it; stage 2 18.0 against 20.8)
__host__ inline bool kron_in_smem(const BmndStageParams& sp, int P, int kmax) {
    return specialised_shape(sp) && kron_jr(P) == 2 && kmax > 0 && sp.variance_k <= 4 &&
           sp.noise_model == BMND_NOISE_POISSON && sp.group_transform == BMND_GROUP_HAAR;
}

// The group buffers (S, X, R, V, SG) of 8x8 patches keep one spare word after
// every row: the lines of the last axis, 8 words apart, then fall into different
// banks (8-way conflicts before; with the joint forward sweep below, a 17 K-group
// final stage of 32 members went from 3.12 to 2.89 ms).  4x4x4 patches conflict
// 4-way at most and measured the same with and without the padding (3.56 ms), so
// they have none.  LB is the row length.
template <int LB>
__host__ __device__ __forceinline__ constexpr int padded(int p) {
    return LB == 8 ? p + p / 8 : p;
}
__host__ inline int64_t padded_patch(const BmndStageParams& sp, int P) {
    return sp.ndim == 2 && specialised_shape(sp) ? padded<8>(P) : P;
}

// exact planes' G entries in pairs (g, g) for packed products
__host__ inline int64_t pair_bytes(int nmax, int kmax) {
    return kmax > 0 ? 8 * static_cast<int64_t>(nmax) * ((kmax + 3) / 4 * 4) : 16;
}

// `early`: the pairs have a place of their own; else one that the group buffers, or
// hard thresholding's sigmas, take after the exact variance
__host__ Layout layout_of(const BmndStageParams& sp, int P, int nmax, int kmax, int64_t ucells, bool sigma, bool early) {
    Layout L{};
    int64_t off = 0;
    auto round16 = [](int64_t b) { return (b + 15) & ~int64_t(15); };
    auto take = [&](int64_t bytes) {
        int64_t o = off;
        off += round16(bytes);
        return o;
    };
    const int64_t np = static_cast<int64_t>(nmax) * P;
    const int64_t npp = static_cast<int64_t>(nmax) * padded_patch(sp, P);
    const bool wiener = sp.filter == BMND_FILTER_WIENER;
    const bool gauss = sp.noise_model == BMND_NOISE_GAUSSIAN;
    const bool keep = sp.exact_risk_weights != 0;
    const int64_t gt2_bytes = pair_bytes(nmax, kmax);
    L.g = take(4 * nmax * nmax);
    if (early) L.gt2 = take(gt2_bytes);
    L.fw = take(4 * BMND_MAX_DIMS * BMND_MAX_EDGE * BMND_MAX_EDGE);
    L.fi = take(4 * BMND_MAX_DIMS * BMND_MAX_EDGE * BMND_MAX_EDGE);
    // group-mass conservation: transposed inverse spatial matrices, and the
    // per-axis factors of the constant synthesis direction (group axis, patch axes)
    const bool mass = sp.mass_conserve != 0;
    L.fit = take(mass ? 4 * BMND_MAX_DIMS * BMND_MAX_EDGE * BMND_MAX_EDGE : 16);
    L.dir = take(mass ? 4 * (BMND_MAX_STACK + BMND_MAX_DIMS * BMND_MAX_EDGE) : 16);
    L.win = take(4 * P);
    L.mdiag = take(sp.windowed_synthesis ? 8 * P : 16);
    L.voff = take(4 * P);
    L.kron_used = kron_in_smem(sp, P, kmax);
    L.kron = take(L.kron_used ? 4 * static_cast<int64_t>(P) * kron_stride(P) : 16);
    L.pos = take(4 * nmax * BMND_MAX_DIMS);
    L.org0 = take(4 * nmax);
    L.shf = take(4 * nmax * BMND_MAX_DIMS);
    L.shl = take(4 * nmax);
    // hard thresholding with a sigma map keeps each coefficient's sigma until the scatter
    const int64_t sg_bytes = sigma && !wiener ? 4 * npp : 16;
    L.sg = take(sg_bytes);
    L.ex = take(4 * static_cast<int64_t>(kmax) * P);

    L.scan = take(8 * (kThreads / 32 + 1));  // the warps' totals, then the block's
    L.plane = take(8 * (nmax > 40 ? nmax : 40));  // also the mass phase's 8 warps x 5 sums
    L.wts = take(4 * nmax);
    L.misc = take(64);
    L.risk = take(8 * (kThreads / 32 + 1));  // exact risk: per-warp partial sums, then the total
    // union region
    L.uni = off;
    int64_t lists = L.uni;
    if (!early) {
        L.gt2 = sg_bytes >= gt2_bytes ? L.sg : lists;
        if (L.gt2 == lists) lists += round16(gt2_bytes);
    }
    const int64_t buf = round16(4 * npp);
    L.s = L.uni;
    L.x = L.s + buf;
    L.r = L.x + buf;  // Wiener: pilot coefficients, then the attenuation
    L.v = L.r;        // hard thresholding: the attenuation
    // Gaussian noise: covariance-map row of every member pair (i > j), needed
    // before R or V is, in their place where they are large enough
    const int64_t lag_bytes = gauss && kmax > 0 ? 4 * static_cast<int64_t>(nmax) * ((nmax + 3) / 4 * 4) : 0;
    L.lag = L.r;
    const int64_t group_bytes = 2 * buf + (buf > lag_bytes ? buf : round16(lag_bytes));
    // union-voxel lists of the exact phase (Poisson noise, or white Gaussian
    // noise with exact risk weights), kept apart from the group buffers when
    // the exact risk reads them after the shrinkage
    const int kl = (gauss && !keep) ? 0 : kmax;
    const int64_t umax = kl > 0 ? (np < ucells ? np : ucells) : 0;
    // member masks per union coordinate of every axis: a union box of at most
    // ucells cells has at most ucells / prod(other patch edges) along an axis
    int64_t axis_masks = 0;
    for (int d = 0; d < sp.ndim; ++d) {
        const int64_t most = ucells * sp.block[d] / P;
        axis_masks += most < sp.shape[d] ? most : sp.shape[d];
    }
    // exact variance: per-warp partial sums of one tile of 4 planes x 32 JR
    // coefficients, added in warp order afterwards.  They take the group buffers'
    // place, as the lists do, behind them; with a single tile (k <= 4 and P <= its
    // width: the default profiles) the lists are done with by then and give
    // theirs.  (Apart from the union region they made 8x8x8 patches at the default
    // stack of 32 need 233 728 bytes, above the limit of 232 448; so, 216 304.)
    if (keep) lists = L.uni + group_bytes;
    L.grid = lists;
    L.lval = L.grid + round16(kl > 0 ? 4 * axis_masks : 0);
    L.lstart = L.lval + round16(4 * umax);
    L.lent = L.lstart + round16(4 * (umax + 1));
    int64_t end = L.lent + round16(kl > 0 ? 4 * (np + 2) : 0);
    const int tile_w = 32 * kron_jr(P);
    const int64_t part_bytes = !gauss && kmax > 0 ? 4 * (kThreads / 32) * 4 * static_cast<int64_t>(tile_w) : 0;
    L.part_over = !keep && kmax <= 4 && P <= tile_w;
    L.part = L.part_over ? L.grid : end;
    if (end < L.part + part_bytes) end = L.part + part_bytes;
    off = end > L.uni + group_bytes ? end : L.uni + group_bytes;
    L.total = off;
    return L;
}

// The exact risk reads the pairs after the shrinkage, so there they keep a place of
// their own, and in the specialised shapes, which are far from the limit; the
// entries' 16-bit offsets must reach them.
__host__ Layout make_layout(const BmndStageParams& sp, int P, int nmax, int kmax, int64_t ucells, bool sigma) {
    if (!sp.exact_risk_weights && !specialised_shape(sp)) {
        const Layout L = layout_of(sp, P, nmax, kmax, ucells, sigma, false);
        if (L.gt2 + pair_bytes(nmax, kmax) <= 0x10000) return L;
    }
    return layout_of(sp, P, nmax, kmax, ucells, sigma, true);
}

template <bool V>
struct BoolTag {
    static constexpr bool value = V;
};

template <typename T>
__device__ __forceinline__ T* sm(unsigned char* base, int64_t off) {
    return reinterpret_cast<T*>(base + off);
}

// Patch geometry: compile-time for the default shapes (ND > 0), runtime otherwise.
template <int ND, int B0, int B1, int B2>
struct Geom {
    int nd_, b_[BMND_MAX_DIMS], P_;
    __device__ explicit Geom(const BmndStageParams& sp) {
        nd_ = sp.ndim;
        P_ = 1;
        for (int d = 0; d < BMND_MAX_DIMS; ++d) {
            b_[d] = d < sp.ndim ? sp.block[d] : 1;
            P_ *= b_[d];
        }
    }
    __device__ __forceinline__ int nd() const { return ND > 0 ? ND : nd_; }
    __device__ __forceinline__ int b(int d) const {
        if (ND > 0) return d == 0 ? B0 : (d == 1 ? B1 : B2);
        return b_[d];
    }
    __device__ __forceinline__ int P() const { return ND > 0 ? B0 * B1 * B2 : P_; }
    // group buffers: words per member, and the word of patch element p
    static constexpr int LB = ND == 0 ? 0 : (ND == 3 ? B2 : (ND == 2 ? B1 : B0));
    __device__ __forceinline__ int PP() const { return ND > 0 ? padded<LB>(B0 * B1 * B2) : P_; }
    __device__ __forceinline__ int at(int g, int p) const { return g * PP() + padded<LB>(p); }
    // f(member, patch element, its word) over an n x P group
    template <typename F>
    __device__ __forceinline__ void each(int n, F f) const {
        for (int e = threadIdx.x; e < n * P(); e += blockDim.x) {
            const int g = e / P(), p = e - g * P();
            f(g, p, at(g, p));
        }
    }
    // product of the patch extents after axis d
    __device__ __forceinline__ int inner(int d) const {
        int v = 1;
#pragma unroll
        for (int e = 0; e < BMND_MAX_DIMS; ++e)
            if (e > d && e < nd()) v *= b(e);
        return v;
    }
    // voxel offset of element p of the patch whose origin is `org`
    __device__ __forceinline__ int64_t offset(const int* org, int p, const int64_t* vstride) const {
        int64_t off = 0;
#pragma unroll
        for (int d = BMND_MAX_DIMS - 1; d >= 0; --d) {
            if (d < nd()) {
                off += static_cast<int64_t>(org[d] + p % b(d)) * vstride[d];
                p /= b(d);
            }
        }
        return off;
    }
};

// Transforms work in place on an (n, block...) group held in shared memory.
// Every axis product accumulates with one fused multiply-add per term in k
// order, which is how NumPy's sgemm evaluates the reference's products.
//
// Group axis, compile-time size N: out[i, p] = sum_k M[i, k] in[k, p] with
// KIND 0: M = G, KIND 1: M = G^T (the inverse, transforms.py:423, :436),
// KIND 2: M = G o G with each entry rounded as fl(g * g) (the squared
// transform of the variance propagation).  Each thread holds one column in
// registers and produces IC of its N outputs; a round takes whole columns
// (all their chunks) and reads them completely before any thread writes, so
// the product can overwrite its input.  blockDim.x must be a multiple of
// 32 * CH so that each warp holds a single chunk.
template <int KIND>
__device__ __forceinline__ float gmat(const float* G, int N, int i, int k) {
    float m = KIND == 1 ? G[k * N + i] : G[i * N + k];
    return KIND == 2 ? mul_rn(m, m) : m;
}

// (C columns of S words per member, column p at padded<LB>(p))
template <int N, int KIND, int LB>
__device__ void group_axis_inplace(float* buf, int C, int S, const float* G) {
    constexpr int IC = N >= 16 ? 8 : N;  // outputs per thread
    constexpr int CH = N / IC;           // threads per column
    // a warp shares one output chunk over 32 consecutive columns: matrix reads
    // are broadcasts, column reads and writes hit consecutive banks
    const int cols = static_cast<int>(blockDim.x) / CH;
    for (int c0 = 0; c0 < C; c0 += cols) {
        const int col = c0 + static_cast<int>(threadIdx.x) % cols;
        const int i0 = (static_cast<int>(threadIdx.x) / cols) * IC;
        const bool act = static_cast<int>(threadIdx.x) < cols * CH && col < C;
        const int p = padded<LB>(col);
        float x[N];
        if (act) {
#pragma unroll
            for (int k = 0; k < N; ++k) x[k] = buf[k * S + p];
        }
        __syncthreads();
        if (act) {
#pragma unroll
            for (int ii = 0; ii < IC; ++ii) {
                const int i = i0 + ii;
                float acc = 0.0f;
                if (KIND != 1 && N % 4 == 0) {
#pragma unroll
                    for (int k = 0; k < N; k += 4) {
                        float4 m = *reinterpret_cast<const float4*>(G + i * N + k);
                        if (KIND == 2) {
                            m.x = mul_rn(m.x, m.x);
                            m.y = mul_rn(m.y, m.y);
                            m.z = mul_rn(m.z, m.z);
                            m.w = mul_rn(m.w, m.w);
                        }
                        acc = fmaf(m.x, x[k], acc);
                        acc = fmaf(m.y, x[k + 1], acc);
                        acc = fmaf(m.z, x[k + 2], acc);
                        acc = fmaf(m.w, x[k + 3], acc);
                    }
                } else {
#pragma unroll
                    for (int k = 0; k < N; ++k) acc = fmaf(gmat<KIND>(G, N, i, k), x[k], acc);
                }
                buf[i * S + p] = acc;
            }
        }
        __syncthreads();
    }
}

// Haar group axis of a power-of-two size N as the matrix product above without
// its zero entries: row 0 and row 1 are dense, the 2^(l-1) rows of level l reach
// N / 2^(l-1) columns each, so a column takes log2(N) + 1 multiply-adds per
// output instead of N.  Leaving out fma(0, x, acc) = acc keeps every result's
// bits for finite x (the caller checks).  C is the chunk of 8 outputs a warp
// takes; entry values come from the matrix, so their rounding is its own.
template <int N, int KIND, int C>
__device__ __forceinline__ void haar_chunk(const float* buf, int P, int p, const float* G,
                                           float (&acc)[N >= 16 ? 8 : N]) {
    constexpr int IC = N >= 16 ? 8 : N;
    constexpr int i0 = C * IC;
    {
        if constexpr (KIND == 1) {
            // out[g] = sum over rows k whose support holds g, ascending
            constexpr int LV = N >= 32 ? 5 : (N >= 16 ? 4 : (N >= 8 ? 3 : (N >= 4 ? 2 : 1)));
            const float x0 = buf[p], m0 = G[0];
#pragma unroll
            for (int ii = 0; ii < IC; ++ii) acc[ii] = fmaf(m0, x0, 0.0f);
#pragma unroll
            for (int l = 0; l < LV; ++l) {
                const int w = N >> l;  // support width of the 2^l rows of this level
#pragma unroll
                for (int j = 0; j < (1 << l); ++j) {
                    const int k = (1 << l) + j, b = j * w;
                    if (b < i0 + IC && b + w > i0) {
                        const float x = buf[k * P + p], m = G[k * N + b];
#pragma unroll
                        for (int ii = 0; ii < IC; ++ii) {
                            const int g = i0 + ii;
                            if (g >= b && g < b + w) acc[ii] = fmaf(g < b + w / 2 ? m : -m, x, acc[ii]);
                        }
                    }
                }
            }
        } else {
            float x[N];  // the columns this chunk's rows reach
#pragma unroll
            for (int k = 0; k < N; ++k) {
                bool used = false;
#pragma unroll
                for (int ii = 0; ii < IC; ++ii) {
                    const int i = i0 + ii;
                    const int top = i == 0 ? 1 : (i < 2 ? 1 : (i < 4 ? 2 : (i < 8 ? 4 : (i < 16 ? 8 : 16))));
                    const int w = N / top, b = i == 0 ? 0 : (i - top) * w;
                    used = used || (k >= b && k < b + w);
                }
                if (used) x[k] = buf[k * P + p];
            }
#pragma unroll
            for (int ii = 0; ii < IC; ++ii) {
                const int i = i0 + ii;
                const int top = i < 2 ? 1 : (i < 4 ? 2 : (i < 8 ? 4 : (i < 16 ? 8 : 16)));
                const int w = N / top, b = i == 0 ? 0 : (i - top) * w;
                float m = G[i * N + b];
                if (KIND == 2) m = mul_rn(m, m);
                float t = 0.0f;
#pragma unroll
                for (int k = 0; k < N; ++k)
                    if (k >= b && k < b + w) t = fmaf(KIND == 2 || i == 0 || k < b + w / 2 ? m : -m, x[k], t);
                acc[ii] = t;
            }
        }
    }
}

template <int N, int KIND>
__device__ __forceinline__ void haar_chunk_any(int chunk, const float* buf, int S, int p, const float* G,
                                               float (&acc)[N >= 16 ? 8 : N]) {
    constexpr int CH = N / (N >= 16 ? 8 : N);
    if (CH == 1 || chunk == 0) haar_chunk<N, KIND, 0>(buf, S, p, G, acc);
    else if (CH == 2 || chunk == 1) haar_chunk<N, KIND, (CH > 1 ? 1 : 0)>(buf, S, p, G, acc);
    else if (chunk == 2) haar_chunk<N, KIND, (CH > 2 ? 2 : 0)>(buf, S, p, G, acc);
    else haar_chunk<N, KIND, (CH > 3 ? 3 : 0)>(buf, S, p, G, acc);
}

template <int N, int KIND, int LB>
__device__ void haar_product(float* buf, int C, int S, const float* G) {
    constexpr int IC = N >= 16 ? 8 : N;
    constexpr int CH = N / IC;
    const int cols = static_cast<int>(blockDim.x) / CH;
    const int chunk = static_cast<int>(threadIdx.x) / cols;  // the same for a whole warp
    for (int c0 = 0; c0 < C; c0 += cols) {
        const int col = c0 + static_cast<int>(threadIdx.x) % cols;
        const bool act = static_cast<int>(threadIdx.x) < cols * CH && col < C;
        const int p = padded<LB>(col);
        float acc[IC];
        if (act) haar_chunk_any<N, KIND>(chunk, buf, S, p, G, acc);
        __syncthreads();
        if (act) {
#pragma unroll
            for (int ii = 0; ii < IC; ++ii) buf[(chunk * IC + ii) * S + p] = acc[ii];
        }
    }
    __syncthreads();  // (the columns of one round are not read by the next)
}

// The forward Haar axis of all the group's buffers in one sweep: s squared (kind
// 2), x and, unless null, r (kind 0).  Two small buffers (hard thresholding of
// at most 16 members and 64 columns) are taken by half of the threads each.
template <int N, int LB>
__device__ void haar_product_all(float* s, float* x, float* r, int C, int S, const float* G) {
    constexpr int IC = N >= 16 ? 8 : N;
    constexpr int CH = N / IC;
    const int tid = threadIdx.x;
    if (r == nullptr && CH <= 2 && C <= 64 && blockDim.x == 256) {
        const bool second = tid >= 128;
        const int t = tid & 127;
        constexpr int cols = 128 / (CH <= 2 ? CH : 2);
        const int chunk = t / cols, col = t % cols;
        const bool act = col < C;
        const int p = padded<LB>(col);
        float acc[IC];
        if (act) {
            if (second) haar_chunk_any<N, 0>(chunk, x, S, p, G, acc);
            else haar_chunk_any<N, 2>(chunk, s, S, p, G, acc);
        }
        __syncthreads();
        if (act) {
            float* buf = second ? x : s;
#pragma unroll
            for (int ii = 0; ii < IC; ++ii) buf[(chunk * IC + ii) * S + p] = acc[ii];
        }
        __syncthreads();
        return;
    }
    const int cols = static_cast<int>(blockDim.x) / CH;
    const int chunk = tid / cols;
    for (int c0 = 0; c0 < C; c0 += cols) {
        const int col = c0 + tid % cols;
        const bool act = tid < cols * CH && col < C;
        const int p = padded<LB>(col);
        float as[IC], ax[IC], ar[IC];
        if (act) {
            haar_chunk_any<N, 2>(chunk, s, S, p, G, as);
            haar_chunk_any<N, 0>(chunk, x, S, p, G, ax);
            if (r) haar_chunk_any<N, 0>(chunk, r, S, p, G, ar);
        }
        __syncthreads();
        if (act) {
#pragma unroll
            for (int ii = 0; ii < IC; ++ii) {
                const int e = (chunk * IC + ii) * S + p;
                s[e] = as[ii];
                x[e] = ax[ii];
                if (r) r[e] = ar[ii];
            }
        }
    }
    __syncthreads();
}

// Haar group axis by its sum pyramid (one thread per column, O(N) operations):
// row (l, j) of the orthonormal Haar matrix, block width w = N / 2^(l-1), is
// (first-half sum - second-half sum) / sqrt(w); its elementwise square gives the
// block sum / w; the inverse adds and subtracts the detail down the pyramid.
// The rounding differs from the matrix product, so only the fast path uses it.
template <int N, int KIND>
__device__ __forceinline__ void haar_column(float* buf, int p, int P) {
    {
        float x[N];
#pragma unroll
        for (int k = 0; k < N; ++k) x[k] = buf[k * P + p];
        float out[N];
        if (KIND == 1) {
            // x = H^T c: start from the DC, refine block by block
            out[0] = x[0] * rsqrtf(static_cast<float>(N));
#pragma unroll
            for (int w = N; w >= 2; w >>= 1) {
                const int nb = N / w;
                const float sc = rsqrtf(static_cast<float>(w));
#pragma unroll
                for (int j = nb - 1; j >= 0; --j) {
                    const float d = x[nb + j] * sc;
                    const float a = out[j];
                    out[2 * j + 1] = a - d;
                    out[2 * j] = a + d;
                }
            }
        } else {
            float sm_[N];
#pragma unroll
            for (int k = 0; k < N; ++k) sm_[k] = x[k];
#pragma unroll
            for (int w = 2; w <= N; w <<= 1) {
                const int nb = N / w;
                const float sc = KIND == 2 ? 1.0f / static_cast<float>(w) : rsqrtf(static_cast<float>(w));
#pragma unroll
                for (int j = 0; j < nb; ++j) {
                    const float a = sm_[2 * j], b = sm_[2 * j + 1];
                    out[nb + j] = (KIND == 2 ? a + b : a - b) * sc;
                    sm_[j] = a + b;
                }
            }
            out[0] = sm_[0] * (KIND == 2 ? 1.0f / static_cast<float>(N) : rsqrtf(static_cast<float>(N)));
        }
#pragma unroll
        for (int k = 0; k < N; ++k) buf[k * P + p] = out[k];
    }
}

template <int N, int KIND, int LB>
__device__ void haar_axis_fast(float* buf, int C, int S) {
    for (int c = static_cast<int>(threadIdx.x); c < C; c += blockDim.x) haar_column<N, KIND>(buf, padded<LB>(c), S);
    __syncthreads();
}

// the forward Haar group axis of three groups in one sweep: s squared (kind
// 2), x and r (kind 0; r may be null)
template <int N, int LB>
__device__ void haar_axis_fast3(float* s, float* x, float* r, int C, int S) {
    for (int c = static_cast<int>(threadIdx.x); c < C; c += blockDim.x) {
        const int p = padded<LB>(c);
        haar_column<N, 2>(s, p, S);
        haar_column<N, 0>(x, p, S);
        if (r) haar_column<N, 0>(r, p, S);
    }
    __syncthreads();
}

template <int LB>
__device__ bool haar_axis_any3(float* s, float* x, float* r, int n, int C, int S) {
    switch (n) {
        case 2: haar_axis_fast3<2, LB>(s, x, r, C, S); return true;
        case 4: haar_axis_fast3<4, LB>(s, x, r, C, S); return true;
        case 8: haar_axis_fast3<8, LB>(s, x, r, C, S); return true;
        case 16: haar_axis_fast3<16, LB>(s, x, r, C, S); return true;
        case 32: haar_axis_fast3<32, LB>(s, x, r, C, S); return true;
        default: return false;
    }
}

template <int KIND, int LB>
__device__ bool haar_axis_any(float* buf, int n, int C, int S) {
    switch (n) {
        case 2: haar_axis_fast<2, KIND, LB>(buf, C, S); return true;
        case 4: haar_axis_fast<4, KIND, LB>(buf, C, S); return true;
        case 8: haar_axis_fast<8, KIND, LB>(buf, C, S); return true;
        case 16: haar_axis_fast<16, KIND, LB>(buf, C, S); return true;
        case 32: haar_axis_fast<32, KIND, LB>(buf, C, S); return true;
        default: return false;
    }
}

// runtime group size (not a power of two): one thread per column
template <int KIND, int LB>
__device__ void group_axis_generic(float* buf, int n, int C, int S, const float* G) {
    for (int c = static_cast<int>(threadIdx.x); c < C; c += blockDim.x) {
        const int p = padded<LB>(c);
        float x[BMND_MAX_STACK];
        for (int k = 0; k < n; ++k) x[k] = buf[k * S + p];
        for (int i = 0; i < n; ++i) {
            float acc = 0.0f;
            for (int k = 0; k < n; ++k) acc = fmaf(gmat<KIND>(G, n, i, k), x[k], acc);
            buf[i * S + p] = acc;
        }
    }
    __syncthreads();
}

// `sparse`: G is the Haar matrix and every value is finite
template <int KIND, int LB>
__device__ void group_axis_any(float* buf, int n, int C, int S, const float* G, bool sparse) {
    if (sparse) {
        switch (n) {
            case 2: haar_product<2, KIND, LB>(buf, C, S, G); return;
            case 4: haar_product<4, KIND, LB>(buf, C, S, G); return;
            case 8: haar_product<8, KIND, LB>(buf, C, S, G); return;
            case 16: haar_product<16, KIND, LB>(buf, C, S, G); return;
            case 32: haar_product<32, KIND, LB>(buf, C, S, G); return;
            default: break;
        }
    }
    switch (n) {
        case 1: group_axis_inplace<1, KIND, LB>(buf, C, S, G); break;
        case 2: group_axis_inplace<2, KIND, LB>(buf, C, S, G); break;
        case 4: group_axis_inplace<4, KIND, LB>(buf, C, S, G); break;
        case 8: group_axis_inplace<8, KIND, LB>(buf, C, S, G); break;
        case 16: group_axis_inplace<16, KIND, LB>(buf, C, S, G); break;
        case 32: group_axis_inplace<32, KIND, LB>(buf, C, S, G); break;
        default: group_axis_generic<KIND, LB>(buf, n, C, S, G); break;
    }
}

// patch axis d with compile-time edge B and INNER elements after it: each thread
// transforms whole lines of B values (matrix in registers), so lines never
// share a thread and the product overwrites its input.  line_base and kStep are
// a line's first word and its element stride in the padded buffers.
template <int B, int STEP>
__device__ __forceinline__ void space_line(float* buf, int base, const float (&m)[B * B]) {
    float x[B];
#pragma unroll
    for (int k = 0; k < B; ++k) x[k] = buf[base + k * STEP];
#pragma unroll
    for (int i = 0; i < B; ++i) {
        float acc = 0.0f;
#pragma unroll
        for (int k = 0; k < B; ++k) acc = fmaf(m[i * B + k], x[k], acc);
        buf[base + i * STEP] = acc;
    }
}

template <int B, int INNER, int LB>
struct Lines {
    static constexpr int kStep = INNER == 1 ? 1 : padded<LB>(INNER);
    __device__ static __forceinline__ int base(int line) {
        const int o = line / INNER;
        const int t = line - o * INNER;
        return INNER == 1 ? padded<LB>(o * B) : o * B * kStep + padded<LB>(t);
    }
};

// Edge 8: two threads of a warp (lanes l and l + 16) share a line, four outputs
// each, so that a half of the matrix, 32 registers instead of 64, stays in a
// thread and 16 members keep all warps of the block busy.
template <int INNER, int LB>
__device__ __forceinline__ void space_axis_half(float* buf, int lines, const float (&m)[32]) {
    using L = Lines<8, INNER, LB>;
    const int lane = threadIdx.x & 31, h = lane >> 4;
    for (int l0 = 0; l0 < lines; l0 += blockDim.x >> 1) {
        const int line = l0 + (static_cast<int>(threadIdx.x) >> 5) * 16 + (lane & 15);
        const int base = L::base(line);
        float x[8];
        if (line < lines) {
#pragma unroll
            for (int k = 0; k < 8; ++k) x[k] = buf[base + k * L::kStep];
        }
        __syncwarp();
        if (line < lines) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                float acc = 0.0f;
#pragma unroll
                for (int k = 0; k < 8; ++k) acc = fmaf(m[i * 8 + k], x[k], acc);
                buf[base + (h * 4 + i) * L::kStep] = acc;
            }
        }
    }
}

// one axis of one buffer (`square`: by the squared matrix) ...
template <int B, int INNER, int LB>
__device__ void space_axis_reg(float* buf, int lines, const float* Msrc, bool square) {
    constexpr int kRows = B == 8 ? 4 : B;
    const int row0 = B == 8 ? (threadIdx.x >> 4 & 1) * 4 : 0;
    float m[kRows * B];
#pragma unroll
    for (int q = 0; q < kRows * B; ++q) {
        const float v = Msrc[row0 * B + q];
        m[q] = square ? mul_rn(v, v) : v;
    }
    if constexpr (B == 8) {
        space_axis_half<INNER, LB>(buf, lines, m);
    } else {
        using L = Lines<B, INNER, LB>;
        for (int line = threadIdx.x; line < lines; line += blockDim.x)
            space_line<B, L::kStep>(buf, L::base(line), m);
    }
    __syncthreads();
}

// ... and of all the group's buffers in one sweep: s by the squared matrix, x and
// r (may be null) by the matrix itself; up to 128 lines of two buffers are taken
// by half of the threads each
template <int B, int INNER, int LB>
__device__ void space_axis_reg_all(float* s, float* x, float* r, int lines, const float* Msrc) {
    const int tid = threadIdx.x;
    constexpr int kRows = B == 8 ? 4 : B;
    const int row0 = B == 8 ? (tid >> 4 & 1) * 4 : 0;
    float m[kRows * B];
#pragma unroll
    for (int q = 0; q < kRows * B; ++q) m[q] = Msrc[row0 * B + q];
    if constexpr (B == 8) {
        space_axis_half<INNER, LB>(x, lines, m);
        if (r) space_axis_half<INNER, LB>(r, lines, m);
#pragma unroll
        for (int q = 0; q < kRows * B; ++q) m[q] = mul_rn(m[q], m[q]);
        space_axis_half<INNER, LB>(s, lines, m);
    } else {
        using L = Lines<B, INNER, LB>;
        const int half = blockDim.x >> 1;
        const bool split = r == nullptr && lines <= half;
        const int step = split ? half : static_cast<int>(blockDim.x);
        if (!split || tid >= half) {
            for (int line = split ? tid - half : tid; line < lines; line += step) {
                const int base = L::base(line);
                space_line<B, L::kStep>(x, base, m);
                if (r) space_line<B, L::kStep>(r, base, m);
            }
        }
        if (!split || tid < half) {
#pragma unroll
            for (int q = 0; q < B * B; ++q) m[q] = mul_rn(m[q], m[q]);
            for (int line = tid; line < lines; line += step) space_line<B, L::kStep>(s, L::base(line), m);
        }
    }
    __syncthreads();
}

// runtime geometry: one thread per line of edge m along axis d
template <class GM>
__device__ void space_axis_generic(const GM& geo, int d, float* buf, int n, const float* M, bool square) {
    const int m = geo.b(d);
    const int inner = geo.inner(d);
    const int lines = n * geo.P() / m;
    for (int line = static_cast<int>(threadIdx.x); line < lines; line += blockDim.x) {
        const int o = line / inner;
        const int t = line - o * inner;
        const int base = o * m * inner + t;
        float x[BMND_MAX_EDGE];
        for (int k = 0; k < m; ++k) x[k] = buf[base + k * inner];
        for (int i = 0; i < m; ++i) {
            float acc = 0.0f;
            for (int k = 0; k < m; ++k) {
                float mk = M[i * m + k];
                if (square) mk = mul_rn(mk, mk);
                acc = fmaf(mk, x[k], acc);
            }
            buf[base + i * inner] = acc;
        }
    }
    __syncthreads();
}

template <int ND, int B0, int B1, int B2, int D>
struct Axis {
    static constexpr int B = D == 0 ? B0 : (D == 1 ? B1 : B2);
    static constexpr int INNER = D == 0 ? (ND > 1 ? B1 : 1) * (ND > 2 ? B2 : 1) : (D == 1 ? (ND > 2 ? B2 : 1) : 1);
    static constexpr int LB = ND == 3 ? B2 : (ND == 2 ? B1 : B0);
    static constexpr int kLines = B0 * B1 * B2 / B;
};
template <int ND, int B0, int B1, int B2, int D>
__device__ __forceinline__ void space_axis_fixed(float* buf, int n, const float* M, bool square) {
    using A = Axis<ND, B0, B1, B2, D>;
    space_axis_reg<A::B, A::INNER, A::LB>(buf, n * A::kLines, M, square);
}

template <int ND, int B0, int B1, int B2, int D>
__device__ __forceinline__ void space_axis_fixed_all(float* s, float* x, float* r, int n, const float* M) {
    using A = Axis<ND, B0, B1, B2, D>;
    space_axis_reg_all<A::B, A::INNER, A::LB>(s, x, r, n * A::kLines, M);
}

// separable transform of an (n, block...) group in place: the group axis
// first, then the patch axes (transforms.py:209-255).  kind: 0 forward,
// 1 inverse, 2 squared forward, 3 transposed inverse (poisson.py:84-114).
template <int ND, int B0, int B1, int B2, class GM>
__device__ void transform_group(const GM& geo, const FilterArgs& a, unsigned char* smem, int n, float* buf,
                                int kind) {
    const float* G = sm<float>(smem, a.L.g);
    const float* F = sm<float>(smem, kind == 1 ? a.L.fi : (kind == 3 ? a.L.fit : a.L.fw));
    const bool fast_haar = a.sp.fast_group_transform && a.sp.group_transform == BMND_GROUP_HAAR &&
                           (kind == 0 ? haar_axis_any<0, GM::LB>(buf, n, geo.P(), geo.PP())
                                      : kind == 1 ? haar_axis_any<1, GM::LB>(buf, n, geo.P(), geo.PP())
                                                  : kind == 2 ? haar_axis_any<2, GM::LB>(buf, n, geo.P(), geo.PP())
                                                              : haar_axis_any<0, GM::LB>(buf, n, geo.P(), geo.PP()));
    if (!fast_haar && a.sp.group_transform != BMND_GROUP_NONE) {
        // kind 3 (transposed inverse): the group transforms are orthonormal, so
        // the transposed inverse of the group axis is the forward transform
        const bool sparse = a.sp.group_transform == BMND_GROUP_HAAR && kind != 3 && !a.den_ro &&
                            sm<int>(smem, a.L.misc)[kMiscWild] == 0;
        if (kind == 0 || kind == 3) group_axis_any<0, GM::LB>(buf, n, geo.P(), geo.PP(), G, sparse);
        else if (kind == 1) group_axis_any<1, GM::LB>(buf, n, geo.P(), geo.PP(), G, sparse);
        else group_axis_any<2, GM::LB>(buf, n, geo.P(), geo.PP(), G, sparse);
    }
    const bool square = kind == 2;
    if constexpr (ND > 0) {
        space_axis_fixed<ND, B0, B1, B2, 0>(buf, n, F, square);
        if constexpr (ND > 1) space_axis_fixed<ND, B0, B1, B2, 1>(buf, n, F + BMND_MAX_EDGE * BMND_MAX_EDGE, square);
        if constexpr (ND > 2)
            space_axis_fixed<ND, B0, B1, B2, 2>(buf, n, F + 2 * BMND_MAX_EDGE * BMND_MAX_EDGE, square);
    } else {
        for (int d = 0; d < geo.nd(); ++d)
            space_axis_generic(geo, d, buf, n, F + d * BMND_MAX_EDGE * BMND_MAX_EDGE, square);
    }
}

// The forward transforms of all the group's buffers in one sweep of passes: the
// variance group S squared (kind 2), the observation X and the pilot R (kind 0,
// R may be null): a barrier per pass instead of one per pass and buffer.  Only
// for compile-time patches and Haar groups of a power of two (by the pyramid or
// by the matrix without its zeros); returns false, having done nothing,
// otherwise.  Every element goes through the same operations as in
// transform_group, so the results are the same bits.
template <int ND, int B0, int B1, int B2, class GM>
__device__ bool transform_forward_all(const GM& geo, const FilterArgs& a, unsigned char* smem, int n, float* S,
                                      float* X, float* R) {
    if constexpr (ND == 0) {
        return false;
    } else {
        if (a.sp.group_transform != BMND_GROUP_HAAR || !is_pow2(n) || n < 2) return false;
        const float* G = sm<float>(smem, a.L.g);
        if (a.sp.fast_group_transform) {
            if (!haar_axis_any3<GM::LB>(S, X, R, n, geo.P(), geo.PP())) return false;
        } else {
            if (a.den_ro || sm<int>(smem, a.L.misc)[kMiscWild] != 0) return false;
            switch (n) {
                case 2: haar_product_all<2, GM::LB>(S, X, R, geo.P(), geo.PP(), G); break;
                case 4: haar_product_all<4, GM::LB>(S, X, R, geo.P(), geo.PP(), G); break;
                case 8: haar_product_all<8, GM::LB>(S, X, R, geo.P(), geo.PP(), G); break;
                case 16: haar_product_all<16, GM::LB>(S, X, R, geo.P(), geo.PP(), G); break;
                case 32: haar_product_all<32, GM::LB>(S, X, R, geo.P(), geo.PP(), G); break;
                default: return false;
            }
        }
        const float* F = sm<float>(smem, a.L.fw);
        space_axis_fixed_all<ND, B0, B1, B2, 0>(S, X, R, n, F);
        if constexpr (ND > 1) space_axis_fixed_all<ND, B0, B1, B2, 1>(S, X, R, n, F + BMND_MAX_EDGE * BMND_MAX_EDGE);
        if constexpr (ND > 2)
            space_axis_fixed_all<ND, B0, B1, B2, 2>(S, X, R, n, F + 2 * BMND_MAX_EDGE * BMND_MAX_EDGE);
        return true;
    }
}

// exact float -> double widening on the integer pipe (IEEE 754 binary32 to
// binary64: rebias the exponent by 1023 - 127, shift the fraction by 29);
// zeros keep their sign, subnormals, infinities and NaNs take the hardware
// conversion.  The scatter widens two or three values per entry, and the
// float64 pipe is a small fraction of the FP32 rate on this GPU.
__device__ __forceinline__ double widen_f64(float f) {
    const uint32_t u = __float_as_uint(f);
    const uint32_t e = (u >> 23) & 0xffu;
    const uint64_t sign = static_cast<uint64_t>(u & 0x80000000u) << 32;
    if ((u & 0x7fffffffu) == 0u) return __longlong_as_double(static_cast<long long>(sign));
    if (e == 0u || e == 0xffu) return static_cast<double>(f);
    const uint64_t bits = sign | (static_cast<uint64_t>(e + 896u) << 52) | (static_cast<uint64_t>(u & 0x7fffffu) << 29);
    return __longlong_as_double(static_cast<long long>(bits));
}

__device__ __forceinline__ float variance_of(float x, float scale_f, float floor_f) {
    float nn = x > 0.0f ? x : 0.0f;
    float v = mul_rn(scale_f, nn);
    return v > floor_f ? v : floor_f;
}

// Tolerance-aware hard-threshold mask of the Poisson path (bmndalgo.py:460-485,
// poisson.py:30-46): in count units cc = mag / scale and tc = thr / scale, a
// coefficient is kept iff cc > tc + 128 eps32 max(cc, tc, 1), evaluated in
// float64.  Multiplying through by scale, the real-arithmetic boundary is
// A = thr + 2^-16 max(mag, thr, scale).  Its float32 estimate a is within
// 2^-23 A of it, and the float64 evaluation within ~2^-50 A, so whenever mag
// lies outside a * (1 -+ 2^-20) the float32 comparison gives the float64
// decision; only the band around the boundary (and non-finite inputs) takes the
// float64 path.
__device__ __forceinline__ bool ht_keep_f64(float mag, float thr, double scale) {
    double cc = static_cast<double>(mag) / scale;
    double tc = static_cast<double>(thr) / scale;
    double cs = cc > tc ? cc : tc;
    if (cs < 1.0) cs = 1.0;
    double tol = 128.0 * 1.1920928955078125e-07 * cs;
    return cc > tc + tol;
}

__device__ __forceinline__ bool ht_keep(float mag, float thr, double scale, float scale_f) {
    const float cs = fmaxf(fmaxf(mag, thr), scale_f);
    if (cs >= 1e-30f && cs <= 1e30f) {
        const float a = add_rn(thr, mul_rn(1.52587890625e-05f, cs));  // 2^-16
        if (mag > mul_rn(a, 1.00000095367431640625f)) return true;   // 1 + 2^-20
        if (mag < mul_rn(a, 0.99999904632568359375f)) return false;  // 1 - 2^-20
    }
    return ht_keep_f64(mag, thr, scale);
}

// Exact overlap-aware variance of the first kk group planes (variance.py:950-975):
//   var[i, j] = sum_v V_v c_v[i, j]^2,   c_v[i, j] = sum_{e in v} G[i, g_e] S[j, p_e]
// over the union voxels v, each voxel's entries taken in ascending member order.
// S[j, p] is read from the precomputed S^T, whose entries are the reference's
// float32 Kronecker products.  c and the sum over voxels are accumulated with
// fused multiply-adds (one rounding per term instead of the reference's two).
//
// Work split: warp w takes the voxels whose entry lists start in its 1/nw share
// of all entries, and accumulates every (plane, coefficient) pair over them;
// lane l holds NQ planes (4, or kk when fewer) of the JR consecutive
// coefficients j0 + JR * l + r, so one entry costs three loads (the entry and
// the NQ G values, both warp broadcasts, and one JR-wide vector of S^T) for
// NQ * JR fused multiply-adds.
// The warps' partial sums are then added in warp order, which fixes the result
// independently of scheduling.  An entry packs member g (low byte) and the row
// offset p * kron_stride(P) of S^T (upper bits).
template <int JR>
struct KronVec;
template <>
struct KronVec<1> {
    float v[1];
    __device__ __forceinline__ void load(const float* p) { v[0] = __ldg(p); }
};
template <>
struct KronVec<2> {
    float v[2];
    __device__ __forceinline__ void load(const float* p) {
        const float2 t = __ldg(reinterpret_cast<const float2*>(p));
        v[0] = t.x;
        v[1] = t.y;
    }
};
template <>
struct KronVec<4> {
    float v[4];
    __device__ __forceinline__ void load(const float* p) {
        const float4 t = __ldg(reinterpret_cast<const float4*>(p));
        v[0] = t.x;
        v[1] = t.y;
        v[2] = t.z;
        v[3] = t.w;
    }
};

template <int NQ>
struct PlaneVec {
    float v[NQ];
    // from the paired table (g, g)
    __device__ __forceinline__ void load_pairs(const unsigned char* p) {
#pragma unroll
        for (int q = 0; q < NQ; ++q) v[q] = reinterpret_cast<const float2*>(p)[q].x;
    }
    __device__ __forceinline__ void load(const float* p) {
        if constexpr (NQ == 4) {
            const float4 t = *reinterpret_cast<const float4*>(p);
            v[0] = t.x;
            v[1] = t.y;
            v[2] = t.z;
            v[3] = t.w;
        } else if constexpr (NQ == 2) {
            const float2 t = *reinterpret_cast<const float2*>(p);
            v[0] = t.x;
            v[1] = t.y;
        } else {
            v[0] = *p;
        }
    }
};

// The warp's (or half-warp's) voxels [u_lo, u_hi) are walked as one stream of
// entries: an entry adds G[i, g] S[j, p] to the running c of its voxel, and the
// first entry of the next voxel first folds V_u c^2 into var.  The loads of
// entry e + 1 are issued before the multiply-adds of entry e, and its entry
// word one step earlier, so the shared-memory and L1 latencies overlap the
// arithmetic across voxel boundaries.  Lane l holds RL coefficients starting
// at j0 + jl (jl = RL l, or RL (l % 16) for the half-warp form).
template <int RL, int NQ>
__device__ __forceinline__ void exact_stream(const float* __restrict__ lval, const int* __restrict__ lstart,
                                             const uint32_t* __restrict__ lent, int u_lo, int u_hi,
                                             const unsigned char* smem, uint32_t plane_byte, uint32_t stride,
                                             const float* __restrict__ stl, float (&var)[RL][NQ]) {
    const unsigned char* gb = smem + plane_byte;
#pragma unroll
    for (int r = 0; r < RL; ++r)
#pragma unroll
        for (int q = 0; q < NQ; ++q) var[r][q] = 0.0f;
    if (u_lo >= u_hi) return;
    int e = lstart[u_lo];
    const int e_end = lstart[u_hi];
    int u = u_lo;
    int next_start = lstart[u + 1];
    float v = lval[u];
    float c[RL][NQ];
#pragma unroll
    for (int r = 0; r < RL; ++r)
#pragma unroll
        for (int q = 0; q < NQ; ++q) c[r][q] = 0.0f;
    uint32_t ent1 = lent[e];
    PlaneVec<NQ> g0;
    KronVec<RL> s0;
    g0.load_pairs(gb + (ent1 & 0xffffu));
    s0.load(stl + (ent1 >> 16) * stride);
    ent1 = lent[e + 1 < e_end ? e + 1 : e];
    for (; e < e_end; ++e) {
        // loads of entry e + 1 (harmless repeats of the last entry at the end)
        PlaneVec<NQ> g1;
        KronVec<RL> s1;
        g1.load_pairs(gb + (ent1 & 0xffffu));
        s1.load(stl + (ent1 >> 16) * stride);
        const uint32_t ent2 = lent[e + 2 < e_end ? e + 2 : e_end - 1];
        if (e == next_start) {
#pragma unroll
            for (int r = 0; r < RL; ++r)
#pragma unroll
                for (int q = 0; q < NQ; ++q) {
                    var[r][q] = fmaf(mul_rn(v, c[r][q]), c[r][q], var[r][q]);
                    c[r][q] = 0.0f;
                }
            ++u;
            v = lval[u];
            next_start = lstart[u + 1];
        }
        // the voxel's first entry: fma(g, s, 0) is the rounded product
#pragma unroll
        for (int r = 0; r < RL; ++r)
#pragma unroll
            for (int q = 0; q < NQ; ++q) c[r][q] = fmaf(g0.v[q], s0.v[r], c[r][q]);
        g0 = g1;
        s0 = s1;
        ent1 = ent2;
    }
#pragma unroll
    for (int r = 0; r < RL; ++r)
#pragma unroll
        for (int q = 0; q < NQ; ++q) var[r][q] = fmaf(mul_rn(v, c[r][q]), c[r][q], var[r][q]);
}

// The same stream for four coefficients per lane in packed pairs (two
// multiply-adds per instruction, each rounded as its scalar form).  It is bound
// by instruction issue, so addresses are kept in 32-bit shared-memory form (the
// generic 64-bit pointers cost more integer instructions than the products):
// an entry word holds the shared-memory byte offset of the member's paired G
// entries and the patch element; two words past the last one are readable.  A
// voxel's first entry starts its sums with a product.
__device__ __forceinline__ uint32_t lds32(uint32_t addr) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ void lds_pairs(float2& a, float2& b, uint32_t addr) {
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(a.x), "=f"(a.y), "=f"(b.x), "=f"(b.y)
                 : "r"(addr));
}

// G pairs of an entry's member (planes from `plane`, a shared-memory address)
template <int NQ>
__device__ __forceinline__ void load_pairs(float2 (&g)[NQ], uint32_t plane, uint32_t ent) {
    const uint32_t at = plane + (ent & 0xffffu);
    if constexpr (NQ == 4) {
        lds_pairs(g[0], g[1], at);
        lds_pairs(g[2], g[3], at + 16);
    } else if constexpr (NQ == 2) {
        lds_pairs(g[0], g[1], at);
    } else {
        asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(g[0].x), "=f"(g[0].y) : "r"(at));
    }
}

// the lane's four coefficients of the entry's row of S^T
__device__ __forceinline__ void load_row(float2 (&sv)[2], const char* row0, uint32_t ent, uint32_t stride_b) {
    const float4 t = __ldg(reinterpret_cast<const float4*>(row0 + static_cast<uint64_t>(ent >> 16) * stride_b));
    sv[0] = make_float2(t.x, t.y);
    sv[1] = make_float2(t.z, t.w);
}

//
// D entries' rows are in flight.  Two suffice where S^T lies in L1 or near it; the
// runtime geometry's tables of more than 64 voxels (1 MB at 8x8x8, one CTA per SM)
// come from L2, whose latency four cover (44 x 48 x 52, 8x8x8, 32 members: one plane
// 51.2 -> 37.2 ms, four 57.9 -> 44.6; the scalar stream before the pairs 39.0, 52.7).
template <int NQ, int D>
__device__ __forceinline__ void exact_pairs(const unsigned char* smem, const float* lval, const int* lstart,
                                            const uint32_t* lent, int u_lo, int u_hi, uint32_t plane_byte,
                                            const float* __restrict__ st, uint32_t stride_b,
                                            float2 (&var)[2][NQ]) {
#pragma unroll
    for (int q = 0; q < NQ; ++q) var[0][q] = var[1][q] = make_float2(0.0f, 0.0f);
    if (u_lo >= u_hi) return;
    const uint32_t plane = static_cast<uint32_t>(__cvta_generic_to_shared(smem)) + plane_byte;
    const uint32_t ents = static_cast<uint32_t>(__cvta_generic_to_shared(lent));
    uint32_t ls = static_cast<uint32_t>(__cvta_generic_to_shared(lstart + u_lo));
    const uint32_t lv = static_cast<uint32_t>(__cvta_generic_to_shared(lval)) -
                        static_cast<uint32_t>(__cvta_generic_to_shared(lstart));  // lval[u] at lv + &lstart[u]
    const char* row0 = reinterpret_cast<const char*>(st);
    uint32_t ep = ents + 4u * static_cast<uint32_t>(lstart[u_lo]);
    const uint32_t end = ents + 4u * static_cast<uint32_t>(lstart[u_hi]);
    uint32_t next = ep;
    float v = 0.0f;  // before the first voxel: a fold of zeros
    float2 c[2][NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) c[0][q] = c[1][q] = make_float2(0.0f, 0.0f);
    auto fold = [&]() {
        const float2 vv = make_float2(v, v);
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            var[0][q] = __ffma2_rn(__fmul2_rn(vv, c[0][q]), c[0][q], var[0][q]);
            var[1][q] = __ffma2_rn(__fmul2_rn(vv, c[1][q]), c[1][q], var[1][q]);
        }
    };
    if constexpr (D > 2) {
        auto at = [&](int ahead) { return lds32(min(ep + 4u * ahead, end - 4u)); };  // (the last entry again at the end)
        float2 g[NQ], sv[D][2];
        uint32_t ent[D];
#pragma unroll
        for (int d = 0; d < D; ++d) {
            ent[d] = at(d);
            load_row(sv[d], row0, ent[d], stride_b);
        }
        while (true) {
#pragma unroll
            for (int d = 0; d < D; ++d) {
                load_pairs<NQ>(g, plane, ent[d]);
                ent[d] = at(D);
                if (ep == next) {
                    fold();
                    v = __uint_as_float(lds32(ls + lv));
                    ls += 4;
                    next = ents + 4u * lds32(ls);
#pragma unroll
                    for (int q = 0; q < NQ; ++q) c[0][q] = c[1][q] = make_float2(0.0f, 0.0f);
                }
#pragma unroll
                for (int q = 0; q < NQ; ++q) {  // (fma(g, s, 0) is the rounded product)
                    c[0][q] = __ffma2_rn(g[q], sv[d][0], c[0][q]);
                    c[1][q] = __ffma2_rn(g[q], sv[d][1], c[1][q]);
                }
                load_row(sv[d], row0, ent[d], stride_b);
                ep += 4;
                if (ep == end) {
                    fold();
                    return;
                }
            }
        }
    }
    float2 g0[NQ], s0[2], g1[NQ], s1[2];
    uint32_t ent = lds32(ep);
    load_pairs<NQ>(g0, plane, ent);
    load_row(s0, row0, ent, stride_b);
    ent = lds32(ep + 4);
    auto step = [&](const float2 (&g)[NQ], const float2 (&sv)[2]) {
        if (ep == next) {
            fold();
#pragma unroll
            for (int q = 0; q < NQ; ++q) {
                c[0][q] = __fmul2_rn(g[q], sv[0]);
                c[1][q] = __fmul2_rn(g[q], sv[1]);
            }
            v = __uint_as_float(lds32(ls + lv));
            ls += 4;
            next = ents + 4u * lds32(ls);
        } else {
#pragma unroll
            for (int q = 0; q < NQ; ++q) {
                c[0][q] = __ffma2_rn(g[q], sv[0], c[0][q]);
                c[1][q] = __ffma2_rn(g[q], sv[1], c[1][q]);
            }
        }
        ep += 4;
    };
    while (true) {
        // the loads of the next entry are issued before this one's products
        load_pairs<NQ>(g1, plane, ent);
        load_row(s1, row0, ent, stride_b);
        ent = lds32(ep + 8);
        step(g0, s0);
        if (ep == end) break;
        load_pairs<NQ>(g0, plane, ent);
        load_row(s0, row0, ent, stride_b);
        ent = lds32(ep + 8);
        step(g1, s1);
        if (ep == end) break;
    }
    fold();
}

// The stream for Haar groups, whose planes 0 .. 3 have one magnitude each: plane 0
// is a everywhere, plane 1 is a on the first half of the members and -a on the
// second, planes 2 and 3 are +-b on the quarters of one half and zero on the
// other.  So an entry needs no G value, only its member's quarter, and three
// products instead of four: ch collects the half-plane of the current half and
// is folded into its variance where the (ascending) members cross the middle.
// Skipped terms are exact zeros, so every sum keeps its bits.  A voxel with one
// entry (a third of 3-D entries' voxels, more in 2-D) is folded at once.
//
// An entry word is the byte offset of its row of S^T, with the quarter in the
// two lowest bits.  RP pairs of coefficients per lane: 2 for P > 64 (S^T in
// global memory, through L1), 1 for P in 33-64 (S^T in shared memory).
template <int RP, int NQ>
__device__ __forceinline__ void exact_haar(const float* lval, const int* lstart, const uint32_t* lent, int u_lo,
                                           int u_hi, float a0, float b0, const float* __restrict__ st_lane,
                                           uint32_t kron_lane, float2 (&var)[RP][NQ]) {
#pragma unroll
    for (int q = 0; q < NQ; ++q)
#pragma unroll
        for (int r = 0; r < RP; ++r) var[r][q] = make_float2(0.0f, 0.0f);
    if (u_lo >= u_hi) return;
    const uint32_t ents = static_cast<uint32_t>(__cvta_generic_to_shared(lent));
    uint32_t ls = static_cast<uint32_t>(__cvta_generic_to_shared(lstart + u_lo));
    const uint32_t lv = static_cast<uint32_t>(__cvta_generic_to_shared(lval)) -
                        static_cast<uint32_t>(__cvta_generic_to_shared(lstart));  // lval[u] at lv + &lstart[u]
    uint32_t ep = ents + 4u * static_cast<uint32_t>(lstart[u_lo]);
    const uint32_t end = ents + 4u * static_cast<uint32_t>(lstart[u_hi]);
    const float2 A = make_float2(a0, a0), nA = make_float2(-a0, -a0), B = make_float2(b0, b0),
                 nB = make_float2(-b0, -b0);
    auto row = [&](float2 (&sv)[RP], uint32_t ent) {
        if constexpr (RP == 2) {
            const float4 t = __ldg(reinterpret_cast<const float4*>(reinterpret_cast<const char*>(st_lane) + (ent & ~3u)));
            sv[0] = make_float2(t.x, t.y);
            sv[RP - 1] = make_float2(t.z, t.w);
        } else {
            asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];"
                         : "=f"(sv[0].x), "=f"(sv[0].y)
                         : "r"(kron_lane + (ent & ~3u)));
        }
    };
    uint32_t ent = lds32(ep);
    uint32_t nx = lds32(ls + 4);
    while (true) {
        const uint32_t next = ents + 4u * nx;
        const float v = __uint_as_float(lds32(ls + lv));
        ls += 4;
        nx = lds32(ls + 4);  // (one word past the last voxel's is readable)
        const float2 vv = make_float2(v, v);
        float2 sv[RP];
        row(sv, ent);
        uint32_t q = ent;
        ep += 4;
        ent = lds32(ep);
        if (ep == next) {
#pragma unroll
            for (int r = 0; r < RP; ++r) {
                const float2 c = __fmul2_rn(A, sv[r]), x = __fmul2_rn(vv, c);
                var[r][0] = __ffma2_rn(x, c, var[r][0]);
                if constexpr (NQ > 1) var[r][1] = __ffma2_rn(x, c, var[r][1]);
            }
            if constexpr (NQ > 2) {
                float2 y[RP], d[RP];
#pragma unroll
                for (int r = 0; r < RP; ++r) {
                    d[r] = __fmul2_rn(B, sv[r]);
                    y[r] = __fmul2_rn(vv, d[r]);
                }
                if (q & 2u) {
#pragma unroll
                    for (int r = 0; r < RP; ++r) var[r][NQ - 1] = __ffma2_rn(y[r], d[r], var[r][NQ - 1]);
                } else {
#pragma unroll
                    for (int r = 0; r < RP; ++r) var[r][NQ - 2] = __ffma2_rn(y[r], d[r], var[r][NQ - 2]);
                }
            }
        } else {
            float2 c0[RP], c1[RP], ch[RP];
            uint32_t half = q & 2u;
            float2 m1 = half ? nA : A, mb = (q & 1u) ? nB : B;
#pragma unroll
            for (int r = 0; r < RP; ++r) {
                c0[r] = __fmul2_rn(A, sv[r]);
                if constexpr (NQ > 1) c1[r] = __fmul2_rn(m1, sv[r]);
                if constexpr (NQ > 2) ch[r] = __fmul2_rn(mb, sv[r]);
            }
            do {
                row(sv, ent);
                q = ent;
                ep += 4;
                ent = lds32(ep);
                mb = (q & 1u) ? nB : B;
                if ((q & 2u) != half) {  // into the second half: plane 2 is complete
                    half = 2u;
                    m1 = nA;
                    if constexpr (NQ > 2) {
#pragma unroll
                        for (int r = 0; r < RP; ++r) {
                            var[r][NQ - 2] = __ffma2_rn(__fmul2_rn(vv, ch[r]), ch[r], var[r][NQ - 2]);
                            ch[r] = __fmul2_rn(mb, sv[r]);
                        }
                    }
                } else if constexpr (NQ > 2) {
#pragma unroll
                    for (int r = 0; r < RP; ++r) ch[r] = __ffma2_rn(mb, sv[r], ch[r]);
                }
#pragma unroll
                for (int r = 0; r < RP; ++r) {
                    c0[r] = __ffma2_rn(A, sv[r], c0[r]);
                    if constexpr (NQ > 1) c1[r] = __ffma2_rn(m1, sv[r], c1[r]);
                }
            } while (ep != next);
#pragma unroll
            for (int r = 0; r < RP; ++r) {
                var[r][0] = __ffma2_rn(__fmul2_rn(vv, c0[r]), c0[r], var[r][0]);
                if constexpr (NQ > 1) var[r][1] = __ffma2_rn(__fmul2_rn(vv, c1[r]), c1[r], var[r][1]);
            }
            if constexpr (NQ > 2) {
                if (half) {
#pragma unroll
                    for (int r = 0; r < RP; ++r)
                        var[r][NQ - 1] = __ffma2_rn(__fmul2_rn(vv, ch[r]), ch[r], var[r][NQ - 1]);
                } else {
#pragma unroll
                    for (int r = 0; r < RP; ++r)
                        var[r][NQ - 2] = __ffma2_rn(__fmul2_rn(vv, ch[r]), ch[r], var[r][NQ - 2]);
                }
            }
        }
        if (ep == end) break;
    }
}

// all tiles of (NQ planes) x (32 JR coefficients); EX[i * P + j] receives the
// standard deviation sqrt(max(var, 0)) of planes i < kk.  NQ = 4 in general;
// groups with fewer exact planes (k < 4, or fewer members) use NQ = kk.  Each
// warp leaves its partial sums in `part`; after one barrier every thread adds
// the warps' partials of its (plane, coefficient) pairs in warp order.
//
// Patches of 33-64 voxels (JR = 2): the two half-warps take the two halves of
// the warp's voxels and each lane holds 4 coefficients, j = 4 (lane % 16) + r,
// so an entry costs the same loads for 4 NQ multiply-adds instead of 2 NQ; the
// halves' sums are added at the end.  (A whole warp per half, without the
// divergence where only one half ends a voxel, took 14 % more instructions.)
template <int JR, int NQ, bool HAAR, int D>
__device__ void exact_planes(const unsigned char* smem, float a0, float b0, uint32_t kron_byte, const float* __restrict__ lval,
                             const int* __restrict__ lstart, const uint32_t* __restrict__ lent, int U,
                             int kk, const float* __restrict__ st, int P,
                             float* __restrict__ EX, float* __restrict__ part, bool part_over) {
    constexpr bool kHalf = JR == 2 && !HAAR;
    constexpr int RL = kHalf ? 4 : JR;  // coefficients per lane
    constexpr int TW = 32 * JR;         // coefficients per tile
    const uint32_t stride = static_cast<uint32_t>(kron_stride(P));
    const int warp = static_cast<int>(threadIdx.x) >> 5, lane = static_cast<int>(threadIdx.x) & 31;
    const int nw = blockDim.x >> 5;
    // voxel range of this warp: voxels whose first entry lies in its entry share
    const int E = lstart[U];
    auto first_voxel = [&](int e, int lo, int hi) {  // first u in [lo, hi] with lstart[u] >= e
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (lstart[mid] < e) lo = mid + 1;
            else hi = mid;
        }
        return lo;
    };
    const int u_lo = first_voxel(static_cast<int>(static_cast<int64_t>(E) * warp / nw), 0, U);
    const int u_hi = warp == nw - 1 ? U : first_voxel(static_cast<int>(static_cast<int64_t>(E) * (warp + 1) / nw), 0, U);
    const int jl = kHalf ? 4 * (lane & 15) : JR * lane;
    for (int i0 = 0; i0 < kk; i0 += NQ) {
        for (int j0 = 0; j0 < P; j0 += TW) {
            float out[RL][NQ];
            if constexpr (HAAR && JR > 1) {
                // JR == 2: the halves of the warp's voxels one after the other (their
                // sums are added as in the generic form below)
                constexpr int RP = JR / 2;
                const int u_mid = JR == 2 ? first_voxel((lstart[u_lo] + lstart[u_hi]) >> 1, u_lo, u_hi) : u_hi;
                const uint32_t kron_lane = static_cast<uint32_t>(__cvta_generic_to_shared(smem)) + kron_byte + 8u * lane;
                float2 var[RP][NQ];
                exact_haar<RP, NQ>(lval, lstart, lent, u_lo, u_mid, a0, b0, st + JR * lane, kron_lane, var);
#pragma unroll
                for (int q = 0; q < NQ; ++q)
#pragma unroll
                    for (int r = 0; r < RP; ++r) {
                        out[2 * r][q] = var[r][q].x;
                        out[2 * r + 1][q] = var[r][q].y;
                    }
                if constexpr (JR == 2) {
                    exact_haar<RP, NQ>(lval, lstart, lent, u_mid, u_hi, a0, b0, st + JR * lane, kron_lane, var);
#pragma unroll
                    for (int q = 0; q < NQ; ++q) {
                        out[0][q] = add_rn(out[0][q], var[0][q].x);
                        out[1][q] = add_rn(out[1][q], var[0][q].y);
                    }
                }
            } else if constexpr (JR == 1) {
                exact_stream<1, NQ>(lval, lstart, lent, u_lo, u_hi, smem, 8u * i0, stride, st + j0 + lane, out);
            } else {
                float2 var[2][NQ];
                int lo = u_lo, hi = u_hi;
                if (kHalf) {
                    // split at the first voxel whose entries start in the second half of the entries
                    const int u_mid = first_voxel((lstart[u_lo] + lstart[u_hi]) >> 1, u_lo, u_hi);
                    if (lane >> 4) lo = u_mid;
                    else hi = u_mid;
                }
                exact_pairs<NQ, D>(smem, lval, lstart, lent, lo, hi, 8u * i0, st + j0 + jl, 4u * stride, var);
#pragma unroll
                for (int q = 0; q < NQ; ++q)
#pragma unroll
                    for (int r = 0; r < 2; ++r) {
                        out[2 * r][q] = var[r][q].x;
                        out[2 * r + 1][q] = var[r][q].y;
                    }
                if (kHalf) {
#pragma unroll
                    for (int r = 0; r < RL; ++r)
#pragma unroll
                        for (int q = 0; q < NQ; ++q)
                            out[r][q] = add_rn(out[r][q], __shfl_xor_sync(0xffffffffu, out[r][q], 16));
                }
            }
            if (part_over) __syncthreads();  // every warp is done with the lists
            if (!kHalf || lane < 16) {
#pragma unroll
                for (int q = 0; q < NQ; ++q)
#pragma unroll
                    for (int r = 0; r < RL; ++r) part[(warp * NQ + q) * TW + jl + r] = out[r][q];
            }
            __syncthreads();
            for (int t = static_cast<int>(threadIdx.x); t < NQ * TW; t += blockDim.x) {
                const int q = t / TW, jj = t - q * TW;
                const int i = i0 + q, j = j0 + jj;
                if (i < kk && j < P) {
                    float v = part[q * TW + jj];
                    for (int w = 1; w < nw; ++w) v = add_rn(v, part[(w * NQ + q) * TW + jj]);
                    EX[i * P + j] = sqrtf(v > 0.0f ? v : 0.0f);
                }
            }
            __syncthreads();
        }
    }
}

template <int JR, int D = 2>
__device__ void exact_planes_any(const unsigned char* smem, bool haar, float a0, float b0, uint32_t kron_byte,
                                 const float* __restrict__ lval, const int* __restrict__ lstart,
                                 const uint32_t* __restrict__ lent, int U, int kk, const float* __restrict__ st, int P,
                                 float* __restrict__ EX, float* __restrict__ part, bool part_over) {
    auto run = [&](auto h) {
        constexpr bool H = decltype(h)::value;
        if (kk == 1) exact_planes<JR, 1, H, D>(smem, a0, b0, kron_byte, lval, lstart, lent, U, kk, st, P, EX, part, part_over);
        else if (kk == 2) exact_planes<JR, 2, H, D>(smem, a0, b0, kron_byte, lval, lstart, lent, U, kk, st, P, EX, part, part_over);
        else exact_planes<JR, 4, H, D>(smem, a0, b0, kron_byte, lval, lstart, lent, U, kk, st, P, EX, part, part_over);
    };
    if (JR > 1 && haar) run(BoolTag<JR != 1>{});
    else run(BoolTag<false>{});
}

// Exact noise risk of the first kk planes (wiener.py:638-711, :505-535; the
// group metric Ginv^T Ginv of the orthonormal group transforms is the
// identity, the reference's diagonal branch):
//   risk = sum_u V_u sum_{g < kk} f_u[g]^T SM f_u[g],  f_u[g][j] = a[g][j] c_u[g][j],
// c_u as in the exact variance and SM = S_inv^T diag(w^2) S_inv, row p at
// sm + p * kron_stride(P).  Lane l holds coefficients j = JR l + r (P <= 32 JR:
// one tile); (f SM)[j] = sum_p f[p] SM[p][j] takes f[p] from its lane by a
// shuffle.  The voxel terms are float32, their sum over voxels float64.
template <int JR, int NQ>
__device__ double exact_risk_tile(const unsigned char* smem, const float* __restrict__ lval, const int* __restrict__ lstart,
                                  const uint32_t* __restrict__ lent, int u_lo, int u_hi,
                                  int i0, int kk,
                                  const float* __restrict__ st, const float* __restrict__ smt,
                                  const float* __restrict__ att, int P) {
    const int lane = static_cast<int>(threadIdx.x) & 31;
    const int stride = kron_stride(P);
    const float* stl = st + JR * lane;
    float gq[JR][NQ];
#pragma unroll
    for (int r = 0; r < JR; ++r)
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            const int j = JR * lane + r, i = i0 + q;
            gq[r][q] = (j < P && i < kk) ? att[i * P + j] : 0.0f;
        }
    double acc = 0.0;
    for (int u = u_lo; u < u_hi; ++u) {
        int e = lstart[u];
        const int e1 = lstart[u + 1];
        float c[JR][NQ];
        {
            const uint32_t ent = lent[e];
            PlaneVec<NQ> gv;
            gv.load_pairs(smem + 8 * i0 + (ent & 0xffffu));
            KronVec<JR> sv;
            sv.load(stl + (ent >> 16) * static_cast<uint32_t>(stride));
#pragma unroll
            for (int r = 0; r < JR; ++r)
#pragma unroll
                for (int q = 0; q < NQ; ++q) c[r][q] = mul_rn(gv.v[q], sv.v[r]);
        }
        for (++e; e < e1; ++e) {
            const uint32_t ent = lent[e];
            PlaneVec<NQ> gv;
            gv.load_pairs(smem + 8 * i0 + (ent & 0xffffu));
            KronVec<JR> sv;
            sv.load(stl + (ent >> 16) * static_cast<uint32_t>(stride));
#pragma unroll
            for (int r = 0; r < JR; ++r)
#pragma unroll
                for (int q = 0; q < NQ; ++q) c[r][q] = fmaf(gv.v[q], sv.v[r], c[r][q]);
        }
        float f[JR][NQ], pr[JR][NQ];
#pragma unroll
        for (int r = 0; r < JR; ++r)
#pragma unroll
            for (int q = 0; q < NQ; ++q) {
                f[r][q] = mul_rn(gq[r][q], c[r][q]);
                pr[r][q] = 0.0f;
            }
        for (int sl = 0; sl < 32; ++sl) {
#pragma unroll
            for (int rr = 0; rr < JR; ++rr) {
                const int p = sl * JR + rr;
                if (p < P) {  // the same for every lane
                    float fp[NQ];
#pragma unroll
                    for (int q = 0; q < NQ; ++q) fp[q] = __shfl_sync(0xffffffffu, f[rr][q], sl);
                    KronVec<JR> mv;
                    mv.load(smt + p * stride + JR * lane);
#pragma unroll
                    for (int r = 0; r < JR; ++r)
#pragma unroll
                        for (int q = 0; q < NQ; ++q) pr[r][q] = fmaf(fp[q], mv.v[r], pr[r][q]);
                }
            }
        }
        float t = 0.0f;
#pragma unroll
        for (int r = 0; r < JR; ++r)
#pragma unroll
            for (int q = 0; q < NQ; ++q) t = fmaf(f[r][q], pr[r][q], t);
        acc = fma(static_cast<double>(lval[u]), static_cast<double>(t), acc);
    }
    return acc;
}

// the group's exact noise risk into *out (every thread returns after it is set):
// warp w takes the voxels whose entry lists start in its share of all entries
// (the exact variance's split); lanes, then warps, add in a fixed order
template <int JR, int NQ>
__device__ void exact_risk(const unsigned char* smem, const float* __restrict__ lval, const int* __restrict__ lstart,
                           const uint32_t* __restrict__ lent, int U, int kk, const float* __restrict__ st, const float* __restrict__ smt,
                           const float* __restrict__ att, int P, double* __restrict__ part) {
    const int warp = static_cast<int>(threadIdx.x) >> 5, lane = static_cast<int>(threadIdx.x) & 31;
    const int nw = blockDim.x >> 5;
    const int E = lstart[U];
    auto first_voxel = [&](int e) {
        int lo = 0, hi = U;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (lstart[mid] < e) lo = mid + 1;
            else hi = mid;
        }
        return lo;
    };
    const int u_lo = first_voxel(static_cast<int>(static_cast<int64_t>(E) * warp / nw));
    const int u_hi = warp == nw - 1 ? U : first_voxel(static_cast<int>(static_cast<int64_t>(E) * (warp + 1) / nw));
    double acc = 0.0;
    for (int i0 = 0; i0 < kk; i0 += NQ)
        acc += exact_risk_tile<JR, NQ>(smem, lval, lstart, lent, u_lo, u_hi, i0, kk, st, smt, att, P);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) part[warp] = acc;
    __syncthreads();
    if (static_cast<int>(threadIdx.x) == 0) {
        double t = 0.0;
        for (int w = 0; w < nw; ++w) t += part[w];
        part[nw] = t;
    }
    __syncthreads();
}

// (kept out of line: inlined, its registers and order followed unrelated changes of
// the kernel, 20.1 to 21.3 ms for stage 1 of 220 x 260; so, 20.2, and stage 2 14.3
// against 14.6)
template <int JR>
__device__ __noinline__ void exact_risk_any(const unsigned char* smem, const float* __restrict__ lval, const int* __restrict__ lstart,
                               const uint32_t* __restrict__ lent, int U,
                               int kk, const float* __restrict__ st, const float* __restrict__ smt,
                               const float* __restrict__ att, int P, double* __restrict__ part) {
    if (kk == 1) exact_risk<JR, 1>(smem, lval, lstart, lent, U, kk, st, smt, att, P, part);
    else if (kk == 2) exact_risk<JR, 2>(smem, lval, lstart, lent, U, kk, st, smt, att, P, part);
    else exact_risk<JR, 4>(smem, lval, lstart, lent, U, kk, st, smt, att, P, part);
}

// Exact Gaussian variances of planes 0 .. 3 of a Haar group (kk of them): with
// plane magnitudes a (planes 0, 1) and b (2, 3), every product of the pair sums
//   sum_i w_i C(0) w_i + sum_{j < i} (w_i w_j) 2 C(lag_ij)
// is +-a^2 or +-b^2 times 2 C, so planes 0 and 1 share one load and one product
// per pair, and planes 2 and 3 take the pairs within one half of the members.
// (One thread per plane and coefficient loaded every covariance four times, 528
// rows per plane, and was bound by those loads.)  Half of the threads sum planes
// 0 and 1, the other half 2 and 3; a thread's coefficient is its index.  The sums
// keep the generic order (ascending i, then j), with up to 8 loads in flight.
__device__ __forceinline__ void gauss_haar(const float* __restrict__ cm, const int* lag, int lrow, int n, int kk, int P,
                                           const float* G, float* EX) {
    const int half_threads = blockDim.x >> 1;
    const bool outer = static_cast<int>(threadIdx.x) < half_threads;  // planes 0 and 1
    const int c = outer ? threadIdx.x : threadIdx.x - half_threads;
    if (c >= P || (!outer && kk <= 2)) return;
    const float w = outer ? G[0] : G[2 * n];
    const float pv = __ldg(cm + c), ww = mul_rn(w, w), diag = mul_rn(mul_rn(w, pv), w);
    const float* cc = cm + c;
    float v0 = 0.0f, v1 = 0.0f;
    const int half = n >> 1, quarter = n >> 2;
    // pairs (i, j0 <= j < j1), all of one sign in plane 1 (planes 2, 3: in v0)
    auto run = [&](int i, int j0, int j1, bool minus) {
        const int* row = lag + i * lrow;
        for (int j = j0; j < j1; j += 8) {
            float cv[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) cv[u] = j + u < j1 ? __ldg(cc + static_cast<int64_t>(row[j + u]) * P) : 0.0f;
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                if (j + u < j1) {
                    const float t = mul_rn(ww, add_rn(cv[u], cv[u]));
                    if (outer) {
                        v0 = add_rn(v0, t);
                        v1 = minus ? sub_rn(v1, t) : add_rn(v1, t);
                    } else {
                        v0 = minus ? sub_rn(v0, t) : add_rn(v0, t);
                    }
                }
            }
        }
    };
    if (outer) {
        for (int i = 0; i < n; ++i) {
            v0 = add_rn(v0, diag);
            v1 = add_rn(v1, diag);
            const int split = i >= half ? half : 0;  // second-half member: the first half counts negatively
            run(i, 0, split, true);
            run(i, split, i, false);
        }
        EX[c] = fmaxf(v0, 0.0f);
        if (kk > 1) EX[P + c] = fmaxf(v1, 0.0f);
    } else {
        for (int h = 0; h < 2 && 2 + h < kk; ++h) {
            v0 = 0.0f;
            const int first = h * half;
            for (int i = first; i < first + half; ++i) {
                v0 = add_rn(v0, diag);
                const int split = i >= first + quarter ? first + quarter : first;
                run(i, first, split, true);
                run(i, split, i, false);
            }
            EX[(2 + h) * P + c] = fmaxf(v0, 0.0f);
        }
    }
}

// One group, by a whole CTA.  APPROX: no exact planes (variance_k = 0).
template <int ND, int B0, int B1, int B2, bool APPROX>
__device__ __forceinline__ void filter_group(const FilterArgs& a, unsigned char* smem, int64_t gid) {
    using GM = Geom<ND, B0, B1, B2>;
    const BmndStageParams& sp = a.sp;
    const GM geo(sp);
    const int tid = static_cast<int>(threadIdx.x);
    const int P = geo.P();
    const int n = a.count[gid];
    if (n <= 0) return;
    if (n > a.nmax) {
        if (tid == 0 && a.err) atomicExch(a.err, 2);
        return;
    }
    const bool wiener = sp.filter == BMND_FILTER_WIENER;
    const int kmax = a.kmax;

    float* G = sm<float>(smem, a.L.g);
    float2* GT2 = sm<float2>(smem, a.L.gt2);
    float* Fw = sm<float>(smem, a.L.fw);
    float* win = sm<float>(smem, a.L.win);
    double* mdiag = sm<double>(smem, a.L.mdiag);
    int* voff = sm<int>(smem, a.L.voff);
    int* pos = sm<int>(smem, a.L.pos);
    int* shf = sm<int>(smem, a.L.shf);
    int* org0 = sm<int>(smem, a.L.org0);
    float* S = sm<float>(smem, a.L.s);
    float* EX = sm<float>(smem, a.L.ex);
    float* X = sm<float>(smem, a.L.x);
    float* R = sm<float>(smem, a.L.r);
    float* V = sm<float>(smem, a.L.v);  // aliases R: the attenuation
    uint32_t* grid = sm<uint32_t>(smem, a.L.grid);
    float* lval = sm<float>(smem, a.L.lval);
    int* lstart = sm<int>(smem, a.L.lstart);
    uint32_t* lent = sm<uint32_t>(smem, a.L.lent);
    int2* scan = sm<int2>(smem, a.L.scan);
    double* plane = sm<double>(smem, a.L.plane);
    float* wts = sm<float>(smem, a.L.wts);
    int* misc = sm<int>(smem, a.L.misc);

    const int k = APPROX ? 0 : sp.variance_k;
    const int kk = k < n ? k : n;
    const int kpad = APPROX ? 0 : (a.kmax + 3) / 4 * 4;
    // ---- setup: constants of the launch, positions, group matrix ----
    {
        float* Fi = sm<float>(smem, a.L.fi);
        if (ND > 0 && !sp.exact_risk_weights) {
            // from the tables spatial_kron_kernel left after S^T: the parameters
            // live in the constant bank, where lanes reading different addresses
            // take turns
            const float* tab = a.st + static_cast<int64_t>(P) * kron_stride(P);
            constexpr int EE = BMND_MAX_DIMS * BMND_MAX_EDGE * BMND_MAX_EDGE;
            for (int e = tid; e < EE; e += blockDim.x) {
                Fw[e] = __ldg(tab + e);
                Fi[e] = __ldg(tab + EE + e);
            }
            for (int e = tid; e < P; e += blockDim.x) win[e] = __ldg(tab + 2 * EE + e);
        } else {
            for (int d = 0; d < geo.nd(); ++d) {
                const int bb = geo.b(d) * geo.b(d);
                for (int q = tid; q < bb; q += blockDim.x) {
                    Fw[d * BMND_MAX_EDGE * BMND_MAX_EDGE + q] = sp.spatial_fwd[d][q];
                    Fi[d * BMND_MAX_EDGE * BMND_MAX_EDGE + q] = sp.spatial_inv[d][q];
                }
            }
            for (int e = tid; e < P; e += blockDim.x) win[e] = sp.window[e];
        }
        for (int e = tid; e < P; e += blockDim.x) {
            int p = e, off = 0;
#pragma unroll
            for (int d = BMND_MAX_DIMS - 1; d >= 0; --d) {
                if (d < geo.nd()) {
                    off += (p % geo.b(d)) * static_cast<int>(a.vstride[d]);
                    p /= geo.b(d);
                }
            }
            voff[e] = off;
        }
        if (sp.windowed_synthesis)  // the only reader of the metric diagonal
            for (int e = tid; e < P; e += blockDim.x) mdiag[e] = sp.spatial_metric_diag[e];
        if (ND > 0 && a.L.kron_used) {
            float4* kron = sm<float4>(smem, a.L.kron);
            const int words = P * kron_stride(P) / 4;
            for (int e = tid; e < words; e += blockDim.x) kron[e] = __ldg(reinterpret_cast<const float4*>(a.st) + e);
        }
        if (a.den_ro) {
            // matrices are stored densely, b x b row-major, per axis
            float* Fit = sm<float>(smem, a.L.fit);
            constexpr int EE = BMND_MAX_EDGE * BMND_MAX_EDGE;
            for (int e = tid; e < BMND_MAX_DIMS * EE; e += blockDim.x) {
                const int d = e / EE, q = e % EE;
                const int b = d < geo.nd() ? geo.b(d) : 1;
                const int i = q / b, k = q % b;
                Fit[e] = q < b * b ? sp.spatial_inv[d][k * b + i] : 0.0f;
            }
        }
    }
    // a member outside the patch grid skips the group (matching never makes one)
    bool bad_member = false;
    if (tid < n) {
        const int32_t lin = a.sel[gid * sp.max_stack + tid];
        bad_member = lin < 0 || lin >= a.n_lins;
        // lins fit in 31 bits (volumes are limited to 2^31 voxels): 32-bit division
        uint32_t rem = static_cast<uint32_t>(lin);
        int origin = 0;
        for (int d = geo.nd() - 1; d >= 0 && !bad_member; --d) {
            const uint32_t c = static_cast<uint32_t>(a.counts[d]);
            const uint32_t q = rem / c;
            pos[tid * BMND_MAX_DIMS + d] = static_cast<int>(rem - q * c);
            origin += static_cast<int>(rem - q * c) * static_cast<int>(a.vstride[d]);
            rem = q;
        }
        org0[tid] = origin;
    }
    if (__syncthreads_or(bad_member)) {
        if (tid == 0 && a.err) atomicExch(a.err, 2);
        return;
    }
    // the exact phase's entries carry quarters of the Haar group (exact_haar)
    const bool quarters = ND > 0 && kron_jr(P) > 1 && sp.group_transform == BMND_GROUP_HAAR && is_pow2(n) &&
                          sp.noise_model == BMND_NOISE_POISSON && k <= 4;
    {
        const float* gtab = a.st + 2 * static_cast<int64_t>(P) * kron_stride(P) + group_table_offset(n);
        for (int e = tid; e < n * n; e += blockDim.x) G[e] = __ldg(gtab + e);
        // G^T restricted to the exact planes, padded to 4, each entry twice:
        // GT2[g * kpad + i] = (G[i, g], G[i, g])
        for (int e = tid; !quarters && e < n * kpad; e += blockDim.x) {
            const int g = e / kpad, i = e % kpad;
            const float v = i < kk ? __ldg(gtab + i * n + g) : 0.0f;
            GT2[e] = make_float2(v, v);
        }
    }
    if (tid == 32) misc[kMiscWild] = 0;
    if (tid < 32) {
        // group origin (min over members), member shifts, union extent, and the
        // patch-linear offset of each shift: element p of member g lies in union
        // cell c with p = lin(c) - shl[g], lin(c) = sum_d c_d inner(d)
        const bool live = tid < n;
        int lin = 0;
        for (int d = 0; d < geo.nd(); ++d) {
            const int v = live ? pos[tid * BMND_MAX_DIMS + d] : 0x7fffffff;
            const int mn = __reduce_min_sync(0xffffffffu, v);
            const int sh = live ? v - mn : 0;
            const int mx = __reduce_max_sync(0xffffffffu, sh);
            if (live) shf[tid * BMND_MAX_DIMS + d] = sh;
            lin += sh * geo.inner(d);
            if (tid == 0) {
                misc[d] = mn;                  // origin
                misc[4 + d] = mx + geo.b(d);   // union extent
            }
        }
        if (live) sm<int>(smem, a.L.shl)[tid] = lin;
    }
    __syncthreads();

    const float scale_f = static_cast<float>(sp.count_scale);
    const float floor_f = static_cast<float>(sp.variance_floor);
    const float* varsrc = (wiener && sp.wiener_variance_source == BMND_SOURCE_PILOT) ? a.pilot : a.noisy;
    const int total = n * P;
    const bool need_approx = (k <= 0) || (kk < n);

    const bool gauss = sp.noise_model == BMND_NOISE_GAUSSIAN;
    const bool exact_risk = sp.exact_risk_weights != 0 && kk > 0;
    if ((!gauss || exact_risk) && kk > 0) {
        // the exact phase's lists cover a union box of at most ucells_cap
        // cells: members within the search window of their reference
        // always fit; a group spread wider is skipped and reported
        int64_t uc = 1;
        for (int d = 0; d < geo.nd(); ++d) uc *= misc[4 + d];
        if (uc > a.ucells_cap) {
            if (tid == 0 && a.err) atomicExch(a.err, 2);
            return;
        }
    }
    if (gauss) {
        // ---- stationary Gaussian noise (variance.py:2036-2106) ----
        // exact planes g < kk: sum_{i,j} G[g,i] G[g,j] C_c((x_i - x_j) mod domain),
        // C_c the covariance map of spatial coefficient c; the other planes
        // share what is left of n times the patch variance C_c(0)
        // lag[i * lrow + j]: the pair's map row; rows x P may exceed 32 bits (a lag
        // domain of 258^3 and 125 coefficients do), so offsets are formed in 64
        int* lag = sm<int>(smem, a.L.lag);
        const int lrow = (n + 3) / 4 * 4;
        if (kk > 0) {
            for (int q = tid; q < n * n; q += blockDim.x) {
                const int i = q / n, j = q - i * n;
                if (j >= i) continue;
                int flat = 0;
                for (int d = 0; d < geo.nd(); ++d) {
                    const int D = sp.cov_domain[d];
                    int l = (pos[i * BMND_MAX_DIMS + d] - pos[j * BMND_MAX_DIMS + d]) % D;
                    if (l < 0) l += D;
                    flat = flat * D + l;
                }
                lag[i * lrow + j] = flat;
            }
            __syncthreads();
        }
        const float* cm = sp.cov_maps;
        if (kk > 0 && sp.group_transform == BMND_GROUP_HAAR && is_pow2(n) && kk <= 4 && 2 * P <= static_cast<int>(blockDim.x)) {
            gauss_haar(cm, lag, lrow, n, kk, P, G, EX);
        } else {
            // one thread per (plane, coefficient): the planes' sums are independent
            for (int t = tid; t < kk * P; t += blockDim.x) {
                const int g = t / P, c = t - g * P;
                const float pv = __ldg(cm + c);  // lag 0: the patch variance of coefficient c
                const float* Gr = G + g * n;
                float value = 0.0f;
                for (int i = 0; i < n; ++i) {
                    const float wi = Gr[i];
                    if (wi == 0.0f) continue;
                    value = add_rn(value, mul_rn(mul_rn(wi, pv), wi));
                    for (int j = 0; j < i; ++j) {
                        const float wj = Gr[j];
                        if (wj == 0.0f) continue;
                        const float cv = __ldg(cm + static_cast<int64_t>(lag[i * lrow + j]) * P + c);
                        value = add_rn(value, mul_rn(mul_rn(wi, wj), add_rn(cv, cv)));
                    }
                }
                EX[g * P + c] = fmaxf(value, 0.0f);
            }
        }
        __syncthreads();
        // the other planes' standard deviation, parked in X (not gathered yet)
        for (int c = tid; c < P; c += blockDim.x) {
            const float pv = __ldg(cm + c);
            float ex_sum = 0.0f;
            for (int g = 0; g < kk; ++g) ex_sum = add_rn(ex_sum, EX[g * P + c]);
            float rest = pv;
            if (kk > 0 && kk < n) {
                rest = div_rn(sub_rn(mul_rn(static_cast<float>(n), pv), ex_sum), static_cast<float>(n - kk));
                rest = fmaxf(rest, 0.0f);
            }
            X[c] = sqrtf(fmaxf(rest, 0.0f));
        }
        __syncthreads();
        geo.each(n, [&](int g, int c, int e) { S[e] = g < kk ? sqrtf(EX[g * P + c]) : X[c]; });
        __syncthreads();
    }

    // ---- union voxels and the exact overlap-aware sigma of the first kk planes ----
    // (with exact risk weights under white Gaussian noise: the union voxels
    // alone, each with the noise variance, variance.py:1451-1496)
    int U = 0;
    if ((!gauss || exact_risk) && kk > 0) {
        int ush[BMND_MAX_DIMS] = {1, 1, 1}, org[BMND_MAX_DIMS] = {0, 0, 0};
        int ucells = 1;
        for (int d = 0; d < geo.nd(); ++d) {
            ush[d] = misc[4 + d];
            org[d] = misc[d];
            ucells *= ush[d];
        }
        // A union cell's members are those whose patch reaches its coordinate on
        // every axis: one member mask per axis coordinate, ANDed per cell.
        int aoff[BMND_MAX_DIMS] = {0, 0, 0}, masks = 0;
        for (int d = 0; d < geo.nd(); ++d) {
            aoff[d] = masks;
            masks += ush[d];
        }
        {
            const int nw = blockDim.x >> 5, warp = tid >> 5, lane = tid & 31;
            for (int q = warp; q < masks; q += nw) {
                int d = 0;
#pragma unroll
                for (int t = 1; t < BMND_MAX_DIMS; ++t)
                    if (t < geo.nd() && q >= aoff[t]) d = t;
                const int c = q - aoff[d];
                const int bd = geo.b(d);
                const bool in = lane < n && static_cast<unsigned>(c - shf[lane * BMND_MAX_DIMS + d]) < static_cast<unsigned>(bd);
                const uint32_t m = __ballot_sync(0xffffffffu, in);
                if (lane == 0) grid[q] = m;
            }
        }
        __syncthreads();
        // Occupied cells (ascending) and their entries (ascending member): thread t
        // takes a contiguous 1/NT of the cells, counts its voxels and entries, gets
        // its offsets from a block scan and writes them.  The voxel's offset in the
        // volume is parked in lval until the variance pass below.
        {
            const int last = geo.nd() - 1;
            const int cpt = (ucells + static_cast<int>(blockDim.x) - 1) / static_cast<int>(blockDim.x);
            const int c0 = min(ucells, tid * cpt), c1 = min(ucells, c0 + cpt);
            const uint32_t* xm = grid + aoff[last];
            const int ux = ush[last];
            // walk(f): f(mask, position) over this thread's occupied cells
            auto walk = [&](auto f) {
                int cc[BMND_MAX_DIMS] = {0, 0, 0};
                int rem = c0;
#pragma unroll
                for (int d = BMND_MAX_DIMS - 1; d >= 0; --d) {
                    if (d < geo.nd()) {
                        const int q = d > 0 ? small_div(rem, 1.0f / static_cast<float>(ush[d])) : 0;
                        cc[d] = rem - q * ush[d];
                        rem = q;
                    }
                }
                int c = c0;
                while (c < c1) {
                    uint32_t outer = 0xffffffffu;
                    int vox = 0, lin = 0;
#pragma unroll
                    for (int d = 0; d < BMND_MAX_DIMS; ++d) {
                        if (d < last) {
                            outer &= grid[aoff[d] + cc[d]];
                            vox += (cc[d] + org[d]) * static_cast<int>(a.vstride[d]);
                            lin += cc[d] * geo.inner(d);
                        }
                    }
                    const int x = cc[last];
                    const int run = min(ux - x, c1 - c);
                    if (outer) {
                        for (int k = 0; k < run; ++k) {
                            const uint32_t m = outer & xm[x + k];
                            if (m) f(m, vox + x + k + org[last], lin + x + k);
                        }
                    }
                    c += run;
                    cc[last] = 0;
#pragma unroll
                    for (int d = BMND_MAX_DIMS - 1; d >= 0; --d) {
                        if (d < last) {
                            if (++cc[d] < ush[d]) break;
                            cc[d] = 0;
                        }
                    }
                }
            };
            uint32_t mine = 0;  // voxels << 16 | entries (both below 2^15)
            walk([&](uint32_t m, int, int) { mine += 0x10000u + static_cast<uint32_t>(__popc(m)); });
            const int nw = blockDim.x >> 5, warp = tid >> 5, lane = tid & 31;
            uint32_t incl = mine;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += t;
            }
            if (lane == 31) scan[warp].x = static_cast<int>(incl);
            __syncthreads();
            uint32_t base = 0, all = 0;
            for (int w = 0; w < nw; ++w) {
                const uint32_t t = static_cast<uint32_t>(scan[w].x);
                if (w < warp) base += t;
                all += t;
            }
            base += incl - mine;
            int w = static_cast<int>(base >> 16), we = static_cast<int>(base & 0xffffu);
            const int* shl = sm<int>(smem, a.L.shl);
            const uint32_t gt2_off = static_cast<uint32_t>(a.L.gt2), row_b = 4u * static_cast<uint32_t>(kron_stride(P));
            const int lg = ilog2_floor(n);
            walk([&](uint32_t m, int vox, int lin) {
                reinterpret_cast<int*>(lval)[w] = vox;
                lstart[w++] = we;
                do {
                    const int g = __ffs(m) - 1;
                    m &= m - 1;
                    const uint32_t pe = static_cast<uint32_t>(lin - shl[g]);
                    lent[we++] = quarters ? pe * row_b + static_cast<uint32_t>((4 * g) >> lg)
                                          : gt2_off + static_cast<uint32_t>(g * kpad * 8) + (pe << 16);
                } while (m);
            });
            if (tid == 0) {
                scan[kThreads / 32] = make_int2(static_cast<int>(all >> 16), static_cast<int>(all & 0xffffu));
                lent[all & 0xffffu] = lent[(all & 0xffffu) + 1] = quarters ? 0u : gt2_off;  // read ahead, never used
            }
        }
        __syncthreads();
        U = scan[kThreads / 32].x;
        if (tid == 0) lstart[U] = scan[kThreads / 32].y;
        __syncthreads();
        // variance of every union voxel, all loads in flight together
        for (int u = tid; u < U; u += blockDim.x) {
            if (gauss) {
                lval[u] = sp.exact_source_variance;
                continue;
            }
            const int vox = reinterpret_cast<const int*>(lval)[u];
            lval[u] = variance_of(__ldg(varsrc + vox), scale_f, floor_f);
        }
        __syncthreads();
        if (gauss) {
            // sigma comes from the covariance maps
        } else if constexpr (ND > 0) {
            exact_planes_any<kron_jr(B0 * B1 * B2)>(smem, quarters, G[0], kk > 2 ? G[2 * n] : 0.0f,
                                                    static_cast<uint32_t>(a.L.kron), lval, lstart, lent, U, kk, a.st,
                                                    P, EX, sm<float>(smem, a.L.part), a.L.part_over != 0);
        } else {
            const int jr = kron_jr(P);
            float* part = sm<float>(smem, a.L.part);
            if (jr == 1) exact_planes_any<1>(smem, false, 0.0f, 0.0f, 0u, lval, lstart, lent, U, kk, a.st, P, EX, part, a.L.part_over != 0);
            else if (jr == 2) exact_planes_any<2>(smem, false, 0.0f, 0.0f, 0u, lval, lstart, lent, U, kk, a.st, P, EX, part, a.L.part_over != 0);
            else exact_planes_any<4, 4>(smem, false, 0.0f, 0.0f, 0u, lval, lstart, lent, U, kk, a.st, P, EX, part, a.L.part_over != 0);
        }
    }

    // ---- approximate sigma from the variance group (squared transforms) ----
    // (after the exact phase: S shares the union region with its lists)
    // The observation (and the pilot) are gathered here too, so the volume the
    // variance comes from is read once (its lists are no longer needed).
    bool gathered = false, wild = false;
    bool fused = false;  // X and R already forward-transformed with S
    if (!gauss && need_approx) {
        geo.each(n, [&](int g, int p, int e) {
            const int off = org0[g] + voff[p];
            const float vs = __ldg(varsrc + off);
            const float vv = variance_of(vs, scale_f, floor_f);
            const float xv = varsrc == a.noisy ? vs : __ldg(a.noisy + off);
            const float rv = !wiener ? 0.0f : (varsrc == a.pilot ? vs : __ldg(a.pilot + off));
            S[e] = vv;
            X[e] = xv;
            if (wiener) R[e] = rv;
            wild |= !(vv < 1e30f && fabsf(xv) < 1e30f && fabsf(rv) < 1e30f);
        });
        if (wild) misc[kMiscWild] = 1;
        gathered = true;
        __syncthreads();
        fused = transform_forward_all<ND, B0, B1, B2>(geo, a, smem, n, S, X, wiener ? R : nullptr);
        if (!fused) transform_group<ND, B0, B1, B2>(geo, a, smem, n, S, 2);
        geo.each(n, [&](int, int, int e) {
            const float v = S[e];
            S[e] = sqrtf(v > 0.0f ? v : 0.0f);
        });
        __syncthreads();
    }

    // ---- final sigma in S (plane limiting, variance.py:1572-1631) ----
    if (gauss) {
        // done above
    } else if (k > 0 && kk == n) {
        geo.each(n, [&](int g, int p, int e) { S[e] = EX[g * P + p]; });
    } else if (k > 0) {
        // TPJ threads per coefficient j (neighbouring lanes), each summing the
        // planes i = sub (mod TPJ); the partial sums are added by shuffles in
        // a fixed order, and each thread rescales its own planes
        const int TPJ = P <= 64 ? 4 : (P <= 128 ? 2 : 1);
        for (int base = 0; base < P * TPJ; base += blockDim.x) {
            const int t = base + tid;
            const int j = t / TPJ, sub = t - j * TPJ;
            const bool live = j < P;
            float sum_a = 0.0f, sum_e = 0.0f, rem_a = 0.0f;
            if (live) {
                for (int i = sub; i < n; i += TPJ) {
                    const float sa = fmaxf(S[geo.at(i, j)], 0.0f);
                    const float va = mul_rn(sa, sa);
                    sum_a = add_rn(sum_a, va);
                    if (i >= kk) rem_a = add_rn(rem_a, va);
                }
                for (int i = sub; i < kk; i += TPJ) {
                    const float se = fmaxf(EX[i * P + j], 0.0f);
                    sum_e = add_rn(sum_e, mul_rn(se, se));
                }
            }
            for (int o = 1; o < TPJ; o <<= 1) {
                sum_a = add_rn(sum_a, __shfl_xor_sync(0xffffffffu, sum_a, o));
                sum_e = add_rn(sum_e, __shfl_xor_sync(0xffffffffu, sum_e, o));
                rem_a = add_rn(rem_a, __shfl_xor_sync(0xffffffffu, rem_a, o));
            }
            if (!live) continue;
            float target = sub_rn(sum_a, sum_e);
            if (target < 0.0f) target = 0.0f;
            const float scl = rem_a > 0.0f ? div_rn(target, rem_a) : 0.0f;
            for (int i = sub; i < n; i += TPJ) {
                float v;
                if (i < kk) {
                    const float se = fmaxf(EX[i * P + j], 0.0f);
                    v = mul_rn(se, se);
                } else if (rem_a > 0.0f) {
                    const float sa = fmaxf(S[geo.at(i, j)], 0.0f);
                    v = mul_rn(mul_rn(sa, sa), scl);
                } else {
                    v = div_rn(target, static_cast<float>(n - kk));
                }
                S[geo.at(i, j)] = sqrtf(v > 0.0f ? v : 0.0f);
            }
        }
    }
    __syncthreads();

    // ---- gather and forward-transform the observation (and the pilot) ----
    if (!gathered) {
        geo.each(n, [&](int g, int p, int e) {
            const int off = org0[g] + voff[p];
            const float xv = __ldg(a.noisy + off);
            const float rv = wiener ? __ldg(a.pilot + off) : 0.0f;
            X[e] = xv;
            if (wiener) R[e] = rv;
            wild |= !(fabsf(xv) < 1e30f && fabsf(rv) < 1e30f);
        });
        if (wild) misc[kMiscWild] = 1;
        __syncthreads();
    }
    if (!fused) {
        transform_group<ND, B0, B1, B2>(geo, a, smem, n, X, 0);
        if (wiener) transform_group<ND, B0, B1, B2>(geo, a, smem, n, R, 0);
    }
    const int64_t probe_base = gid * static_cast<int64_t>(a.nmax) * P;
    if (a.probe.active) {
        geo.each(n, [&](int g, int p, int e) {
            if (a.probe.coef) a.probe.coef[probe_base + g * P + p] = X[e];
            if (a.probe.sigma) a.probe.sigma[probe_base + g * P + p] = S[e];
        });
    }

    // ---- shrinkage: coefficients in X, attenuation in V, and in S each
    // coefficient's aggregation error: a^2 (classic), a^2 sigma^2 (variance) or
    // a^2 sigma^2 + (1 - a)^2 signal power (risk) (aggregationweights.py:213-259) ----
    const float eps_f = static_cast<float>(sp.eps);
    float* SG = sm<float>(smem, a.L.sg);
    float sig_sum = 0.0f;  // Wiener sigma map: this thread's share of the group's sigma sum
    geo.each(n, [&](int g, int p, int e) {
        float sig = S[e];
        if (a.sig_num) {
            if (wiener) sig_sum += sig;
            else SG[e] = sig;
        }
        float nv = mul_rn(sig, sig);
        float att;
        float spw = 0.0f;  // Wiener signal power (risk weights)
        if (!wiener && sp.soft_threshold) {
            // soft thresholding (bmndalgo.py:476-486): sign(c) max(|c| - lambda sigma, 0)
            const float thr = mul_rn(sp.ht_lambda, sig);
            const float mag = fabsf(X[e]);
            const float shr = fmaxf(sub_rn(mag, thr), 0.0f);
            att = mag > 0.0f ? div_rn(shr, mag) : 0.0f;
            X[e] = copysignf(shr, X[e]);
            V[e] = att;
            S[e] = sp.weight_model == BMND_WEIGHT_CLASSIC ? att * att : att * att * nv;
            if (exact_risk && g < kk) S[e] = 0.0f;  // the exact pass below holds these planes' noise
            return;
        } else if (!wiener && gauss) {
            // |c| >= lambda sigma, the group DC always kept (bmndalgo.py:462-475)
            float thr = mul_rn(sp.ht_lambda, sig);
            att = (fabsf(X[e]) >= thr || (g == 0 && p == 0)) ? 1.0f : 0.0f;
        } else if (!wiener) {
            float thr = mul_rn(sp.ht_lambda, sig);
            att = ht_keep(fabsf(X[e]), thr, sp.count_scale, scale_f) ? 1.0f : 0.0f;
        } else if (gauss) {
            // |R|^2 / (|R|^2 + mu^2 max(sigma^2, 1e-8)) (wiener.py:50-69)
            float eff = mul_rn(sp.wiener_scale, fmaxf(nv, fmaxf(eps_f, 1e-8f)));
            float pr = fabsf(R[e]);
            pr = mul_rn(pr, pr);
            float den = add_rn(pr, eff);
            float gain = den > 0.0f ? div_rn(pr, den) : 0.0f;
            att = fminf(fmaxf(gain, 0.0f), 1.0f);
            spw = pr;
        } else {
            // signal power by gain mode (wiener.py:24-47)
            float eff = mul_rn(sp.wiener_scale, nv);
            float pr = fabsf(R[e]);
            pr = mul_rn(pr, pr);
            float spow = pr;
            if (sp.wiener_gain_mode != BMND_GAIN_CLASSIC) {
                spow = sub_rn(pr, sp.wiener_gain_mode == BMND_GAIN_NOISE_FLOOR ? nv : eff);
                if (spow < 0.0f) spow = 0.0f;
            }
            float gain = div_rn(spow, add_rn(add_rn(spow, eff), eps_f));
            att = fminf(fmaxf(gain, 0.0f), 1.0f);
            spw = spow;
        }
        X[e] = mul_rn(X[e], att);
        V[e] = att;
        float err = att * att;
        if (sp.weight_model != BMND_WEIGHT_CLASSIC) err *= nv;
        // exact risk weights: the noise of the first kk planes comes from the
        // exact pass below; their bias term stays (wiener.py:760-797)
        if (exact_risk && g < kk) err = 0.0f;
        if (sp.weight_model == BMND_WEIGHT_RISK) {
            const float rj = 1.0f - att;
            err += rj * rj * spw;
        }
        S[e] = err;
    });
    __syncthreads();

    // ---- exact noise risk of the first kk planes (wiener.py:638-711) ----
    // (stages with exact risk weights run the runtime-geometry instantiation,
    // so the specialised ones carry none of this code)
    double* riskp = sm<double>(smem, a.L.risk);
    if constexpr (ND == 0) {
        if (exact_risk) {
            const float* smt = a.st + static_cast<int64_t>(P) * kron_stride(P);
            const int jr = kron_jr(P);
            if (jr == 1) exact_risk_any<1>(smem, lval, lstart, lent, U, kk, a.st, smt, V, P, riskp);
            else if (jr == 2) exact_risk_any<2>(smem, lval, lstart, lent, U, kk, a.st, smt, V, P, riskp);
            else exact_risk_any<4>(smem, lval, lstart, lent, U, kk, a.st, smt, V, P, riskp);
        }
    }

    if (a.probe.active && a.probe.atten)
        geo.each(n, [&](int g, int p, int e) { a.probe.atten[probe_base + g * P + p] = V[e]; });

    // Wiener sigma map: the group's mean coefficient sigma (bmndalgo.py:874-875),
    // summed per warp and then over warps in warp order
    if (a.sig_num && wiener) {
        float v = sig_sum;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if ((tid & 31) == 0) sm<float>(smem, a.L.scan)[tid >> 5] = v;
        __syncthreads();
        if (tid == 0) {
            float t = 0.0f;
            for (int w = 0; w < static_cast<int>(blockDim.x >> 5); ++w) t += sm<float>(smem, a.L.scan)[w];
            sm<float>(smem, a.L.misc)[12] = t / static_cast<float>(total);
        }
        __syncthreads();
    }

    // ---- aggregation weights (aggregationweights.py:213-259) ----
    // The reference sums the plane risks in float64.  Here the per-coefficient
    // products and sums are float32 (relative error ~P 2^-24 in a weight, far
    // inside the output tolerance): float64 arithmetic runs at a small
    // fraction of the FP32 rate on this GPU and dominated the filter's time.
    {
        const int warp = tid >> 5, lane = tid & 31, nwarps = blockDim.x >> 5;
        for (int g = warp; g < n; g += nwarps) {
            float risk = 0.0f;
            for (int j = lane; j < P; j += 32) {
                float err = S[geo.at(g, j)];
                if (sp.windowed_synthesis) err *= static_cast<float>(mdiag[j]);
                risk += err;
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) risk += __shfl_xor_sync(0xffffffffu, risk, o);
            if (lane == 0) plane[g] = static_cast<double>(risk);
        }
    }
    __syncthreads();
    if (tid < n) {
        float risk = 0.0f;
        if (exact_risk) {
            // one weight for the group: its exact risk in float64
            // (wiener.py:760-822, aggregationweights.py:656-676)
            double r = riskp[blockDim.x >> 5];
            for (int g = 0; g < n; ++g) r += plane[g];
            risk = static_cast<float>(r);
        } else if (sp.weight_group_scope) {
            // one weight for the whole group: the summed risk (the group
            // transforms are orthonormal, so the group metric is the identity)
            for (int g = 0; g < n; ++g) risk += static_cast<float>(plane[g]);
        } else {
            for (int g = 0; g < n; ++g) {
                const float gi = G[g * n + tid];  // Ginv[o, g] = G[g, o]
                risk = fmaf(gi * gi, static_cast<float>(plane[g]), risk);
            }
        }
        wts[tid] = (isfinite(risk) && risk >= 0.0f) ? 1.0f / (risk + static_cast<float>(sp.eps)) : 0.0f;
    }
    __syncthreads();

    // ---- group-mass conservation, second pass (poisson.py:161-265) ----
    if (a.den_ro) {
        float* dirv = sm<float>(smem, a.L.dir);  // [n] group axis, then [MAX_DIMS][MAX_EDGE] patch axes
        double* red = sm<double>(smem, a.L.plane);  // reduction scratch: 5 sums per warp
        // constant synthesis direction: per axis solve(inverse, 1) = forward 1
        // (G on the group axis, the forward spatial matrix on each patch axis)
        if (tid < n) {
            float sgv = 0.0f;
            for (int j = 0; j < n; ++j) sgv += G[tid * n + j];
            dirv[tid] = a.sp.group_transform == BMND_GROUP_NONE ? 1.0f : sgv;
        }
        if (tid >= 64 && tid < 64 + BMND_MAX_DIMS * BMND_MAX_EDGE) {
            const int d = (tid - 64) / BMND_MAX_EDGE, k = (tid - 64) % BMND_MAX_EDGE;
            float v = 0.0f;
            if (d < geo.nd() && k < geo.b(d))
                for (int m = 0; m < geo.b(d); ++m) v += Fw[d * BMND_MAX_EDGE * BMND_MAX_EDGE + k * geo.b(d) + m];
            dirv[BMND_MAX_STACK + d * BMND_MAX_EDGE + k] = v;
        }
        // output functional O = w_g win[p] / den (float32 arithmetic, as the
        // reference's gather), into S; the target sum(O x noisy) in float64
        double t_target = 0.0;
        geo.each(n, [&](int g, int p, int e) {
            const int64_t off = geo.offset(pos + g * BMND_MAX_DIMS, p, a.vstride);
            const float o = (wts[g] * win[p]) / static_cast<float>(a.den_ro[off]);
            S[e] = o;
            t_target += static_cast<double>(o) * static_cast<double>(__ldg(a.noisy + off));
        });
        __syncthreads();
        transform_group<ND, B0, B1, B2>(geo, a, smem, n, S, 3);  // coefficient functional F
        __syncthreads();
        float dmax_g = 0.0f, dmax_s = 1.0f;
        for (int g = 0; g < n; ++g) dmax_g = fmaxf(dmax_g, fabsf(dirv[g]));
        for (int d = 0; d < geo.nd(); ++d) {
            float m = 0.0f;
            for (int k = 0; k < geo.b(d); ++k) m = fmaxf(m, fabsf(dirv[BMND_MAX_STACK + d * BMND_MAX_EDGE + k]));
            dmax_s *= m;
        }
        const float dmax = dmax_g * dmax_s;
        auto dir_of = [&](int g, int p) -> float {
            float v = dirv[g];
#pragma unroll
            for (int d = BMND_MAX_DIMS - 1; d >= 0; --d) {
                if (d < geo.nd()) {
                    v *= dirv[BMND_MAX_STACK + d * BMND_MAX_EDGE + p % geo.b(d)];
                    p /= geo.b(d);
                }
            }
            return v / dmax;
        };
        double t_cur = 0.0, t_den = 0.0, t_resp = 0.0;
        float t_max = 0.0f;
        geo.each(n, [&](int g, int p, int e) {
            const double f = static_cast<double>(S[e]);
            t_cur += f * static_cast<double>(X[e]);
            t_den += f * f;
            t_resp += f * static_cast<double>(dir_of(g, p));
            t_max = fmaxf(t_max, fabsf(S[e]));
        });
        const int warp = tid >> 5, lane = tid & 31, nwarps = blockDim.x >> 5;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            t_target += __shfl_xor_sync(0xffffffffu, t_target, o);
            t_cur += __shfl_xor_sync(0xffffffffu, t_cur, o);
            t_den += __shfl_xor_sync(0xffffffffu, t_den, o);
            t_resp += __shfl_xor_sync(0xffffffffu, t_resp, o);
            t_max = fmaxf(t_max, __shfl_xor_sync(0xffffffffu, t_max, o));
        }
        __syncthreads();  // red aliases plane[], last read by the weights
        if (lane == 0) {
            red[warp * 5 + 0] = t_target;
            red[warp * 5 + 1] = t_cur;
            red[warp * 5 + 2] = t_den;
            red[warp * 5 + 3] = t_resp;
            red[warp * 5 + 4] = static_cast<double>(t_max);
        }
        __syncthreads();
        if (tid == 0) {
            double target = 0.0, cur = 0.0, fden = 0.0, resp = 0.0, fmx = 0.0;
            for (int w = 0; w < nwarps; ++w) {
                target += red[w * 5 + 0];
                cur += red[w * 5 + 1];
                fden += red[w * 5 + 2];
                resp += red[w * 5 + 3];
                fmx = fmax(fmx, red[w * 5 + 4]);
            }
            double corr = 0.0;
            bool ok = true;
            if (fden <= sp.eps) {
                // rescale a vanishing functional by its largest entry
                if (!(fmx > 0.0) || !isfinite(fmx)) ok = false;
                else {
                    target /= fmx;
                    cur /= fmx;
                    resp /= fmx;
                }
            }
            const double residual = target - cur;
            if (ok && residual != 0.0) {
                if (!(resp != 0.0) || !isfinite(resp)) ok = false;
                else corr = residual / resp;
            }
            if (!ok && a.err) atomicExch(a.err, 1);
            red[0] = ok ? corr : 0.0;
        }
        __syncthreads();
        const double corr = red[0];
        if (corr != 0.0)
            geo.each(n, [&](int g, int p, int e) {
                X[e] = static_cast<float>(static_cast<double>(X[e]) + corr * static_cast<double>(dir_of(g, p)));
            });
        __syncthreads();
    }

    // ---- inverse transform and scatter ----
    transform_group<ND, B0, B1, B2>(geo, a, smem, n, X, 1);
    if (a.probe.active) {
        if (a.probe.weights && tid < n) a.probe.weights[gid * static_cast<int64_t>(a.nmax) + tid] = wts[tid];
        if (a.probe.filt)
            geo.each(n, [&](int g, int p, int e) { a.probe.filt[probe_base + g * P + p] = X[e]; });
        return;
    }
    if (a.store.store) {
        // deterministic aggregation: every member's weighted filtered patch
        // goes to the store row of its entry; the sums happen in aggregate.cu
        int* slot = sm<int>(smem, a.L.shl);  // free after the exact phase
        if (tid < n) {
            const int s = a.store.slot_of[gid * static_cast<int64_t>(sp.max_stack) + tid];
            slot[tid] = s;
            a.store.wstore[s] = wts[tid];
        }
        __syncthreads();
        geo.each(n, [&](int g, int p, int e) {
            a.store.store[static_cast<int64_t>(slot[g]) * a.store.row + p] = mul_rn(X[e], mul_rn(wts[g], win[p]));
        });
        return;
    }
    geo.each(n, [&](int g, int p, int e) {
        const int64_t off = geo.offset(pos + g * BMND_MAX_DIMS, p, a.vstride);
        float ww = mul_rn(wts[g], win[p]);
        atomicAdd(a.num + off, widen_f64(mul_rn(X[e], ww)));
        if (a.den_ro) return;  // the re-aggregation pass adds to the numerator only
        atomicAdd(a.den + off, widen_f64(ww));
        if (a.sig_num) {
            // sigma map numerator (patchaggregation.py:229-294): per coefficient
            // (hard thresholding) or the group's mean (Wiener)
            const float sv = wiener ? sm<float>(smem, a.L.misc)[12] : SG[e];
            atomicAdd(a.sig_num + off, widen_f64(mul_rn(sv, ww)));
        }
    });
}

// One CTA per group, CTAS resident.  (Persistent CTAs walking the groups, which would set up the
// constants once, spill: the compiler then keeps 1.9 KB of local memory a thread.)
// Resident CTAs per SM cover each other's barriers and serial phases: 64
// registers and 38 KB (16 members) or 56 KB (32) allow four for patches of 64
// elements (against three: 75.1 -> 72.3 ms for 0.93 M groups of 8x8, 3.56 -> 3.38
// ms for 42 K groups of 4x4x4, 14.3 -> 12.6 ms for a Gaussian image); 5x5x5
// patches hold three, and four where there are no exact planes (55 KB; 17.2 ->
// 14.8 ms for 250 K groups).
// 8x8 stages whose exact planes take the general stream (more than four, or no Haar
// group) hold three: at 64 registers its loop spills and four CTAs of 51 KB leave L1
// 28 KB for S^T and the volumes (220 x 260, 32 members: 8 planes 3.12 -> 2.75 ms, 16
// planes 6.69 -> 4.05, 32 planes 8.77 -> 6.61, DCT group 2.50 -> 2.40).
template <int ND, int B0, int B1, int B2, int NT, int CTAS, bool APPROX = false>
__global__ void __launch_bounds__(NT, CTAS)
    group_filter_kernel(FilterArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    filter_group<ND, B0, B1, B2, APPROX>(a, smem, blockIdx.x);
}

// S^T[p * stride + j] = S[j, p] with S = kron(F_0, ..., F_{nd-1}) built axis by
// axis in float32 (fl(fl(F0 * F1) * F2)), as the reference builds its spatial
// matrix (variance.py:744-755); columns j >= P of the padded rows are zero
__global__ void spatial_kron_kernel(BmndStageParams sp, int P, int stride, float* st) {
    if (blockIdx.x == 0 && P >= 64 && !sp.exact_risk_weights) {
        // the matrices and the window as a table after S^T (the place of the risk metric)
        constexpr int E1 = BMND_MAX_EDGE * BMND_MAX_EDGE, EE = BMND_MAX_DIMS * E1;
        float* tab = st + static_cast<int64_t>(P) * stride;
        for (int e = threadIdx.x; e < EE; e += blockDim.x) {
            tab[e] = sp.spatial_fwd[e / E1][e % E1];
            tab[EE + e] = sp.spatial_inv[e / E1][e % E1];
        }
        for (int e = threadIdx.x; e < P; e += blockDim.x) tab[2 * EE + e] = sp.window[e];
    }
    for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < P * stride; idx += gridDim.x * blockDim.x) {
        const int p = idx / stride, j = idx % stride;
        if (j >= P) {
            st[idx] = 0.0f;
            continue;
        }
        int jd[BMND_MAX_DIMS], pd[BMND_MAX_DIMS];
        int rj = j, rp = p;
        for (int d = sp.ndim - 1; d >= 0; --d) {
            jd[d] = rj % sp.block[d];
            rj /= sp.block[d];
            pd[d] = rp % sp.block[d];
            rp /= sp.block[d];
        }
        float v = sp.spatial_fwd[0][jd[0] * sp.block[0] + pd[0]];
        for (int d = 1; d < sp.ndim; ++d) v = mul_rn(v, sp.spatial_fwd[d][jd[d] * sp.block[d] + pd[d]]);
        st[idx] = v;
    }
}

// risk metric SM = S_inv^T diag(w^2) S_inv of the windowed synthesis
// (variance.py:1546-1557): S_inv the Kronecker product of the inverse patch
// matrices (float32 products in axis order, variance.py:744-755), w^2 and
// w^2 S_inv rounded to float32 as the reference's, each entry summed in
// float64 and rounded once.  Row p at sm[p * stride], zero beyond column P.
__global__ void risk_metric_kernel(BmndStageParams sp, int P, int stride, float* sm) {
    auto synth = [&](int x, int c) {
        int xd[BMND_MAX_DIMS], cd[BMND_MAX_DIMS];
        for (int d = sp.ndim - 1; d >= 0; --d) {
            xd[d] = x % sp.block[d];
            x /= sp.block[d];
            cd[d] = c % sp.block[d];
            c /= sp.block[d];
        }
        float v = sp.spatial_inv[0][xd[0] * sp.block[0] + cd[0]];
        for (int d = 1; d < sp.ndim; ++d) v = mul_rn(v, sp.spatial_inv[d][xd[d] * sp.block[d] + cd[d]]);
        return v;
    };
    for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < P * stride; idx += gridDim.x * blockDim.x) {
        const int p = idx / stride, j = idx % stride;
        if (j >= P) {
            sm[idx] = 0.0f;
            continue;
        }
        double acc = 0.0;
        for (int x = 0; x < P; ++x) {
            const float w2 = mul_rn(sp.window[x], sp.window[x]);
            acc += static_cast<double>(synth(x, p)) * static_cast<double>(mul_rn(w2, synth(x, j)));
        }
        sm[idx] = static_cast<float>(acc);
    }
}

// every group size's group matrix, n = 1 .. BMND_MAX_STACK (group_table_offset)
__global__ void group_table_kernel(int kind, float* __restrict__ gtab) {
    for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < kGroupTableFloats; idx += gridDim.x * blockDim.x) {
        int n = 1;
        while (group_table_offset(n + 1) <= idx) ++n;
        const int e = idx - group_table_offset(n);
        gtab[idx] = group_entry(kind, n, e / n, e % n);
    }
}

__global__ void finalize_kernel(const double* __restrict__ num, const double* __restrict__ den,
                                const float* __restrict__ noisy, float* __restrict__ out,
                                int64_t n, float eps_f, int no_eps) {
    for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        float d = static_cast<float>(den[i]);
        // mass conservation divides without eps (bmndalgo.py:617-624)
        out[i] = d > 0.0f ? div_rn(static_cast<float>(num[i]), no_eps ? d : add_rn(d, eps_f)) : noisy[i];
    }
}

// sigma map = sigma_num / den where den > 0, else the global sigma
// (bmndalgo.py:1048-1057)
__global__ void finalize_sigma_kernel(const double* __restrict__ sig_num, const double* __restrict__ den,
                                      float global_sigma, float* __restrict__ out, int64_t n) {
    for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const float d = static_cast<float>(den[i]);
        out[i] = d > 0.0f ? div_rn(static_cast<float>(sig_num[i]), d) : global_sigma;
    }
}

}  // namespace

int64_t union_cells_bound(const BmndStageParams& sp) {
    int64_t u = 1;
    for (int d = 0; d < sp.ndim; ++d) {
        int counts = sp.shape[d] - sp.block[d] + 1;
        int span = 2 * sp.search_radius[d];
        if (span > counts - 1) span = counts - 1;
        u *= span + sp.block[d];
    }
    return u;
}

int64_t group_filter_smem_bytes(const BmndStageParams& sp) {
    int P = patch_volume(sp);
    int kmax = sp.variance_k < sp.max_stack ? sp.variance_k : sp.max_stack;
    if (kmax < 0) kmax = 0;
    return make_layout(sp, P, sp.max_stack, kmax, union_cells_bound(sp), true).total;
}

int32_t launch_group_filter(const BmndStageParams& sp, const float* noisy, const float* pilot,
                            const int32_t* sel, const int32_t* count, int64_t n_refs, double* num,
                            double* den, float* st, double* sig_num, cudaStream_t stream, const double* den_ro,
                            int* err, const GroupProbe* probe, const AggStore* store) {
    if (n_refs == 0) return BMND_OK;
    {
        const int P = patch_volume(sp);
        const int stride = kron_stride(P);
        spatial_kron_kernel<<<(P * stride + 255) / 256, 256, 0, stream>>>(sp, P, stride, st);
        BMND_LAUNCH_CHECK("spatial_kron_kernel");
        if (sp.exact_risk_weights) {
            risk_metric_kernel<<<(P * stride + 255) / 256, 256, 0, stream>>>(sp, P, stride,
                                                                            st + static_cast<int64_t>(P) * stride);
            BMND_LAUNCH_CHECK("risk_metric_kernel");
        }
        group_table_kernel<<<(kGroupTableFloats + 255) / 256, 256, 0, stream>>>(
            sp.group_transform, st + 2 * static_cast<int64_t>(P) * stride);
        BMND_LAUNCH_CHECK("group_table_kernel");
    }
    FilterArgs a{};
    a.st = st;
    a.sp = sp;
    a.P = patch_volume(sp);
    a.nmax = sp.max_stack;
    a.kmax = sp.variance_k < sp.max_stack ? sp.variance_k : sp.max_stack;
    if (a.kmax < 0) a.kmax = 0;
    int64_t s = 1;
    for (int d = sp.ndim - 1; d >= 0; --d) {
        a.vstride[d] = s;
        s *= sp.shape[d];
    }
    a.n_lins = 1;
    for (int d = 0; d < sp.ndim; ++d) {
        a.counts[d] = sp.shape[d] - sp.block[d] + 1;
        a.n_lins *= a.counts[d];
    }
    a.sig_num = sig_num;
    a.ucells_cap = union_cells_bound(sp);
    a.L = make_layout(sp, a.P, a.nmax, a.kmax, a.ucells_cap, sig_num != nullptr);
    a.noisy = noisy;
    a.pilot = pilot;
    a.sel = sel;
    a.count = count;
    a.n_refs = n_refs;
    a.num = num;
    a.den = den;
    a.den_ro = den_ro;
    a.err = err;
    if (probe) a.probe = *probe;
    if (store) {
        a.store = *store;
        if (sig_num || den_ro) return fail(BMND_ERR_INVALID_ARG, "the entry store excludes sigma maps and mass passes");
    }
    if (a.probe.active && den_ro) return fail(BMND_ERR_INVALID_ARG, "the group probe has no mass-conservation pass");
    if (a.L.total > 227 * 1024)
        return fail(BMND_ERR_UNSUPPORTED, "group filter shared memory exceeds 227 KB for this profile");
    if (n_refs > 0x7fffffffLL) return fail(BMND_ERR_UNSUPPORTED, "too many groups");
    auto run = [&](auto kernel, int threads) -> int32_t {
        // give shared memory only what the resident CTAs need, so the rest of
        // the unified L1 caches the Kronecker table and the volumes
        int per_sm = 0, sms = 0;
        if (int32_t rc = kernel_residency(reinterpret_cast<const void*>(kernel), threads,
                                          static_cast<size_t>(a.L.total), true, &per_sm, &sms))
            return rc;
        kernel<<<static_cast<unsigned>(n_refs), threads, a.L.total, stream>>>(a);
        BMND_LAUNCH_CHECK("group_filter_kernel");
        return BMND_OK;
    };
    if (!specialised_shape(sp)) return run(group_filter_kernel<0, 0, 0, 0, kThreads, 2>, kThreads);
    if (sp.ndim == 2) {
        const bool general = a.kmax > 0 && !a.L.kron_used && sp.noise_model == BMND_NOISE_POISSON;
        return general ? run(group_filter_kernel<2, 8, 8, 1, kThreads, 3>, kThreads)
                       : run(group_filter_kernel<2, 8, 8, 1, kThreads, 4>, kThreads);
    }
    if (sp.block[0] == 4) return run(group_filter_kernel<3, 4, 4, 4, kThreads, 4>, kThreads);
    return a.kmax > 0 ? run(group_filter_kernel<3, 5, 5, 5, kThreads, 3>, kThreads)
                      : run(group_filter_kernel<3, 5, 5, 5, kThreads, 4, true>, kThreads);
}

int32_t launch_finalize_sigma(const BmndStageParams& sp, const double* sig_num, const double* den,
                              float global_sigma, float* out, cudaStream_t stream) {
    int64_t n = volume_voxels(sp);
    if (n == 0) return BMND_OK;
    int64_t blocks = (n + 255) / 256;
    if (blocks > 152 * 16) blocks = 152 * 16;
    finalize_sigma_kernel<<<static_cast<unsigned>(blocks), 256, 0, stream>>>(sig_num, den, global_sigma, out, n);
    BMND_LAUNCH_CHECK("finalize_sigma_kernel");
    return BMND_OK;
}

int32_t launch_finalize(const BmndStageParams& sp, const double* num, const double* den,
                        const float* noisy, float* out, cudaStream_t stream) {
    int64_t n = volume_voxels(sp);
    if (n == 0) return BMND_OK;
    int threads = 256;
    int64_t blocks = (n + threads - 1) / threads;
    if (blocks > 152 * 16) blocks = 152 * 16;
    finalize_kernel<<<static_cast<unsigned>(blocks), threads, 0, stream>>>(num, den, noisy, out, n,
                                                                            static_cast<float>(sp.eps),
                                                                            sp.mass_conserve ? 1 : 0);
    BMND_LAUNCH_CHECK("finalize_kernel");
    return BMND_OK;
}

}  // namespace bmnd
