// boxmatch.cu -- exhaustive window matching by shared row sums, exact rescoring.
//
// A patch distance is a box sum of per-voxel terms t(v[y], v[y + d]) for a
// window offset d, and neighbouring references share most of those terms: the
// default schedules put a reference on every 3rd last-axis position and on
// almost every position of the axes before it, so a 5x5x5 patch needs 5 x 13.5
// / 3 = 22 new terms per reference and offset instead of 125 (2-D 8x8: 12
// instead of 64).
//
//   box_rows_*   (one CTA per tile of patch origins) writes, for every
//                reference, the screening distance of every window offset;
//   box_select_  (one warp per reference) bounds the exact float32 distance of
//                every candidate from its screening distance, rescores in the
//                exact kernel's float32 order only those whose acceptance or
//                place among the best the bounds leave open, and writes the
//                match table.  The result equals the exact kernel's bit for
//                bit; references it cannot settle (queue overflow, non-finite
//                values, duplicates) get count = -1 and are redone by it.
//
// Screening terms:
//   * squared differences of the source (SSD), or of sqrt(2 c) for the Poisson
//     deviance of real-valued sources.  With u = |r - c| / (r + c) the deviance
//     term t = 2 [r ln(2r/s) + c ln(2c/s)] and q = 2 (sqrt r - sqrt c)^2 satisfy
//     q / rho(u^2) <= t <= q, rho(w) <= 1 + 0.0834 w + 0.36 w^2 and <= 1.4427:
//     two operations per term, and tight where r and c are close, as they are
//     between patches of a stage-1 estimate;
//   * -s log2 s (one SFU operation per term) for integer counts, whose u is
//     large: t summed over the patch is 2 ln 2 [F(r) + F(c) - sum s log2 s]
//     with F the box sum of c + c log2 c, prepared once per volume.
//
// Measured (one GB300, matching of one stage, against one warp or CTA per
// reference evaluating every term): 128 x 144 x 160, 5x5x5 patches of an
// estimate 16.7 ms (rows 6.3, selection 8.4 + 1.9) against 78.6; 320 x 256,
// 8x8 patches of an estimate 0.68 ms against 3.37; 96 x 104 x 113, 4x4x4
// patches of counts 3.0 ms against 4.7 (each reference is the only one of its
// 27 origins there, so little is shared); SSD, both stages: 80 x 96 x 90
// 4.4 ms against 15.0, 768 x 640 2.2 ms against 15.2 (tensor-core products).
// A low-count volume's smooth estimate leaves hundreds of candidates per
// reference open: 90^3 at peak 5, both stages 15.3 ms against 19.4.
// No pipe is full (72 x 76 x 70, ncu): the row kernels issue 0.62-0.65 instructions
// per clock and scheduler with the 4 warps that 128 registers leave it (5x5x5 spills
// 216 bytes), waiting for shared-memory loads and dependent results; load/store pipe
// 44 %, FMA 30 %, log form's SFU 30 %.  The selection issues 0.80 (ALU 48 %, FMA
// 40 %): instructions bound it, its heavy form (0.61) the latency of its row loads.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <cmath>

#include "match_common.cuh"

namespace bmnd {
namespace {

constexpr int kG = 8;          // last-axis offsets per work unit: one 32-byte sector per reference
constexpr int kTileX = 96;     // 2-D: last-axis origins per tile (32 columns of the default step 3)
constexpr int kSelWarps = 4;   // references per CTA of the selection
constexpr int kQueue = 192;    // exact rescoring queue per reference
constexpr int kAmb = 384;      // candidates whose acceptance alone is open, per reference
constexpr int kRowThreads3 = 512, kRowThreads2 = 256;
// rows of a chunk of references where no workspace bounds them
constexpr uint64_t kRowScratch = 1ull << 30;
constexpr float kLn2x2 = 1.38629436f;
constexpr float kTinyCount = 7.88860905e-31f;  // 2^-100

__device__ float g_box_count_table[kTable * kTable];  // deviance_term(r, c), r, c < 64

struct BoxArgs {
    const float* src;
    float inv_scale;
    int32_t poisson;   // 0: SSD of the source, 1: Poisson deviance
    int32_t n[3];      // source extents; a 2-D source is (rows, 1, columns)
    int32_t cnt[3];    // patch-grid extents
    int32_t rad[3];
    int32_t nz, ny, nx;  // window offsets per axis
    int32_t px;        // nx rounded up to a multiple of kG
    int64_t rowlen;    // nz * ny * px
    int32_t* map;      // per patch origin: its reference, or -1
    int32_t* colflag;  // per last-axis position: >= 0 where a reference lies
    float* fvox;       // c + c log2 c per voxel, or null (no integer-count form)
    float* fbox;       // its box sum per patch origin
    int64_t nvox;
    int64_t lo, hi;    // references of this chunk
    float* rows;       // (hi - lo) x rowlen screening distances
    int32_t* heavy;    // references of the chunk with many open candidates
    int32_t* heavy_n;  // their number
    float* cuts;       // 3 per entry of heavy: certain-accept, certain-reject and top-list cuts
    int32_t* mode;     // per reference of the chunk: 0 SSD, 1 sqrt form, 2 log form
    const float* noise;  // SSD bias per window offset, or null
    float gamma;
    int32_t per_cta;   // selection: references per CTA (its other warps help with their rescoring)
    int32_t tz, per;   // tile origins along the first axis, first-axis offsets per CTA
    int32_t ytiles;
};

// the patch-grid position of reference r as (z, y, x); false outside the grid
__device__ __forceinline__ bool ref_position(const MatchArgs& a, const BoxArgs& b, int64_t r, int (&c)[3]) {
    const int32_t* p = a.refs + r * a.ndim;
    c[0] = p[0];
    c[1] = a.ndim == 3 ? p[1] : 0;
    c[2] = p[a.ndim - 1];
    return c[0] >= 0 && c[0] < b.cnt[0] && c[1] >= 0 && c[1] < b.cnt[1] && c[2] >= 0 && c[2] < b.cnt[2];
}

__device__ __forceinline__ int64_t grid_lin(const BoxArgs& b, int z, int y, int x) {
    return (static_cast<int64_t>(z) * b.cnt[1] + y) * b.cnt[2] + x;
}

// a negative count becomes 0, NaN stays NaN (as the exact terms treat them)
__device__ __forceinline__ float count_of(float v, float inv) {
    const float c = mul_rn(v, inv);
    return c < 0.0f ? 0.0f : c;
}

__global__ void box_prepare_kernel(MatchArgs a, BoxArgs b) {
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    const int64_t first = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    for (int64_t r = first; r < a.n_refs; r += stride) {
        int c[3];
        if (!ref_position(a, b, r, c)) continue;
        b.map[grid_lin(b, c[0], c[1], c[2])] = static_cast<int32_t>(r);
        b.colflag[c[2]] = 1;
    }
    if (!b.fvox) return;
    for (int64_t i = first; i < b.nvox; i += stride) {
        const float c = count_of(b.src[i], b.inv_scale);
        b.fvox[i] = c > 0.0f ? c + c * log2f(c) : 0.0f * c;
    }
    for (int64_t i = first; i < kTable * kTable; i += stride)
        g_box_count_table[i] = deviance_term(static_cast<float>(i / kTable), static_cast<float>(i % kTable));
}

// box sums of fvox, summed row by row (3 short chains instead of one long one,
// which keeps the rounding error of the log form's bound small)
template <int WZ, int WY, int WX>
__global__ void box_fsum_kernel(BoxArgs b) {
    const int64_t n = static_cast<int64_t>(b.cnt[0]) * b.cnt[1] * b.cnt[2];
    for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const int x = static_cast<int>(i % b.cnt[2]);
        const int y = static_cast<int>((i / b.cnt[2]) % b.cnt[1]);
        const int z = static_cast<int>(i / (static_cast<int64_t>(b.cnt[2]) * b.cnt[1]));
        float sz = 0.0f;
#pragma unroll 1
        for (int dz = 0; dz < WZ; ++dz) {
            float sy = 0.0f;
#pragma unroll
            for (int dy = 0; dy < WY; ++dy) {
                const float* row = b.fvox + (static_cast<int64_t>(z + dz) * b.n[1] + (y + dy)) * b.n[2] + x;
                float sx = 0.0f;
#pragma unroll
                for (int dx = 0; dx < WX; ++dx) sx += __ldg(row + dx);
                sy += sx;
            }
            sz += sy;
        }
        b.fbox[i] = sz;
    }
}

template <int TERM>
__device__ __forceinline__ float box_transform(float v, float inv) {
    if (TERM == 0) return v;
    const float c = count_of(v, inv);
    if (TERM == 1) return sqrtf(c + c);
    return c < kTinyCount ? kTinyCount : c;  // s log2 s of two zeros then is about -1e-28
}

// h[j] += sum over i < W of term(a[i], b[i + j]), j < kG
template <int W, int TERM, typename LA, typename LB>
__device__ __forceinline__ void row_terms(LA la, LB lb, float (&h)[kG]) {
    float bv[W + kG - 1];
#pragma unroll
    for (int k = 0; k < W + kG - 1; ++k) bv[k] = lb(k);
#pragma unroll
    for (int j = 0; j < kG; ++j) h[j] = 0.0f;
#pragma unroll
    for (int i = 0; i < W; ++i) {
        const float av = la(i);
#pragma unroll
        for (int j = 0; j < kG; ++j) {
            if (TERM == 2) {
                const float s = av + bv[i + j];
                h[j] = fmaf(-s, sfu_lg2(s), h[j]);
            } else {
                const float d = bv[i + j] - av;
                h[j] = fmaf(d, d, h[j]);
            }
        }
    }
}

// screening distances of offsets g * kG + j at (dz, dy) of the reference in
// slot `slot` at (z, y, x); offsets outside the patch grid get +infinity
template <int TERM>
__device__ __forceinline__ void store_unit(const BoxArgs& b, int slot, int z, int y, int x, int dz, int dy, int g,
                                           const float (&v)[kG]) {
    const int zc = z + dz, yc = y + dy, xc = x - b.rad[2] + g * kG;
    const bool ok = zc >= 0 && zc < b.cnt[0] && yc >= 0 && yc < b.cnt[1];
    const int jlo = -xc;                                                // first j with xc + j >= 0
    const int jhi = min(b.cnt[2] - xc, b.nx - g * kG);                  // one past the last j
    const int64_t lin = grid_lin(b, zc, yc, xc);
    float fr = 0.0f;
    if (TERM == 2) fr = __ldg(b.fbox + grid_lin(b, z, y, x));
    const int widx = ((dz + b.rad[0]) * b.ny + (dy + b.rad[1]));
    float o[kG];
#pragma unroll
    for (int j = 0; j < kG; ++j) {
        o[j] = INFINITY;
        if (ok && j >= jlo && j < jhi) {
            o[j] = v[j];
            if (TERM == 2) o[j] = kLn2x2 * ((fr + __ldg(b.fbox + lin + j)) + v[j]);
            if (TERM == 0 && b.noise)
                o[j] = sub_rn(v[j], mul_rn(b.gamma, __ldg(b.noise + static_cast<int64_t>(widx) * b.nx + g * kG + j)));
        }
    }
    float4* dst = reinterpret_cast<float4*>(b.rows + slot * b.rowlen + static_cast<int64_t>(widx) * b.px + g * kG);
    dst[0] = make_float4(o[0], o[1], o[2], o[3]);
    dst[1] = make_float4(o[4], o[5], o[6], o[7]);
}

// ---------------------------------------------------------------------------
// 3-D: a CTA takes one last-axis position x0 and a (first axis tz) x (second
// axis 33 - W) tile of origins.  A warp's lanes are 32 second-axis rows; it
// takes one (dz, dy, 8 last-axis offsets) unit at a time and marches along the
// first axis: every step sums the W terms of each row and offset (the row's
// W + 7 candidate values serve 8 W terms), the last W row sums are kept in
// registers for the first-axis sum, and the second-axis sum takes three
// shuffles.  Both tiles lie in shared memory with the second axis innermost,
// so every load is conflict-free.  One 512-thread CTA per SM: the largest
// tile keeps the halo small (32 x 32 rows for 28 x 28 origins).
// ---------------------------------------------------------------------------
template <int W, int TERM>
__device__ __forceinline__ void march3(const BoxArgs& b, const float* A, const float* B, const int32_t* map_s, int XB,
                                       int YB, int ZA, int z0, int y0, int x0, int dz, int dy, int g) {
    constexpr int RG = W - 1;
    const int lane = threadIdx.x & 31;
    float ring[RG][kG];
    for (int t0 = 0; t0 < ZA; t0 += RG) {
#pragma unroll
        for (int s = 0; s < RG; ++s) {
            const int t = t0 + s;
            if (t < ZA) {
                const float* at = A + t * (W * 32);
                const float* bt = B + t * XB * YB;
                float h[kG];
                row_terms<W, TERM>([&](int i) { return at[i * 32]; }, [&](int k) { return bt[k * YB]; }, h);
                if (t >= RG) {
                    float v[kG];
#pragma unroll
                    for (int j = 0; j < kG; ++j) {
                        float q = h[j];
#pragma unroll
                        for (int e = 0; e < RG; ++e) q += ring[e][j];
                        // second-axis box sum over lanes l .. l + W - 1
                        const float q2 = q + __shfl_down_sync(0xffffffffu, q, 1);
                        const float q4 = q2 + __shfl_down_sync(0xffffffffu, q2, 2);
                        v[j] = W == 5 ? q4 + __shfl_down_sync(0xffffffffu, q, 4) : q4;
                    }
                    const int oz = t - RG;
                    const int slot = map_s[oz * 32 + lane];
                    if (slot >= 0) store_unit<TERM>(b, slot, z0 + oz, y0 + lane, x0, dz, dy, g, v);
                }
#pragma unroll
                for (int j = 0; j < kG; ++j) ring[s][j] = h[j];
            }
        }
    }
}

template <int W>
__global__ void __launch_bounds__(kRowThreads3, 1) box_rows_3d_kernel(BoxArgs b) {
    extern __shared__ __align__(16) float smf[];
    const int x0 = blockIdx.x;
    if (b.colflag[x0] < 0) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = kRowThreads3 / 32;
    const int y0 = static_cast<int>(blockIdx.y % b.ytiles) * (33 - W);
    int z0 = static_cast<int>(blockIdx.y / b.ytiles) * b.tz;
    const int dz0 = static_cast<int>(blockIdx.z) * b.per - b.rad[0];
    const int per = min(b.per, b.rad[0] + 1 - dz0);
    const int XB = W - 1 + b.px, YB = 32 + 2 * b.rad[1];
    int32_t* map_s = reinterpret_cast<int32_t*>(smf);  // [tz][32]
    float* A = smf + b.tz * 32;                        // [ZA][W][32]
    // the tile shrinks to the first-axis range that holds references of this chunk
    __shared__ int zrange[2];
    if (tid == 0) {
        zrange[0] = b.tz;
        zrange[1] = -1;
    }
    __syncthreads();
#pragma unroll 4
    for (int i = tid; i < b.tz * 32; i += kRowThreads3) {
        const int z = z0 + i / 32, l = i % 32, y = y0 + l;
        int m = -1;
        if (l < 33 - W && z < b.cnt[0] && y < b.cnt[1]) m = b.map[grid_lin(b, z, y, x0)];
        const bool in = m >= b.lo && m < b.hi;
        map_s[i] = in ? static_cast<int32_t>(m - b.lo) : -1;
        if (__any_sync(0xffffffffu, in) && lane == 0) {
            atomicMin(&zrange[0], i / 32);
            atomicMax(&zrange[1], i / 32);
        }
    }
    __syncthreads();
    const int zfirst = zrange[0], tz = zrange[1] - zfirst + 1;
    if (zrange[1] < 0) return;
    z0 += zfirst;
    map_s += zfirst * 32;
    const int ZA = tz + W - 1, ZB = ZA + per - 1;
    float* B = A + ZA * W * 32;  // [ZB][XB][YB]
    // the tile's own values; all integers below 4096: the log form
    bool counts = b.fvox != nullptr;
#pragma unroll 4
    for (int i = tid; i < ZA * W * 32; i += kRowThreads3) {
        const int l = i % 32, k = (i / 32) % W, z = z0 + i / (32 * W), y = y0 + l;
        float v = 0.0f;
        if (z < b.n[0] && y < b.n[1]) v = __ldg(b.src + (static_cast<int64_t>(z) * b.n[1] + y) * b.n[2] + x0 + k);
        if (counts) {
            const float c = count_of(v, b.inv_scale);
            counts = c < 4096.0f && rintf(c) == c;
        }
        A[i] = v;
    }
    const int term = b.poisson ? (__syncthreads_and(counts) ? 2 : 1) : 0;
    auto transform = [&](float v) {
        return term == 0 ? v : (term == 1 ? box_transform<1>(v, b.inv_scale) : box_transform<2>(v, b.inv_scale));
    };
    for (int i = tid; i < ZA * W * 32; i += kRowThreads3) A[i] = transform(A[i]);
    // eight rows a warp in flight: with one CTA per SM nothing else covers the
    // loads' latency
    for (int xi = lane; xi < XB; xi += 32) {
        const int x = x0 - b.rad[2] + xi;
        const bool inx = x >= 0 && x < b.n[2];
        for (int row0 = warp * 8; row0 < ZB * YB; row0 += nwarps * 8) {
            float v[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const int zi = (row0 + k) / YB, yi = row0 + k - zi * YB;
                const int z = z0 + dz0 + zi, y = y0 - b.rad[1] + yi;
                const bool in = inx && zi < ZB && z >= 0 && z < b.n[0] && y >= 0 && y < b.n[1];
                v[k] = in ? __ldg(b.src + (static_cast<int64_t>(z) * b.n[1] + y) * b.n[2] + x) : 0.0f;
            }
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const int zi = (row0 + k) / YB, yi = row0 + k - zi * YB;
                if (zi < ZB) B[(zi * XB + xi) * YB + yi] = transform(v[k]);
            }
        }
    }
    if (blockIdx.z == 0)
        for (int i = tid; i < tz * 32; i += kRowThreads3)
            if (map_s[i] >= 0) b.mode[map_s[i]] = term;
    __syncthreads();
    const int ng = b.px / kG;
    for (int u = warp; u < per * b.ny * ng; u += nwarps) {
        const int g = u % ng, r = u / ng, dyi = r % b.ny, dzi = r / b.ny;
        const float* Bu = B + (dzi * XB + g * kG) * YB + dyi + lane;
        const int dz = dz0 + dzi, dy = dyi - b.rad[1];
        if (term == 0) march3<W, 0>(b, A + lane, Bu, map_s, XB, YB, ZA, z0, y0, x0, dz, dy, g);
        else if (term == 1) march3<W, 1>(b, A + lane, Bu, map_s, XB, YB, ZA, z0, y0, x0, dz, dy, g);
        else march3<W, 2>(b, A + lane, Bu, map_s, XB, YB, ZA, z0, y0, x0, dz, dy, g);
    }
}

// ---------------------------------------------------------------------------
// 2-D: a warp's lanes are 32 of the columns (last-axis positions) that hold
// references; a unit is one row offset and 8 column offsets.  It marches down
// the rows; the 8-row sum is built from pair, quad and octet sums whose delays
// stay in registers.  Columns 3 apart (the default step) load without bank
// conflicts.
// ---------------------------------------------------------------------------
template <int TERM>
__device__ __forceinline__ void march2(const BoxArgs& b, const float* A, const float* B, const int32_t* map_s, int XA,
                                       int XB, int ZA, int z0, int x, int dz, int g) {
    float d1[kG], d2[2][kG], d4[4][kG];  // previous row, pair and quad sums
#pragma unroll
    for (int j = 0; j < kG; ++j) {
        d1[j] = 0.0f;
        d2[0][j] = d2[1][j] = 0.0f;
        d4[0][j] = d4[1][j] = d4[2][j] = d4[3][j] = 0.0f;
    }
    for (int t0 = 0; t0 < ZA; t0 += 4) {
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            const int t = t0 + s;
            if (t < ZA) {
                const float* at = A + t * XA;
                const float* bt = B + t * XB;
                float h[kG], v[kG];
                row_terms<8, TERM>([&](int i) { return at[i]; }, [&](int k) { return bt[k]; }, h);
#pragma unroll
                for (int j = 0; j < kG; ++j) {
                    const float s2 = h[j] + d1[j];
                    const float s4 = s2 + d2[s & 1][j];
                    v[j] = s4 + d4[s][j];
                    d1[j] = h[j];
                    d2[s & 1][j] = s2;
                    d4[s][j] = s4;
                }
                if (t >= 7) {
                    const int slot = map_s[(t - 7) * kTileX];
                    if (slot >= 0) store_unit<TERM>(b, slot, z0 + t - 7, 0, x, dz, 0, g, v);
                }
            }
        }
    }
}

__global__ void __launch_bounds__(kRowThreads2, 2) box_rows_2d_kernel(BoxArgs b) {
    extern __shared__ __align__(16) float smf[];
    __shared__ int cols[kTileX];
    __shared__ int ncol_s;
    constexpr int W = 8;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = kRowThreads2 / 32;
    const int x0 = static_cast<int>(blockIdx.x) * kTileX;
    const int z0 = static_cast<int>(blockIdx.y) * b.tz;
    const int dz0 = static_cast<int>(blockIdx.z) * b.per - b.rad[0];
    const int per = min(b.per, b.rad[0] + 1 - dz0);
    const int ZA = b.tz + W - 1, ZB = ZA + b.per - 1, XA = kTileX + W - 1, XB = kTileX + W - 2 + b.px;
    float* A = smf;               // [ZA][XA]
    float* B = A + ZA * XA;       // [ZB][XB]
    int32_t* map_s = reinterpret_cast<int32_t*>(B + ZB * XB);  // [tz][kTileX]
    bool any = false;
#pragma unroll 4
    for (int i = tid; i < b.tz * kTileX; i += kRowThreads2) {
        const int z = z0 + i / kTileX, x = x0 + i % kTileX;
        int m = -1;
        if (z < b.cnt[0] && x < b.cnt[2]) m = b.map[grid_lin(b, z, 0, x)];
        const bool in = m >= b.lo && m < b.hi;
        map_s[i] = in ? static_cast<int32_t>(m - b.lo) : -1;
        any |= in;
    }
    if (!__syncthreads_or(any)) return;
    if (warp == 0) {
        int n = 0;
        for (int i0 = 0; i0 < kTileX; i0 += 32) {
            const int x = x0 + i0 + lane;
            const bool has = x < b.cnt[2] && b.colflag[x] >= 0;
            const unsigned m = __ballot_sync(0xffffffffu, has);
            if (has) cols[n + __popc(m & ((1u << lane) - 1u))] = i0 + lane;
            n += __popc(m);
        }
        if (lane == 0) ncol_s = n;
    }
    bool counts = b.fvox != nullptr;
#pragma unroll 4
    for (int i = tid; i < ZA * XA; i += kRowThreads2) {
        const int z = z0 + i / XA, x = x0 + i % XA;
        float v = 0.0f;
        if (z < b.n[0] && x < b.n[2]) v = __ldg(b.src + static_cast<int64_t>(z) * b.n[2] + x);
        if (counts) {
            const float c = count_of(v, b.inv_scale);
            counts = c < 4096.0f && rintf(c) == c;
        }
        A[i] = v;
    }
    const int term = b.poisson ? (__syncthreads_and(counts) ? 2 : 1) : 0;
    auto transform = [&](float v) {
        return term == 0 ? v : (term == 1 ? box_transform<1>(v, b.inv_scale) : box_transform<2>(v, b.inv_scale));
    };
    for (int i = tid; i < ZA * XA; i += kRowThreads2) A[i] = transform(A[i]);
    for (int zi = warp; zi < ZB; zi += nwarps) {
        const int z = z0 + dz0 + zi;
        const bool in = z >= 0 && z < b.n[0];
        const float* src = b.src + static_cast<int64_t>(in ? z : 0) * b.n[2];
        for (int xi0 = lane; xi0 < XB; xi0 += 160) {
            float v[5];
#pragma unroll
            for (int k = 0; k < 5; ++k) {
                const int x = x0 - b.rad[2] + xi0 + k * 32;
                v[k] = in && xi0 + k * 32 < XB && x >= 0 && x < b.n[2] ? __ldg(src + x) : 0.0f;
            }
#pragma unroll
            for (int k = 0; k < 5; ++k)
                if (xi0 + k * 32 < XB) B[zi * XB + xi0 + k * 32] = transform(v[k]);
        }
    }
    if (blockIdx.z == 0)
        for (int i = tid; i < b.tz * kTileX; i += kRowThreads2)
            if (map_s[i] >= 0) b.mode[map_s[i]] = term;
    __syncthreads();
    const int ncol = ncol_s;
    const int ng = b.px / kG, passes = (ncol + 31) / 32;
    for (int u = warp; u < passes * per * ng; u += nwarps) {
        const int g = u % ng, r = u / ng, dzi = r % per, pass = r / per;
        const int ci = pass * 32 + lane;
        const int cx = cols[min(ci, ncol - 1)];
        // idle lanes follow the last column and store nothing new: the same values to the same place
        const float* Au = A + cx;
        const float* Bu = B + dzi * XB + cx + g * kG;
        const int dz = dz0 + dzi;
        if (term == 0) march2<0>(b, Au, Bu, map_s + cx, XA, XB, ZA, z0, x0 + cx, dz, g);
        else if (term == 1) march2<1>(b, Au, Bu, map_s + cx, XA, XB, ZA, z0, x0 + cx, dz, g);
        else march2<2>(b, Au, Bu, map_s + cx, XA, XB, ZA, z0, x0 + cx, dz, g);
    }
}

// ---------------------------------------------------------------------------
// Bounds of the exact float32 distance from the screening value Q (a sum over
// the patch), both monotone in Q.  With u = 2^-24, S = sum (r + c), and
// sum c <= (sqrt(sum r) + sqrt(Q/2))^2 (Minkowski on the square roots; the log
// form first turns its deviance into a bound on Q):
//   * the exact kernel's own rounding: per term the sum, two divisions and two
//     logarithms, at most u (4 s + 8 sqrt(s t)); summed by Cauchy and raised to
//     u (6 S + 12 sqrt(S Q) + (P + 8) Q);
//   * square-root form: rounded square roots and differences, at most
//     u (4 sqrt(Q S) + 4 u S + 20 Q), raised to u (6, 8, 32);
//   * log form: M = S (L + 1) + P bounds the summed magnitudes, L = log2 of the
//     largest pooled count; SFU logarithms (2^-22 each), the chains of at most
//     16 additions and the box sums stay below 1.39 x 42 u M = 3.5e-6 M, raised
//     to 5e-6 M.  A reference of zeros has the deviance 2 ln 2 sum c, and no summed
//     magnitude exceeds 101 c (|log2 c| <= 100 where c is not clamped): 5.1e-4 Q,
//     and 1e-20 for the clamped values.  Zero candidates then have equal bounds and
//     the race by position settles them (an empty background: with P in M every
//     candidate of such a reference was evaluated exactly: 72 x 76 x 70, 63 % empty,
//     5x5x5, 5.4 ms, so 2.0);
//   * series form (refined candidates): truncation, SFU functions, rounding and
//     the sum's order stay below 1.6e-5 of the sum;
//   * SSD: (P + 20) u Q from both summation orders, raised to 1.05 (P + 32) u.
// The Poisson bounds carry the rounding of the canonical keys (2^-18 of the
// value's power of two, at least 2^-18), so comparing bounds compares keys.
// ---------------------------------------------------------------------------
// approximate square root; the bounds carry 1e-3 of slack on what it enters
__device__ __forceinline__ float fast_sqrt(float x) {
    float y;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

struct Bound {
    int mode;
    float P, invP, Sr, rtS, rmax, rtmax, irmin, bias;

    // with the rounding of the canonical keys
    __device__ __forceinline__ void eval(float Q, float& lo, float& hi) const {
        raw(Q, lo, hi);
        if (mode != 0) {
            const float mg = 4.1e-6f * fmaxf(1.0f, fabsf(hi));
            hi += mg;
            lo -= mg;
        }
    }

    // square-root form: every term's w = ((r - c) / s)^2 is at most 1/16, since
    // 2 (sqrt r - sqrt c)^2 >= (r - c)^2 / s gives w <= Q / s <= Q / min r
    __device__ __forceinline__ bool close(float Q) const {
        if (mode != 1) return false;
        const float U = 5.96046448e-8f, q = fmaxf(Q, 0.0f);
        const float m = rtS + fast_sqrt(0.5f * q);
        const float S = 1.001f * (Sr + m * m);
        return (q + U * (6.0f * fast_sqrt(S * q) + 8.0f * U * S + 32.0f * q)) * irmin <= 0.0624f;
    }

    __device__ __forceinline__ void raw(float Q, float& lo, float& hi) const {
        const float U = 5.96046448e-8f;
        const float q = fmaxf(Q, 0.0f);
        if (mode == 0) {
            // a zero sum of squares is exact
            const float e = bias == 0.0f && Q == 0.0f ? 0.0f : 1.05f * U * (P + 32.0f) * (q + 2.0f * bias) + 1e-37f;
            lo = Q - e;
            hi = Q + e;
            return;
        }
        float l, h;
        if (mode == 1) {
            const float m = rtS + fast_sqrt(0.5f * q);
            const float S = 1.001f * (Sr + m * m);
            const float rs = fast_sqrt(S * q);
            const float eq = U * (6.0f * rs + 8.0f * U * S + 32.0f * q);
            const float ex = U * (6.0f * S + 12.0f * rs + (P + 8.0f) * q);
            const float w = fminf((q + eq) * irmin, 1.0f);
            const float rho = fminf(1.0f + w * fmaf(0.36f, w, 0.0834f), 1.4427f);
            h = Q + eq + ex;
            l = __fdividef(q - eq, rho) - ex;
        } else if (mode == 3) {
            const float m = rtS + fast_sqrt(0.74f * q);
            const float S = 1.001f * (Sr + m * m);
            const float e = 1.6e-5f * q + U * (6.0f * S + 12.0f * fast_sqrt(S * q) + (P + 8.0f) * q) + 1e-30f;
            h = Q + e;
            l = Q - e;
        } else {
            const float x = fast_sqrt(0.74f * q + 0.02f * (Sr + P));
            const float m = rtS + x, cm = rtmax + x;
            float S = 1.001f * (Sr + m * m);
            const float L = fmaxf(1.0f, __log2f(rmax + cm * cm) + 0.01f);
            float e2 = 5e-6f * (S * (L + 1.0f) + P);
            if (Sr == 0.0f) {
                e2 = fminf(e2, 5.1e-4f * q + 1e-20f);
                S = fminf(S, 0.7221f * (q + e2));
            }
            const float d = q + e2;
            const float ex = U * (6.0f * S + 12.0f * fast_sqrt(S * d) + (P + 8.0f) * d);
            h = Q + e2 + ex;
            l = Q - e2 - ex;
        }
        const float ip = invP;
        hi = h * ip;
        lo = l * ip;
    }
};

// The largest probed Q below q1 whose upper bound lies below `target`
// (-infinity: none), and the smallest probed Q above q0 whose lower bound lies
// above it (+infinity: none): 32 distances delta 2^lane, then 32 linear steps
// in the bracket, which is within 3 % of the bound's own width.
__device__ float below(const Bound& b, float target, float q1, float delta, int lane) {
    float lo, hi;
    const float off = delta * __int_as_float((127 + lane) << 23);
    b.eval(q1 - off, lo, hi);
    const unsigned m = __ballot_sync(0xffffffffu, hi < target);
    if (!m) return -INFINITY;
    const int f = __ffs(m) - 1;
    const float far = __shfl_sync(0xffffffffu, off, f);
    const float near = f > 0 ? __shfl_sync(0xffffffffu, off, max(f - 1, 0)) : 0.0f;
    const float q = q1 - (near + (far - near) * (1.0f / 32.0f) * static_cast<float>(lane + 1));
    b.eval(q, lo, hi);
    const unsigned m2 = __ballot_sync(0xffffffffu, hi < target);
    return m2 ? __shfl_sync(0xffffffffu, q, __ffs(m2) - 1) : q1 - far;
}

__device__ float above(const Bound& b, float target, float q0, float delta, int lane) {
    float lo, hi;
    const float off = delta * __int_as_float((127 + lane) << 23);
    b.eval(q0 + off, lo, hi);
    const unsigned m = __ballot_sync(0xffffffffu, lo > target);
    if (!m) return INFINITY;
    const int f = __ffs(m) - 1;
    const float far = __shfl_sync(0xffffffffu, off, f);
    const float near = f > 0 ? __shfl_sync(0xffffffffu, off, max(f - 1, 0)) : 0.0f;
    const float q = q0 + (near + (far - near) * (1.0f / 32.0f) * static_cast<float>(lane + 1));
    b.eval(q, lo, hi);
    const unsigned m2 = __ballot_sync(0xffffffffu, lo > target);
    return m2 ? __shfl_sync(0xffffffffu, q, __ffs(m2) - 1) : q0 + far;
}

// an upper estimate of the k-th smallest of the warp's 4 x 32 values (exact up
// to the low bits); +infinity when fewer are finite
__device__ float kth_of_kept(const float (&t)[4], int k) {
    uint32_t o[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) o[i] = order_bits(t[i]);
    uint32_t lo = __reduce_min_sync(0xffffffffu, o[0]);  // o[0] is the lane's smallest
    uint32_t hi = order_bits(INFINITY);
    while (hi - lo > 255u) {
        const uint32_t mid = lo + ((hi - lo) >> 1);
        int n = 0;
#pragma unroll
        for (int i = 0; i < 4; ++i) n += o[i] <= mid ? 1 : 0;
        n = __reduce_add_sync(0xffffffffu, n);
        if (n >= k) hi = mid;
        else lo = mid + 1;
    }
    return ordered_float(hi);
}

// the warp's list of smallest values, sorted across the lanes (lane l the l-th),
// takes in the lanes' values k that lie below the K-th
__device__ __forceinline__ void keep_smallest(uint64_t& list, uint64_t k, int K, int lane) {
    unsigned m = __ballot_sync(0xffffffffu, k < __shfl_sync(0xffffffffu, list, K - 1));
    while (m) {
        const uint64_t x = __shfl_sync(0xffffffffu, k, __ffs(m) - 1);
        m &= m - 1;
        const uint64_t up = __shfl_up_sync(0xffffffffu, list, 1);
        if (list > x) list = lane > 0 && up > x ? up : x;
    }
}

constexpr int32_t kOpenBit = static_cast<int32_t>(0x80000000u);  // its acceptance is open
constexpr int32_t kIndexMask = 0x7fffffff;

struct SelectSmem {
    float ref[kSelWarps][128];
    float term[kSelWarps][128];       // one candidate's exact terms
    int32_t poff[128];
    uint64_t key[kSelWarps][kQueue];  // key bounds (low << 32 | high), then the composite key
    uint64_t top[kSelWarps][32];
    int32_t idx[kSelWarps][kQueue];   // row index, kOpenBit
    int32_t amb[kSelWarps][kAmb];
    int nq[kSelWarps], na[kSelWarps], acc[kSelWarps];
    int mode[kSelWarps], pos[kSelWarps][3];
    float tkey[kSelWarps];
    float red[kSelWarps];
    Bound bound[kSelWarps];
    int want[kSelWarps];  // exact keys wanted
    int gone[kSelWarps];
};

// one term of the exact kernel's float32 distance
template <bool SSD>
__device__ __forceinline__ float exact_term(float r, float v, float inv, bool counts) {
    if (SSD) {
        const float d = sub_rn(v, r);
        return mul_rn(d, d);
    }
    const float c = count_of(v, inv);
    const int ci = __float2int_rz(c), ri = __float2int_rz(r);
    if (counts && ci < kTable && ri < kTable && __int2float_rn(ci) == c && __int2float_rn(ri) == r)
        return g_box_count_table[ri * kTable + ci];
    return deviance_term(r, c);
}

// exact float32 distance in the exact kernel's order of operations
template <bool SSD>
__device__ __forceinline__ float exact_of(const MatchArgs& a, const float* ref, const float* cand,
                                          const int32_t* poff, bool counts) {
    float d = 0.0f;
    for (int p = 0; p < a.P; ++p)
        d = add_rn(d, exact_term<SSD>(ref[p], __ldg(cand + poff[p]), a.inv_scale, counts));  // zero where r + c = 0
    if (SSD) return d;
    if (d < 0.0f) d = 0.0f;
    return div_rn(d, static_cast<float>(a.P));
}

// the deviance term s w f(w), w = ((r - c) / s)^2, by its power series (terms
// w^(k-1) / (k (2k - 1)), k <= 12: truncated below 1.5e-6 for w <= 1/2), which
// has no cancellation; farther apart the ratio form (its error, 1.4e-6 s, is
// below 2.6e-6 of such a term).  CLOSE: every w is at most 1/16, where five
// coefficients truncate below 2e-8.
template <bool CLOSE>
__device__ __forceinline__ float series_terms(const MatchArgs& a, const float* ref, const float* cand,
                                              const int32_t* poff) {
    float sum = 0.0f, unused = 0.0f;
#pragma unroll 4
    for (int p = 0; p < a.P; ++p) {
        const float r = ref[p];
        const float c = count_of(__ldg(cand + poff[p]), a.inv_scale);
        const float d = r - c, u = d * sfu_rcp(fmaxf(r + c, 1.17549435e-38f)), w = u * u;
        float f = 1.0f / 45.0f;
        if (!CLOSE) {
            f = 1.0f / 276.0f;
            f = fmaf(f, w, 1.0f / 231.0f);
            f = fmaf(f, w, 1.0f / 190.0f);
            f = fmaf(f, w, 1.0f / 153.0f);
            f = fmaf(f, w, 1.0f / 120.0f);
            f = fmaf(f, w, 1.0f / 91.0f);
            f = fmaf(f, w, 1.0f / 66.0f);
            f = fmaf(f, w, 1.0f / 45.0f);
        }
        f = fmaf(f, w, 1.0f / 28.0f);
        f = fmaf(f, w, 1.0f / 15.0f);
        f = fmaf(f, w, 1.0f / 6.0f);
        f = fmaf(f, w, 1.0f);
        float t = d * u * f;
        if (!CLOSE && w > 0.5f) t = kLn2x2 * ratio_term(r, r + r, c, unused);
        sum += t;
    }
    return sum;
}

// the key a distance bound compares as (SSD: the distance itself)
template <bool SSD>
__device__ __forceinline__ float key_of(float d) {
    return SSD ? d : canonical_key(fmaxf(d, 0.0f));
}

// f(i, row[i]) for every entry of the row, 32 at a time over the lanes, with
// eight loads in flight; entries past the end read as infinity
template <typename F>
__device__ __forceinline__ void scan_row(const float* row, int n, int lane, F f) {
    for (int i0 = 0; i0 < n; i0 += 256) {
        float q[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int i = i0 + k * 32 + lane;
            q[k] = i < n ? row[i] : INFINITY;
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) f(i0 + k * 32 + lane, q[k]);
    }
}

// HEAVY = false: one warp per reference, up to kSelWarps per CTA, over the chunk;
// a reference with more open candidates than the queue holds goes to the heavy
// list, with the cuts it found.
// HEAVY = true: one CTA per reference of that list.  Its warps share the
// refinement of the row: every open candidate's value becomes its series-form
// deviance (SSD: exact distance) and the passes run again on the tighter bounds;
// if that is not enough (keys that tie), the values become the exact keys.
// 7.4 K references of a smooth 40 x 49 x 66 estimate, 6.1 K of them heavy: 2.7 ms
// with every first pass made again and the queue tried up to 96 entries only,
// 1.5 ms so.
template <bool SSD, bool HEAVY>
__global__ void __launch_bounds__(kSelWarps * 32, 8) box_select_kernel(MatchArgs a, BoxArgs b) {
    extern __shared__ __align__(16) unsigned char raw[];
    SelectSmem& s = *reinterpret_cast<SelectSmem*>(raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int P = a.P, K = a.max_m, R = a.required;
    const unsigned before = (1u << lane) - 1u;
    for (int i = tid; i < P; i += kSelWarps * 32) {
        int rem = i;
        int64_t off = 0;
        for (int d = a.ndim - 1; d >= 0; --d) {
            off += static_cast<int64_t>(rem % a.block[d]) * a.vstride[d];
            rem /= a.block[d];
        }
        s.poff[i] = static_cast<int32_t>(off);
    }
    float bias = 0.0f;
    if (SSD && b.noise) {
        const int nb = b.nz * b.ny * b.nx;
        for (int i = tid; i < nb; i += kSelWarps * 32) bias = fmaxf(bias, fabsf(mul_rn(b.gamma, __ldg(b.noise + i))));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) bias = fmaxf(bias, __shfl_xor_sync(0xffffffffu, bias, o));
        if (lane == 0) s.red[warp] = bias;
        __syncthreads();
        bias = fmaxf(fmaxf(s.red[0], s.red[1]), fmaxf(s.red[2], s.red[3]));
    }
    const int64_t items = HEAVY ? *b.heavy_n : b.hi - b.lo;
    const int per_cta = HEAVY ? 1 : b.per_cta;
    for (int64_t base = blockIdx.x * per_cta; base < items; base += gridDim.x * per_cta) {
        __syncthreads();  // the previous references' shared data is no longer read
        const bool mine = HEAVY || (warp < per_cta && base + warp < items);
        const int64_t r = HEAVY ? b.heavy[base] : b.lo + base + (mine ? warp : 0);
        int c[3] = {0, 0, 0};
        bool ok = mine && ref_position(a, b, r, c);
        int64_t center_lin = 0;
        if (ok) {
            center_lin = grid_lin(b, c[0], c[1], c[2]);
            ok = b.map[center_lin] == r;  // of duplicates one has a row, the others are redone
        }
        int n_cert = 0, nq = 0, na = 0, mode = 0, defer = 0;
        bool direct = false;  // the top list is already there
        const float thr = mine ? (a.thresholds ? a.thresholds[r] : (a.thr_dev ? *a.thr_dev : a.scalar_threshold)) : 0.0f;
        const float tkey = SSD ? thr : canonical_key(thr);
        if (ok) {
            mode = b.mode[r - b.lo];
            const float* ref0 = a.src + (static_cast<int64_t>(c[0]) * b.n[1] + c[1]) * b.n[2] + c[2];
            float Sr = 0.0f, rmin = INFINITY, rmax = 0.0f;
            for (int p = lane; p < P; p += 32) {
                float v = __ldg(ref0 + s.poff[p]);
                if (!SSD) {
                    v = count_of(v, a.inv_scale);
                    Sr += v;
                    rmin = fminf(rmin, v);
                    rmax = fmaxf(rmax, v);
                }
                s.ref[warp][p] = v;
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                Sr += __shfl_xor_sync(0xffffffffu, Sr, o);
                rmin = fminf(rmin, __shfl_xor_sync(0xffffffffu, rmin, o));
                rmax = fmaxf(rmax, __shfl_xor_sync(0xffffffffu, rmax, o));
            }
            Bound bd;
            bd.mode = SSD ? 0 : mode;
            bd.P = static_cast<float>(P);
            bd.invP = 1.0f / bd.P;
            bd.Sr = 1.001f * Sr;
            bd.rtS = sqrtf(bd.Sr);
            bd.rmax = rmax;
            bd.rtmax = sqrtf(rmax);
            bd.irmin = rmin > 1e-30f ? 1.0f / rmin : 1e30f;
            bd.bias = bias;
            const float q_thr = SSD ? thr : thr * static_cast<float>(P);
            // smallest step of the cut searches: far below any bound's width
            const float tiny = SSD ? 1e-7f * bias + 1e-32f : 1e-8f * (bd.Sr + bd.P);
            float* row = b.rows + (r - b.lo) * b.rowlen;
            const int n = static_cast<int>(b.rowlen);
            int window = 1;
#pragma unroll
            for (int d = 0; d < 3; ++d)
                window *= min(c[d] + b.rad[d], b.cnt[d] - 1) - max(c[d] - b.rad[d], 0) + 1;
            int settled = 0;  // HEAVY: accepted, and no longer in the row
            float cuts[3] = {0.0f, 0.0f, 0.0f};
#pragma unroll 1
            for (int level = 0; level < (HEAVY ? 2 : 1); ++level) {
                // the cuts of the first level come with the list: its refinement takes
                // every candidate below them (of 4.4 M such candidates of a smooth
                // estimate the race below left 4.1 M, at half of this kernel's work)
                const bool handed = HEAVY && !SSD && level == 0;
                float q_cert, q_rej, q_top;
                uint64_t v_top = ~0ull;
                if (handed) {
                    q_cert = b.cuts[3 * base];
                    q_rej = b.cuts[3 * base + 1];
                    q_top = b.cuts[3 * base + 2];
                } else {
                    // certainly accepted: Q <= q_cert; certainly rejected: Q >= q_rej
                    q_cert = below(bd, thr, q_thr, 1e-7f * fabsf(q_thr) + tiny, lane);
                    q_rej = above(bd, thr, q_thr, 1e-7f * fabsf(q_thr) + tiny, lane);
                    // pass 1: the certain accepts, and the 4 smallest of every lane
                    int finite = 0;
                    n_cert = 0;
                    float t[4] = {INFINITY, INFINITY, INFINITY, INFINITY};
                    scan_row(row, n, lane, [&](int, float q) {
                        finite += q < INFINITY ? 1 : 0;
                        n_cert += q <= q_cert ? 1 : 0;
                        if (q < t[3]) {
                            t[3] = q;
    #pragma unroll
                            for (int e = 3; e > 0; --e) {
                                const float lo = fminf(t[e - 1], t[e]), hi = fmaxf(t[e - 1], t[e]);
                                t[e - 1] = lo;
                                t[e] = hi;
                            }
                        }
                    });
                    finite = __reduce_add_sync(0xffffffffu, finite);
                    n_cert = __reduce_add_sync(0xffffffffu, n_cert);
                    if (level == 0 && finite != window) {
                        ok = false;  // infinities or NaN among the values: the exact kernel decides
                        break;
                    }
                    // beyond q_top a candidate cannot reach the top K (nor the first R)
                    auto cut = [&](float v) {
                        float lo, hi;
                        bd.eval(v, lo, hi);
                        return v < INFINITY ? above(bd, hi, v, 1e-7f * fabsf(v) + tiny, lane) : INFINITY;
                    };
                    q_top = q_rej;
                    if (n_cert >= K) q_top = cut(kth_of_kept(t, K));
                    if (n_cert < R) q_top = fmaxf(q_top, R <= window ? cut(kth_of_kept(t, R)) : INFINITY);
                    // pass 2: queue what the bounds leave open
                    nq = 0;
                    na = 0;
                    scan_row(row, n, lane, [&](int i, float q) {
                        const bool take = q < INFINITY && q <= q_top;
                        const bool open = q > q_cert && q < q_rej;
                        if (!__any_sync(0xffffffffu, take || open)) return;
                        const unsigned mt = __ballot_sync(0xffffffffu, take);
                        const unsigned ma = __ballot_sync(0xffffffffu, open && !take);
                        if (take) {
                            const int at = nq + __popc(mt & before);
                            if (at < kQueue) s.idx[warp][at] = i;
                        } else if (open) {
                            const int at = na + __popc(ma & before);
                            if (at < kAmb) s.amb[warp][at] = i;
                        }
                        nq += __popc(mt);
                        na += __popc(ma);
                    });
                    // the race by keys: best holds the K smallest (upper key, position),
                    // sorted across the lanes; whoever's (lower key, position) lies above
                    // its last entry is out.  Where keys tie (flat regions) this leaves
                    // the first positions.
                    const bool listed = nq <= kQueue;
                    if (!HEAVY && !SSD && !listed) {
                        // the race pays off where keys tie, not where the bounds are wide
                        float lo, hi;
                        bd.raw(kth_of_kept(t, min(K, window)), lo, hi);
                        if (!(key_of<false>(lo) == key_of<false>(hi))) {
                            defer = 1;
                            cuts[0] = q_cert;
                            cuts[1] = q_rej;
                            cuts[2] = q_top;
                            break;
                        }
                    }
                    const int entries = listed ? nq : n;
                    uint64_t best = ~0ull;
                    __syncwarp();
                    for (int j0 = 0; j0 < entries; j0 += 32) {
                        const int j = j0 + lane;
                        const int i = listed && j < entries ? s.idx[warp][j] : j;
                        const float q = j < entries ? row[i] : INFINITY;
                        uint64_t k = ~0ull;
                        if (q < INFINITY && q <= q_top) {
                            float lo, hi;
                            bd.raw(q, lo, hi);
                            k = composite_key(key_of<SSD>(hi), i);
                        }
                        keep_smallest(best, k, K, lane);
                    }
                    v_top = __shfl_sync(0xffffffffu, best, K - 1);
                    int kept = 0, known_acc = 0;
                    for (int j0 = 0; j0 < entries; j0 += 32) {
                        const int j = j0 + lane;
                        const int i = listed && j < entries ? s.idx[warp][j] : j;
                        const float q = j < entries ? row[i] : INFINITY;
                        bool race = false, amb = false;
                        float klo = 0.0f, khi = 0.0f;
                        const bool open = q > q_cert && q < q_rej;
                        if (q < INFINITY && q <= q_top) {
                            bd.raw(q, klo, khi);
                            klo = key_of<SSD>(klo);
                            khi = key_of<SSD>(khi);
                            race = composite_key(klo, i) <= v_top;
                            if (!race && open) {
                                known_acc += khi < tkey ? 1 : 0;
                                amb = khi >= tkey && klo < tkey;
                            }
                        }
                        const unsigned mr = __ballot_sync(0xffffffffu, race);
                        const unsigned ma = __ballot_sync(0xffffffffu, amb);
                        if (race) {
                            const int at = kept + __popc(mr & before);
                            if (at < kQueue) {
                                s.idx[warp][at] = i | (open ? kOpenBit : 0);
                                s.key[warp][at] = (static_cast<uint64_t>(__float_as_uint(klo)) << 32) | __float_as_uint(khi);
                            }
                        } else if (amb) {
                            const int at = na + __popc(ma & before);
                            if (at < kAmb) s.amb[warp][at] = i;
                        }
                        kept += __popc(mr);
                        na += __popc(ma);
                        __syncwarp();
                    }
                    nq = kept;
                    const bool fits = nq <= kQueue && na <= kAmb;
                    if (fits && (!HEAVY || level == 1)) {
                        n_cert += __reduce_add_sync(0xffffffffu, known_acc);
                        break;
                    }
                    if (!HEAVY) {
                        defer = 1;
                        cuts[0] = q_cert;
                        cuts[1] = q_rej;
                        cuts[2] = q_top;
                        break;
                    }
                }
                // refinement: this warp's quarter of the row
                const bool exact = SSD || level == 1;
                auto needed = [&](int i, float q) {
                    const bool open = q > q_cert && q < q_rej;
                    if (!(q < INFINITY) || open || q > q_top) return open;
                    if (handed) return true;
                    float lo, hi;
                    bd.raw(q, lo, hi);
                    return composite_key(key_of<SSD>(lo), i) <= v_top;
                };
                __syncthreads();  // every warp has read the row
                int gone = 0;  // certain accepts of this quarter that leave the row
                int fill = 0;
                auto refine = [&](int to) {
                    for (int at = lane; at < to; at += 32) {
                        const int i = s.idx[warp][at];
                        const int dx = i % b.px, rem = i / b.px, dy = rem % b.ny, dz = rem / b.ny;
                        const float* cand = ref0 + (static_cast<int64_t>(dz - b.rad[0]) * b.n[1] + (dy - b.rad[1])) * b.n[2] +
                                            (dx - b.rad[2]);
                        float d;
                        if (!exact) {
                            d = bd.close(row[i]) ? series_terms<true>(a, s.ref[warp], cand, s.poff)
                                             : series_terms<false>(a, s.ref[warp], cand, s.poff);
                        } else {
                            d = exact_of<SSD>(a, s.ref[warp], cand, s.poff, mode == 2);
                            if (SSD && b.noise) d = sub_rn(d, mul_rn(b.gamma, __ldg(b.noise + rem * b.nx + dx)));
                            d = SSD ? d : canonical_key(d);
                        }
                        row[i] = d;
                    }
                };
                for (int i0 = warp * 32; i0 < n; i0 += kSelWarps * 32) {
                    const int i = i0 + lane;
                    const float q = i < n ? row[i] : INFINITY;
                    bool open = needed(i, q);
                    gone += q <= q_cert && !open ? 1 : 0;
                    if (!open && i < n) row[i] = INFINITY;
                    if (open && exact && !SSD) {
                        float lo, hi;
                        bd.raw(q, lo, hi);
                        const float klo = key_of<SSD>(lo), khi = key_of<SSD>(hi);
                        if (klo == khi) {
                            row[i] = khi;
                            open = false;
                        }
                    }
                    const unsigned m = __ballot_sync(0xffffffffu, open);
                    if (open) s.idx[warp][fill + __popc(m & before)] = i;
                    fill += __popc(m);
                    __syncwarp();
                    if (fill > kQueue - 32) {  // whole warps' worth at a time
                        const int whole = fill & ~31;
                        refine(whole);
                        __syncwarp();
                        const int keep = lane < fill - whole ? s.idx[warp][whole + lane] : 0;
                        __syncwarp();
                        fill -= whole;
                        if (lane < fill) s.idx[warp][lane] = keep;
                        __syncwarp();
                    }
                }
                refine(fill);
                gone = __reduce_add_sync(0xffffffffu, gone);
                if (lane == 0) s.gone[warp] = gone;
                __syncthreads();  // the row is complete
                settled += s.gone[0] + s.gone[1] + s.gone[2] + s.gone[3];
                bd.mode = 3;
                if (exact) {
                    // the K smallest by (exact key, position); row order is position order
                    uint64_t list = ~0ull;
                    n_cert = 0;
                    scan_row(row, n, lane, [&](int i, float q) {
                        n_cert += q < tkey ? 1 : 0;
                        keep_smallest(list, q < INFINITY ? composite_key(q, i) : ~0ull, K, lane);
                    });
                    n_cert = __reduce_add_sync(0xffffffffu, n_cert);
                    if (list != ~0ull) {
                        const int i = static_cast<int>(list & 0xffffffffu);
                        const int dx = i % b.px, rem = i / b.px, dy = rem % b.ny, dz = rem / b.ny;
                        list = (list & 0xffffffff00000000ull) |
                               static_cast<uint32_t>(grid_lin(b, c[0] + dz - b.rad[0], c[1] + dy - b.rad[1],
                                                              c[2] + dx - b.rad[2]));
                    }
                    s.top[warp][lane] = lane < K ? list : ~0ull;
                    direct = true;
                    nq = 0;
                    na = 0;
                    break;
                }
            }
            n_cert += settled;
            if (defer && lane == 0) {
                const int at = atomicAdd(b.heavy_n, 1);
                b.heavy[at] = static_cast<int32_t>(r);
#pragma unroll
                for (int e = 0; e < 3; ++e) b.cuts[3 * static_cast<int64_t>(at) + e] = cuts[e];
            }
            if (lane == 0) {
                bd.mode = SSD ? 0 : 3;
                s.bound[warp] = bd;
            }
        }
        const bool live = ok && !defer && (!HEAVY || warp == 0);
        if (lane == 0) {
            s.nq[warp] = live ? nq : 0;
            s.na[warp] = live ? na : 0;
            s.acc[warp] = n_cert;
            s.mode[warp] = mode;
            s.tkey[warp] = tkey;
#pragma unroll
            for (int d = 0; d < 3; ++d) s.pos[warp][d] = c[d];
        }
        __syncthreads();
        auto locate = [&](int w, int i, int64_t& lin, int& widx) -> const float* {
            const int dx = i % b.px, rem = i / b.px;
            const int dy = rem % b.ny, dz = rem / b.ny;
            const int z = s.pos[w][0] + dz - b.rad[0], y = s.pos[w][1] + dy - b.rad[1], x = s.pos[w][2] + dx - b.rad[2];
            lin = grid_lin(b, z, y, x);
            widx = rem * b.nx + dx;
            return a.src + (static_cast<int64_t>(z) * b.n[1] + y) * b.n[2] + x;
        };
        // the queue's key bounds, and the open acceptances, tightened by the series
        // form (not for counts, whose bounds are tight and whose exact terms are
        // tabulated; a refined row has it already); an acceptance it leaves open
        // joins the queue
        if (!SSD) {
            const int e0 = s.na[0], e1 = e0 + s.na[1], e2 = e1 + s.na[2], e3 = e2 + s.na[3];
            const int f0 = e3 + s.nq[0], f1 = f0 + s.nq[1], f2 = f1 + s.nq[2], f3 = f2 + s.nq[3];
            __syncthreads();  // the counts are read before the queue grows
            for (int i = tid; i < f3; i += kSelWarps * 32) {
                const bool amb = i < e3;
                const int w = amb ? (i >= e0) + (i >= e1) + (i >= e2) : (i >= f0) + (i >= f1) + (i >= f2);
                const int j = amb ? i - (w == 0 ? 0 : (w == 1 ? e0 : (w == 2 ? e1 : e2)))
                                  : i - (w == 0 ? e3 : (w == 1 ? f0 : (w == 2 ? f1 : f2)));
                if (!amb && (HEAVY || s.mode[w] == 2)) continue;
                if (!amb && static_cast<uint32_t>(s.key[w][j] >> 32) == static_cast<uint32_t>(s.key[w][j])) continue;
                const int ri = amb ? s.amb[w][j] : s.idx[w][j] & kIndexMask;
                int64_t lin;
                int widx;
                const float* cand = locate(w, ri, lin, widx);
                float lo, hi;
                s.bound[w].raw(series_terms<false>(a, s.ref[w], cand, s.poff), lo, hi);
                const float klo = key_of<false>(lo), khi = key_of<false>(hi);
                const uint64_t kb = (static_cast<uint64_t>(__float_as_uint(klo)) << 32) | __float_as_uint(khi);
                if (!amb) {
                    s.key[w][j] = kb;
                } else if (khi < s.tkey[w]) {
                    atomicAdd(&s.acc[w], 1);
                } else if (klo < s.tkey[w]) {
                    const int at = atomicAdd(&s.nq[w], 1);
                    if (at < kQueue) {
                        s.idx[w][at] = ri | kOpenBit;
                        s.key[w][at] = kb;
                    }
                }
            }
            __syncthreads();
        } else {
            if (lane == 0 && s.na[warp] > 0) {  // (few: the bounds of SSD are tight)
                for (int j = 0; j < s.na[warp]; ++j) {
                    const int at = s.nq[warp]++;
                    if (at < kQueue) {
                        s.idx[warp][at] = s.amb[warp][j] | kOpenBit;
                        s.key[warp][at] = (static_cast<uint64_t>(__float_as_uint(-INFINITY)) << 32) |
                                          __float_as_uint(INFINITY);
                    }
                }
            }
            __syncwarp();
        }
        // An exact key is needed only where the order or the acceptance is open: the
        // key bounds overlap another candidate's, or straddle the threshold.  Those
        // go to the amb list.
        {
            const int q = min(s.nq[warp], kQueue);
            int want = 0;
            for (int i0 = 0; i0 < q; i0 += 32) {
                const int i = i0 + lane;
                bool known = true;
                if (i < q) {
                    const uint64_t kb = s.key[warp][i];
                    const float klo = __uint_as_float(static_cast<uint32_t>(kb >> 32));
                    const float khi = __uint_as_float(static_cast<uint32_t>(kb));
                    known = klo == khi;
                    if (!known && (khi < tkey || klo >= tkey)) {
                        int meets = 0;
                        for (int j = 0; j < q; ++j) {
                            const uint64_t ob = s.key[warp][j];
                            const float olo = __uint_as_float(static_cast<uint32_t>(ob >> 32));
                            const float ohi = __uint_as_float(static_cast<uint32_t>(ob));
                            meets += olo <= khi && klo <= ohi ? 1 : 0;
                        }
                        known = meets == 1;  // itself
                    }
                }
                const unsigned m = __ballot_sync(0xffffffffu, !known);
                if (!known) s.amb[warp][want + __popc(m & before)] = i;
                want += __popc(m);
                __syncwarp();
            }
            // the others take their upper key
            for (int i = lane; i < q; i += 32) {
                int64_t lin;
                int widx;
                (void)locate(warp, s.idx[warp][i] & kIndexMask, lin, widx);
                const float khi = __uint_as_float(static_cast<uint32_t>(s.key[warp][i]));
                s.key[warp][i] = composite_key(khi, static_cast<int32_t>(lin));
            }
            if (lane == 0) s.want[warp] = want;
        }
        __syncthreads();
        {
            const int e0 = s.want[0], e1 = e0 + s.want[1], e2 = e1 + s.want[2], e3 = e2 + s.want[3];
            auto finish = [&](int w, int j, float d, int64_t lin, int widx) {
                if (SSD && b.noise) d = sub_rn(d, mul_rn(b.gamma, __ldg(b.noise + widx)));
                const float key = SSD ? d : canonical_key(d);
                s.key[w][j] = composite_key(key, static_cast<int32_t>(lin));
            };
            // few: a warp per candidate, lanes over the terms, the sum in patch order;
            // many: a thread per candidate
            const bool by_warp = e3 <= 24 * kSelWarps;
            for (int i = by_warp ? warp : tid; i < e3; i += by_warp ? kSelWarps : kSelWarps * 32) {
                const int w = (i >= e0) + (i >= e1) + (i >= e2);
                const int j = s.amb[w][i - (w == 0 ? 0 : (w == 1 ? e0 : (w == 2 ? e1 : e2)))];
                int64_t lin;
                int widx;
                const float* cand = locate(w, s.idx[w][j] & kIndexMask, lin, widx);
                const bool counts = s.mode[w] == 2;
                if (!by_warp) {
                    finish(w, j, exact_of<SSD>(a, s.ref[w], cand, s.poff, counts), lin, widx);
                    continue;
                }
                for (int p = lane; p < P; p += 32)
                    s.term[warp][p] = exact_term<SSD>(s.ref[w][p], __ldg(cand + s.poff[p]), a.inv_scale, counts);
                __syncwarp();
                if (lane == 0) {
                    float d = 0.0f;
#pragma unroll 8
                    for (int p = 0; p < P; ++p) d = add_rn(d, s.term[warp][p]);
                    if (!SSD) {
                        if (d < 0.0f) d = 0.0f;
                        d = div_rn(d, static_cast<float>(P));
                    }
                    finish(w, j, d, lin, widx);
                }
                __syncwarp();
            }
        }
        __syncthreads();
        if (mine && !defer && (!HEAVY || warp == 0)) {
            const int q = s.nq[warp];
            if (!ok || q > kQueue) {
                if (lane == 0) a.count[r] = -1;
                continue;
            }
            // rank of every queued key; the accepted ones come first
            const uint64_t tbits = static_cast<uint64_t>(order_bits(tkey)) << 32;
            int open_acc = 0;
            for (int i = lane; i < q; i += 32) open_acc += s.idx[warp][i] < 0 && s.key[warp][i] < tbits ? 1 : 0;
            const int total = s.acc[warp] + __reduce_add_sync(0xffffffffu, open_acc);
            int ntop = 0;
            if (direct) {
                const uint64_t k = s.top[warp][lane];
                const bool in = k != ~0ull && (k < tbits || (total < R && lane < R));
                ntop = __popc(__ballot_sync(0xffffffffu, in));
            }
            for (int i0 = 0; i0 < q; i0 += 32) {
                const int i = i0 + lane;
                const uint64_t k = i < q ? s.key[warp][i] : ~0ull;
                int rank = 0;
                for (int j = 0; j < q; ++j) rank += s.key[warp][j] < k ? 1 : 0;
                const bool in = i < q && rank < K && (k < tbits || (total < R && rank < R));
                if (in) s.top[warp][rank] = k;
                ntop += __popc(__ballot_sync(0xffffffffu, in));
            }
            __syncwarp();
            const int32_t l = lane < ntop ? static_cast<int32_t>(s.top[warp][lane] & 0xffffffffu) : -1;
            const bool other = lane < ntop && l != static_cast<int32_t>(center_lin);
            const unsigned om = __ballot_sync(0xffffffffu, other);
            int cnt = min(K, 1 + __popc(om));
            if (a.pow2) {
                int target = 1;
                while ((target << 1) <= cnt) target <<= 1;
                if (a.min_m > target) target = a.min_m;
                if (target < cnt) cnt = target;
            }
            // entries past the count are -1; the reference comes first
            int32_t* out = a.sel + r * K;
            const int at = 1 + __popc(om & before);
            if (lane < K && lane >= cnt) out[lane] = -1;
            if (lane == 0) out[0] = static_cast<int32_t>(center_lin);
            if (other && at < cnt) out[at] = l;
            if (lane == 0) {
                a.count[r] = cnt;
                a.accepted[r] = total;
            }
        }
    }
}

uint64_t round256(uint64_t v) { return (v + 255) & ~uint64_t(255); }

// Whether a matching takes these kernels, its tiles and its scratch
struct BoxPlan {
    bool applies, want_f;
    BoxArgs b;  // geometry and tiles; no pointers but the source's
    int ztiles, splits;
    int64_t columns;
    size_t smem;
    // scratch: origin map and column flags, the counts' box sums, the rows of a chunk of references
    uint64_t o_flag, o_fvox, o_fbox, o_rows, per_ref;
    uint64_t least, full;  // bytes: for a few references at a time, for chunks of up to kRowScratch
    int64_t chunk(const MatchArgs& a, uint64_t bytes) const {
        return std::min<int64_t>(static_cast<int64_t>((bytes - o_rows - 1024) / per_ref), a.n_refs);
    }
};

// Whether sharing row terms beats the kernel that would run instead.  The row
// kernels work on all origins in the columns that hold references, the others on
// the references alone, so it takes dense references.  Measured on one GB300, the
// other kernel's ms against this file's (matching alone, no scratch allocated):
//   * bounded screening, and exact terms of values that are no counts, lose at
//     every density down to one reference per 64 origins, where the list ends
//     (1024 x 1000, one per 63: 1.70 / 1.11; 128 x 120 x 132, 4x4x4, one per 60:
//     5.78 / 4.06; terms of counts at a scale of 1.5: 2 to 4 times);
//   * tabulated terms of counts: 1024 x 1000 one per 16 2.85 / 2.02, one per 25
//     1.86 / 1.73, one per 36 1.30 / 1.59; 420 x 388 one per 16 0.45 / 0.41, one per
//     24 0.29 / 0.36; 64 x 64 34 / 115 us; 128 x 120 x 132, 4x4x4, one per 33 6.23 /
//     4.14, one per 44 4.69 / 3.96, one per 53 with every other column used 3.84 /
//     5.90; 72 x 76 x 70, one per 31 1.10 / 0.93, one per 41 0.84 / 0.90, 5x5x5
//     1.60 / 1.34.  Windows of 29^3 lose (5x5x5, 85.6 / 94.5; 23^3: 35.0 / 35.6);
//   * exact SSD, a warp per reference: windows below a hundred offsets in 3-D lose
//     (128 x 120 x 132, 3^3: 0.35 / 0.54 ms), small ones of few references (72 x 76
//     x 70, 5x5x5, 5^3: 0.19 / 0.31; 420 x 388, 11^2: 0.147 / 0.149), and sparse ones
//     in 2-D (one per 47 0.23 / 0.21, one per 61 0.16 / 0.21).  In 3-D sparse ones win
//     where the last axis is among the sparse (72 x 76 x 70, 4x4x4, steps 4, 4, 4
//     0.72 / 0.55, steps 6, 5, 2 0.74 / 0.86), which is not known here.  Where the
//     scratch has to be allocated, which takes 0.1 ms and 0.9 ms per GB, 2-D needs
//     more references (6.4 K: 0.34 / 0.37; 9.9 K: 0.51 / 0.39) and wider windows.
// Real-valued stages come here whatever their size: few references gain 0.1 ms at
// best in the screened kernel, and those it cannot settle cost 3.1 ms there
// (24 x 24 x 40, peak 30; here 0.5 in all).
bool pays_off(const MatchArgs& a, const BoxArgs& b, int code, int precision, bool allocates, int64_t n_lins) {
    if (a.n_refs * 64 < n_lins) return false;
    if (precision != BMND_MATCH_EXACT) return true;
    const int64_t window = static_cast<int64_t>(b.nz) * b.ny * b.nx;
    if (code == BMND_DIST_SSD) {
        if (a.ndim == 2 && a.n_refs < std::max<int64_t>(allocates ? 8192 : 0, n_lins / 50)) return false;
        return window >= 343 || ((a.ndim == 2 || window >= 100) && a.n_refs * window >= (allocates ? 10000000 : 2500000));
    }
    if (!counts_kernel_applies(a, code)) return true;
    const int64_t least = a.ndim == 2 ? 4096 + n_lins / (allocates ? 25 : 28)
                                      : std::max<int64_t>(8192, a.P == 64 ? 4096 + n_lins / 52 : n_lins / 48);
    return a.n_refs >= least && b.rowlen <= 20000;
}

// First-axis extent of a chunk of references against the patch edge W: a tile's
// halo of W - 1 origins is computed again for every chunk.  Exact SSD and tabulated
// counts, which lose little to this file's kernels at wide windows, take over from
// short chunks (5x5x5, SSD, 41^3 offsets, 16 origins a chunk: 43.5 ms, here 47.0).
bool chunks_pay_off(const MatchArgs& a, const BoxArgs& b, int W, int code, int precision, int64_t chunk) {
    if (precision != BMND_MATCH_EXACT || (code != BMND_DIST_SSD && !counts_kernel_applies(a, code))) return true;
    return chunk >= a.n_refs || b.cnt[0] * chunk >= 4 * W * a.n_refs;
}

BoxPlan plan_box_match(const MatchArgs& a, int code, int precision, bool allocates) {
    BoxPlan p{};
    BoxArgs& b = p.b;
    const bool ssd = code == BMND_DIST_SSD;
    const int* bl = a.block;
    const bool shape2 = a.ndim == 2 && bl[0] == 8 && bl[1] == 8;
    const bool shape5 = a.ndim == 3 && bl[0] == 5 && bl[1] == 5 && bl[2] == 5;
    const bool shape4 = a.ndim == 3 && bl[0] == 4 && bl[1] == 4 && bl[2] == 4;
    if (a.table || a.fixup || a.null_moments || a.max_m > 32 || !(shape2 || shape4 || shape5)) return p;
    if (ssd ? a.poisson_bias != 0 : (code != BMND_DIST_POISSON_DEVIANCE || !a.stab)) return p;
    if (precision != BMND_MATCH_EXACT && precision != BMND_MATCH_FAST && precision != BMND_MATCH_REAL_VALUED)
        return p;
    const int W = shape2 ? 8 : (shape5 ? 5 : 4);
    const int ax[3] = {0, a.ndim == 3 ? 1 : -1, a.ndim - 1};
    for (int d = 0; d < 3; ++d) {
        b.cnt[d] = ax[d] < 0 ? 1 : a.counts[ax[d]];
        b.rad[d] = ax[d] < 0 ? 0 : a.radius[ax[d]];
        b.n[d] = ax[d] < 0 ? 1 : a.counts[ax[d]] + bl[ax[d]] - 1;
        if (b.rad[d] > 64) return p;
    }
    b.src = a.src;
    b.inv_scale = a.inv_scale;
    b.poisson = ssd ? 0 : 1;
    b.nz = 2 * b.rad[0] + 1;
    b.ny = 2 * b.rad[1] + 1;
    b.nx = 2 * b.rad[2] + 1;
    b.px = (b.nx + kG - 1) / kG * kG;
    b.rowlen = static_cast<int64_t>(b.nz) * b.ny * b.px;
    b.nvox = static_cast<int64_t>(b.n[0]) * b.n[1] * b.n[2];
    b.noise = a.noise_ssd;
    b.gamma = a.gamma;
    const int64_t n_lins = static_cast<int64_t>(b.cnt[0]) * b.cnt[1] * b.cnt[2];
    p.want_f = !ssd && precision != BMND_MATCH_REAL_VALUED && a.inv_scale == 1.0f;
    if (b.rowlen > (1 << 20) || a.n_refs > 0x7fffffffLL || !pays_off(a, b, code, precision, allocates, n_lins))
        return p;

    // tiles: the largest whose shared memory fits; first-axis offsets are split
    // over CTAs until every SM has several
    auto smem_of = [&](int tz, int per) -> size_t {
        const size_t ZA = tz + W - 1, ZB = ZA + per - 1;
        if (shape2)
            return 4 * (ZA * (kTileX + W - 1) + ZB * static_cast<size_t>(kTileX + W - 2 + b.px) +
                        static_cast<size_t>(tz) * kTileX);
        return 4 * (ZA * W * 32 + ZB * static_cast<size_t>(W - 1 + b.px) * (32 + 2 * b.rad[1]) +
                    static_cast<size_t>(tz) * 32);
    };
    const size_t limit = shape2 ? 110 * 1024 : 220 * 1024;
    const int tz_cap = shape2 ? 48 : 29;
    int& ztiles = p.ztiles;
    ztiles = (b.cnt[0] + tz_cap - 1) / tz_cap;
    b.tz = (b.cnt[0] + ztiles - 1) / ztiles;
    b.ytiles = shape2 ? 1 : (b.cnt[1] + 32 - W) / (33 - W);
    p.columns = shape2 ? (b.cnt[2] + kTileX - 1) / kTileX : (b.cnt[2] + 2) / 3;
    auto tiles = [&]() { return p.columns * b.ytiles * ztiles; };
    // (small grids: shorter tiles until there is a CTA or two for every SM)
    while (b.tz > 2 * W && tiles() * b.nz < 152 * 2) {
        b.tz = (b.tz + 1) / 2;
        ztiles = (b.cnt[0] + b.tz - 1) / b.tz;
    }
    int& splits = p.splits;
    splits = static_cast<int>(std::min<int64_t>(b.nz, (152 * 8 + tiles() - 1) / tiles()));
    b.per = (b.nz + splits - 1) / splits;
    while (smem_of(b.tz, b.per) > limit && b.per > 1) --b.per;
    while (smem_of(b.tz, b.per) > limit && b.tz > 4) {
        b.tz = (b.tz + 1) / 2;
        ztiles = (b.cnt[0] + b.tz - 1) / b.tz;
    }
    p.smem = smem_of(b.tz, b.per);
    if (p.smem > limit) return p;
    splits = (b.nz + b.per - 1) / b.per;
    if (static_cast<int64_t>(b.ytiles) * ztiles > 65535 || splits > 65535) return p;

    p.o_flag = round256(4ull * n_lins);
    p.o_fvox = p.o_flag + round256(4ull * b.cnt[2]);
    p.o_fbox = p.o_fvox + (p.want_f ? round256(4ull * b.nvox) : 0);
    p.o_rows = p.o_fbox + (p.want_f ? round256(4ull * n_lins) : 0);
    p.per_ref = 4ull * b.rowlen + 20;
    p.least = p.o_rows + 1024 + p.per_ref * std::min<int64_t>(a.n_refs, 512);
    p.full = std::max(p.least, p.o_rows + 1024 + std::min<uint64_t>(p.per_ref * a.n_refs, kRowScratch));
    p.applies = chunks_pay_off(a, b, W, code, precision, p.chunk(a, p.full));
    return p;
}

}  // namespace

BoxScratch box_match_scratch(const MatchArgs& a, int code, int precision) {
    const BoxPlan p = plan_box_match(a, code, precision, false);
    return p.applies ? BoxScratch{p.least, p.full} : BoxScratch{0, 0};
}

int32_t launch_box_match(MatchArgs& a, int code, int precision, cudaStream_t stream, bool* done) {
    *done = false;
    const BoxPlan p = plan_box_match(a, code, precision, !a.box_ws);
    if (!p.applies) return BMND_OK;
    BoxArgs b = p.b;
    const bool ssd = code == BMND_DIST_SSD, want_f = p.want_f;
    const bool shape2 = a.ndim == 2, shape5 = a.ndim == 3 && a.block[0] == 5;
    const int64_t n_lins = static_cast<int64_t>(b.cnt[0]) * b.cnt[1] * b.cnt[2];
    const bool given = a.box_ws && a.box_ws_bytes >= p.least;
    char* base = given ? a.box_ws : nullptr;
    int64_t chunk = p.chunk(a, given ? a.box_ws_bytes : p.full);
    if (!chunks_pay_off(a, b, shape2 ? 8 : (shape5 ? 5 : 4), code, precision, chunk)) return BMND_OK;
    bool owned = false;
    if (!given && !a.no_alloc) {
        if (cudaMallocAsync(reinterpret_cast<void**>(&base), p.full, stream) == cudaSuccess) {
            owned = true;
            note_device_alloc();
        } else {
            (void)cudaGetLastError();
            base = nullptr;
        }
    }
    if (!base) return BMND_OK;
    const int64_t nchunks = (a.n_refs + chunk - 1) / chunk;
    chunk = (a.n_refs + nchunks - 1) / nchunks;
    b.map = reinterpret_cast<int32_t*>(base);
    b.colflag = reinterpret_cast<int32_t*>(base + p.o_flag);
    b.fvox = want_f ? reinterpret_cast<float*>(base + p.o_fvox) : nullptr;
    b.fbox = want_f ? reinterpret_cast<float*>(base + p.o_fbox) : nullptr;
    b.rows = reinterpret_cast<float*>(base + p.o_rows);
    b.mode = reinterpret_cast<int32_t*>(base + p.o_rows + round256(4ull * b.rowlen * chunk));
    b.heavy_n = b.mode + chunk;
    b.heavy = b.heavy_n + 1;
    b.cuts = reinterpret_cast<float*>(b.heavy + chunk);

    auto run = [&]() -> int32_t {
        BMND_CUDA_TRY(cudaMemsetAsync(base, 0xff, p.o_fvox, stream));
        const int64_t work = std::max<int64_t>(a.n_refs, want_f ? b.nvox : 1);
        const unsigned nb = static_cast<unsigned>(std::min<int64_t>((work + 255) / 256, 152 * 16));
        box_prepare_kernel<<<nb, 256, 0, stream>>>(a, b);
        BMND_LAUNCH_CHECK("box_prepare_kernel");
        if (want_f) {
            const unsigned fb = static_cast<unsigned>(std::min<int64_t>((n_lins + 255) / 256, 152 * 16));
            if (shape2) box_fsum_kernel<8, 1, 8><<<fb, 256, 0, stream>>>(b);
            else if (shape5) box_fsum_kernel<5, 5, 5><<<fb, 256, 0, stream>>>(b);
            else box_fsum_kernel<4, 4, 4><<<fb, 256, 0, stream>>>(b);
            BMND_LAUNCH_CHECK("box_fsum_kernel");
        }
        int per_sm = 0, sms = 0;
        const void* rows_fn = shape2 ? reinterpret_cast<const void*>(box_rows_2d_kernel)
                                     : (shape5 ? reinterpret_cast<const void*>(box_rows_3d_kernel<5>)
                                               : reinterpret_cast<const void*>(box_rows_3d_kernel<4>));
        if (int32_t rc = kernel_residency(rows_fn, shape2 ? kRowThreads2 : kRowThreads3, p.smem, false, &per_sm, &sms))
            return rc;
        const void* sel_fn = ssd ? reinterpret_cast<const void*>(box_select_kernel<true, false>)
                                 : reinterpret_cast<const void*>(box_select_kernel<false, false>);
        const void* heavy_fn = ssd ? reinterpret_cast<const void*>(box_select_kernel<true, true>)
                                   : reinterpret_cast<const void*>(box_select_kernel<false, true>);
        if (int32_t rc = kernel_residency(heavy_fn, kSelWarps * 32, sizeof(SelectSmem), false, &per_sm, &sms)) return rc;
        const int64_t heavy_ctas = static_cast<int64_t>(sms) * std::max(per_sm, 1);
        if (int32_t rc = kernel_residency(sel_fn, kSelWarps * 32, sizeof(SelectSmem), false, &per_sm, &sms)) return rc;
        const int64_t sel_ctas = static_cast<int64_t>(sms) * std::max(per_sm, 1);
        for (b.lo = 0; b.lo < a.n_refs; b.lo += chunk) {
            b.hi = std::min<int64_t>(b.lo + chunk, a.n_refs);
            BMND_CUDA_TRY(cudaMemsetAsync(b.heavy_n, 0, 4, stream));
            if (shape2) {
                const dim3 grid(static_cast<unsigned>(p.columns), static_cast<unsigned>(p.ztiles),
                                static_cast<unsigned>(p.splits));
                box_rows_2d_kernel<<<grid, kRowThreads2, p.smem, stream>>>(b);
            } else {
                const dim3 grid(static_cast<unsigned>(b.cnt[2]), static_cast<unsigned>(b.ytiles * p.ztiles),
                                static_cast<unsigned>(p.splits));
                if (shape5) box_rows_3d_kernel<5><<<grid, kRowThreads3, p.smem, stream>>>(b);
                else box_rows_3d_kernel<4><<<grid, kRowThreads3, p.smem, stream>>>(b);
            }
            BMND_LAUNCH_CHECK("box_rows_kernel");
            // few references: fewer per CTA, whose warps then share their rescoring
            b.per_cta = static_cast<int32_t>(std::clamp<int64_t>((b.hi - b.lo + sel_ctas - 1) / sel_ctas, 1, kSelWarps));
            const int64_t sel_items = (b.hi - b.lo + b.per_cta - 1) / b.per_cta;
            const unsigned ctas = static_cast<unsigned>(std::min(sel_items, sel_ctas));
            const unsigned hctas = static_cast<unsigned>(std::min<int64_t>(b.hi - b.lo, heavy_ctas));
            const size_t ss = sizeof(SelectSmem);
            if (ssd) box_select_kernel<true, false><<<ctas, kSelWarps * 32, ss, stream>>>(a, b);
            else box_select_kernel<false, false><<<ctas, kSelWarps * 32, ss, stream>>>(a, b);
            BMND_LAUNCH_CHECK("box_select_kernel");
            if (ssd) box_select_kernel<true, true><<<hctas, kSelWarps * 32, ss, stream>>>(a, b);
            else box_select_kernel<false, true><<<hctas, kSelWarps * 32, ss, stream>>>(a, b);
            BMND_LAUNCH_CHECK("box_select_kernel (heavy)");
        }
        return BMND_OK;
    };
    const int32_t rc = run();
    if (owned) {
        const cudaError_t e = cudaFreeAsync(base, stream);
        if (!rc && e != cudaSuccess) return cuda_fail(e, "cudaFreeAsync");
    }
    if (rc) return rc;
    *done = true;
    return BMND_OK;
}

}  // namespace bmnd
