// match_common.cuh -- arguments and distance terms shared by the block-matching kernels.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "bmnd_common.cuh"

namespace bmnd {

struct MatchArgs {
    int32_t ndim;
    int32_t counts[BMND_MAX_DIMS];
    int32_t radius[BMND_MAX_DIMS];
    int64_t grid_stride[BMND_MAX_DIMS];  // source offset of one patch-grid step per axis
    int32_t max_m;
    int32_t min_m;
    int32_t required;  // min(min_m, max_m)
    int32_t pow2;
    int32_t stab;
    int32_t P;
    float inv_scale;
    float scalar_threshold;
    const float* src;       // volume or patch table
    int32_t table;          // 1: src is a patch table (element p at offset p)
    int32_t block[BMND_MAX_DIMS];   // patch extents (volume source)
    int64_t vstride[BMND_MAX_DIMS]; // voxel strides (volume source)
    const int32_t* refs;
    const float* thresholds;  // per reference, or null -> scalar_threshold
    int64_t n_refs;
    int32_t* sel;
    int32_t* count;
    int32_t* accepted;
    int32_t use_table;  // integer-count lookup of Poisson-deviance terms
    int32_t fixup;      // only redo references whose count is negative
    int32_t approx;     // screened kernel: zero bound, the screening distances decide
    // approx mode, volume source (or null): c = max(x * inv_scale, 0) per
    // voxel, and the sum of B(c) = c + c log2 c over the patch at each origin
    const float* cv;
    const float* boxb;
    // SSD noise-bias correction (blockmatching.py:1133-1139): distance -=
    // gamma * noise_ssd[offset of the candidate from the reference], or null
    const float* noise_ssd;
    float gamma;
    // Poisson SSD noise-bias correction (blockmatching.py:1140-1145,
    // :432-443): distance -= gamma * sum_p bias_scale * (r_p + c_p) over
    // r_p + c_p > 0, for every candidate but the reference itself
    int32_t poisson_bias;
    float bias_scale;
    // threshold computed on the device (one float), overrides the scalar one
    const float* thr_dev;
    int32_t no_alloc;  // 1: no stream-ordered scratch (approx mode then runs the bounded form)
    float* aux_ws;          // caller workspace for the approximate form's per-voxel arrays, or null
    int64_t aux_ws_floats;  // its size in floats
    char* ssd_ws;           // caller workspace for the tensor-core SSD matching, or null
    uint64_t ssd_ws_bytes;
    char* box_ws;           // caller scratch the box-sum matching may use, or null
    uint64_t box_ws_bytes;
    // subsampled mode: prescreen on the patch's even sub-lattice (box sums in
    // boxb_sub), then the screening form for the presel smallest
    int32_t sub;
    int32_t presel;
    const float* boxb_sub;
    // candidate standardisation (blockmatching.py:372-428): null means then
    // variances by pooled count 0..null_max, or null
    const double* null_moments;
    int32_t null_max;
};

constexpr int kTable = 64;  // counts 0..63 are tabulated

// 2 * [r ln(2r/s) + c ln(2c/s)] with the reference's float32 operation order
// (blockmatching.py:347-355); 0 when r + c == 0 (the term is skipped there)
__device__ __forceinline__ float deviance_term(float r, float c) {
    float s = add_rn(r, c);
    if (!(s > 0.0f)) return 0.0f;
    float contrib = 0.0f;
    if (r > 0.0f) contrib = add_rn(contrib, mul_rn(r, logf(div_rn(mul_rn(2.0f, r), s))));
    if (c > 0.0f) contrib = add_rn(contrib, mul_rn(c, logf(div_rn(mul_rn(2.0f, c), s))));
    return mul_rn(2.0f, contrib);
}

template <int CODE>
__device__ __forceinline__ float patch_distance(const float* __restrict__ ref,
                                                const float* __restrict__ src, int64_t origin,
                                                const int32_t* __restrict__ poff, int P,
                                                float inv) {
    float d = 0.0f;
    if (CODE == BMND_DIST_SSD) {
        for (int p = 0; p < P; ++p) {
            float diff = sub_rn(__ldg(src + origin + poff[p]), ref[p]);
            d = add_rn(d, mul_rn(diff, diff));
        }
        return d;
    }
    for (int p = 0; p < P; ++p) {
        float r = mul_rn(ref[p], inv);
        if (r < 0.0f) r = 0.0f;
        float c = mul_rn(__ldg(src + origin + poff[p]), inv);
        if (c < 0.0f) c = 0.0f;
        if (CODE == BMND_DIST_POISSON_DEVIANCE) {
            if (add_rn(r, c) > 0.0f) d = add_rn(d, deviance_term(r, c));
        } else if (CODE == BMND_DIST_PEARSON) {
            float s = add_rn(r, c);
            if (s > 0.0f) {
                float diff = sub_rn(c, r);
                d = add_rn(d, div_rn(mul_rn(diff, diff), s));
            }
        } else {
            float rs = mul_rn(2.0f, sqrtf(add_rn(r, 0.375f)));
            float cs = mul_rn(2.0f, sqrtf(add_rn(c, 0.375f)));
            float diff = sub_rn(cs, rs);
            d = add_rn(d, mul_rn(mul_rn(0.5f, diff), diff));
        }
    }
    if (d < 0.0f) d = 0.0f;
    return div_rn(d, static_cast<float>(P));
}

// Screening of one candidate with the ratio form
//   t = 2 ln 2 [r log2(2r/s) + c log2(2c/s)],  s = r + c,
// using the SFU reciprocal and log2.  Near r = c both logs are near zero and
// carry only the SFU's absolute error, so the form has no cancellation.
// Per term the screening error is below s (e_lg + 1.45 e_rcp + 2^-22.5 +
// 1.27 2^-23) in log2 units (r |log2 q_r| + c |log2 q_c| <= 1.27 s), and the
// exact float32 path's own error below 2^-21 s; the bound uses the sum of s
// over the patch.  kScreenAbs is that per-unit-s constant in distance units,
// times a safety factor 2, with the SFU errors e_lg, e_rcp measured on GB300
// over the argument ranges used here.
// measured: lg2.approx abs error <= 2^-22.06 max(|log2 x|, 1) (so r e_lg + c e_lg
// <= 2^-22.06 2.27 s), rcp.approx relative error <= 2^-23.28
constexpr float kScreenAbs = 2.0f * (1.38629436f * (5.41e-07f + 1.45f * 9.83e-08f + 1.69e-07f + 1.52e-07f) +
                                     4.77e-07f);

// SFU reciprocal and log2 of normal arguments (callers clamp to FLT_MIN)
__device__ __forceinline__ float sfu_rcp(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float sfu_lg2(float x) {
    float y;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// r2 = 2 r; returns r log2(2r/s) + c log2(2c/s)
__device__ __forceinline__ float ratio_term(float r, float r2, float c, float& ss) {
    const float kMin = 1.17549435e-38f;
    const float s = r + c;
    const float rs = sfu_rcp(fmaxf(s, kMin));
    const float lr = sfu_lg2(fmaxf(r2 * rs, kMin));
    const float lc = sfu_lg2(fmaxf((c + c) * rs, kMin));
    ss += s;
    return fmaf(r, lr, c * lc);
}

// exact float32 matching, one warp per reference (blockmatch.cu); with
// a.fixup set only the references whose count is negative are (re)done
int32_t launch_exact(MatchArgs& a, int code, cudaStream_t stream);

// whether exact requests take the kernel of tabulated count terms (blockmatch.cu)
bool counts_kernel_applies(const MatchArgs& a, int code);

// Box-sum matching (boxmatch.cu): *done is set when it ran; the references it
// leaves to the exact kernel have count = -1
int32_t launch_box_match(MatchArgs& a, int code, int precision, cudaStream_t stream, bool* done);
// the scratch it would use (zero: it does not take the matching)
BoxScratch box_match_scratch(const MatchArgs& a, int code, int precision);

}  // namespace bmnd
