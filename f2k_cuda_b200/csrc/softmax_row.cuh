// Per-row softmax arithmetic of the attention kernel: a thread owns one query row of a
// 128-key tile in registers (fp32 scores as loaded from tensor memory).
//
//   row_max64       maximum of 64 scores folded into 8 independent chains
//   exp_chunk16     P = 2^(c*s + neg_mc) for 16 scores -> 8 packed bf16 pairs, and the sum of
//                   the unrounded values (four partial sums)
//
// 2^x is the special-function unit's (ex2.approx, 4 lanes per clock per scheduler; the two softmax groups of a
// CTA share it). A cubic polynomial on the FMA pipe for some of the key pairs does not pay: 0, 1, 2 of 8 pairs
// 266, 268, 270 us at 4608 tokens x 32 heads (attention alone), 68, 68, 72 at 2125: it costs issue slots the row
// needs elsewhere.
#pragma once

#include "ptx.cuh"

namespace f2k {

// Running maxima of 64 scores folded into kMaxChains independent chains (3-input max, two new
// scores per step and chain); `first` starts the chains.
constexpr int kMaxChains = 8;
template <bool kFirst>
__device__ __forceinline__ void row_max64(const uint32_t* s, float (&m)[kMaxChains]) {
    using namespace f2k::ptx;
#pragma unroll
    for (int i = 0; i < 64; i += 2 * kMaxChains)
#pragma unroll
        for (int k = 0; k < kMaxChains; ++k) {
            const float a = __uint_as_float(s[i + 2 * k]), b = __uint_as_float(s[i + 2 * k + 1]);
            m[k] = (kFirst && i == 0) ? fmaxf(a, b) : fmax3(m[k], a, b);
        }
}
__device__ __forceinline__ float row_max_finish(const float (&m)[kMaxChains]) {
    using namespace f2k::ptx;
    return fmaxf(fmax3(m[0], m[1], m[2]), fmax3(fmax3(m[3], m[4], m[5]), m[6], m[7]));
}

// 16 scores -> 8 packed bf16 pairs.
__device__ __forceinline__ void exp_chunk16(const uint32_t* s, uint32_t* pk, float c, float neg_mc,
                                            float (&sum)[4]) {
    using namespace f2k::ptx;
#pragma unroll
    for (int i = 0; i < 16; i += 4) {
        float x0, x1, x2, x3;
        fma2(x0, x1, __uint_as_float(s[i + 0]), __uint_as_float(s[i + 1]), c, c, neg_mc, neg_mc);
        fma2(x2, x3, __uint_as_float(s[i + 2]), __uint_as_float(s[i + 3]), c, c, neg_mc, neg_mc);
        const float p0 = ex2_approx(x0), p1 = ex2_approx(x1), p2 = ex2_approx(x2), p3 = ex2_approx(x3);
        add2(sum[0], sum[1], sum[0], sum[1], p0, p1);
        add2(sum[2], sum[3], sum[2], sum[3], p2, p3);
        pk[i / 2 + 0] = pack_bf16x2(p0, p1);
        pk[i / 2 + 1] = pack_bf16x2(p2, p3);
    }
}

}  // namespace f2k
