// Tokens whose activations do not fit the products with codes in place, and the plain sums that stand in for them.
//
// Codes in place are bf16 subnormals (q * 2^-133) that meet activations times a power of two (qmv_frag.cuh).  A value that this takes past the
// largest bf16 would be an infinity; sums of a token of very small values lose bits; and an infinity would meet codes of zero and biases of the
// other sign (with f16 operands, which have none of the other limits, too).  Every result says which it may be: an infinity or a NaN comes out
// as one, and what has lost bits is tiny (sums err by 2^-139 units at most; a result of 2^-110 and more has its 24 bits all the same).  So
// the kernels that took over from ones that scale every row by itself look at the sums that they store.  Where one is odd, they look for
// tokens that are out of range and add those up from the definition, a warp an output (28672 x 4096 from L2, 8 tokens: 15 us, one of them out
// of range 320, a NaN 18).  With x times 2^96 that is a token with a value from 2^31 on, or all of them below 2^-64; one whose results all come out as zero, where
// its values lie below 2^-112, is left as it is.  (Noting the largest value of every token while it is staged costs 0.2 us a launch of 15, and
// looking for tokens behind every result of zero 2 to 4, with each token of zeros that fills up a batch.)
#pragma once

#include "common.cuh"

namespace mtc {
namespace far_tokens {

constexpr int kUp = 96, kUnit = 133 - kUp;      // x times 2^kUp; sums in units of 2^-kUnit

// v: a sum in those units (f16: 2^-24)
template <int XT>
__device__ __forceinline__ bool odd(float v) {
    const float m = fabsf(v);
    return !(m < __int_as_float(0x7F800000) && (XT == MTC_F16 || m >= __int_as_float((127 - 110) << 23) || m == 0.0f));
}

// Whether the token x[0 .. K) is out of range, by one warp.  A NaN leaves no mark (the products carry it).
template <int XT>
__device__ __forceinline__ bool out_of_range(const void *x, int K) {
    constexpr uint32_t above = XT == MTC_F32 ? (254u - kUp) << 23 : XT == MTC_BF16 ? (254u - kUp) << 7 : 0x7C00u;
    constexpr uint32_t enough = XT == MTC_F32 ? (127u - 64u) << 23 : XT == MTC_BF16 ? (127u - 64u) << 7 : 1u;
    constexpr uint32_t nan = XT == MTC_F32 ? 0x7F800000u : XT == MTC_BF16 ? 0x7F80u : 0x7C00u;
    uint32_t m = 0;
    const uint4 *const p = static_cast<const uint4 *>(x);
#pragma unroll 8
    for (int i = threadIdx.x & 31; i < K / (XT == MTC_F32 ? 4 : 8); i += 32) {
        const uint4 q = p[i];
        const uint32_t v[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint32_t lo = XT == MTC_F32 ? v[j] & 0x7FFFFFFFu : v[j] & 0x7FFFu, hi = XT == MTC_F32 ? 0u : v[j] >> 16 & 0x7FFFu;
            m = max(m, max(lo > nan ? 0u : lo, hi > nan ? 0u : hi));
        }
    }
    m = __reduce_max_sync(0xffffffffu, m);
    return m != 0 && m - enough >= above - enough;
}

// One output by one warp: the definition, in f32.  K a multiple of 32, groups of 32 and more.
template <int BITS, int XT>
__device__ __forceinline__ float sum(const uint32_t *w, const void *scales, const void *biases, const void *x, int K, int gs_shift) {
    float acc = 0.0f;
#pragma unroll 1
    for (int c = threadIdx.x & 31; c < K >> 5; c += 32) {
        const float s = ld_as_f32(scales, (c << 5) >> gs_shift, XT), b = ld_as_f32(biases, (c << 5) >> gs_shift, XT);
        float part = 0.0f;
#pragma unroll 1
        for (int i = 0; i < 32; ++i) {
            const int k = (c << 5) + i;
            part = fmaf(fmaf(static_cast<float>(code_at(w, k, BITS)), s, b), ld_written_as_f32(x, k, XT), part);
        }
        acc += part;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    return acc;
}

}  // namespace far_tokens
}  // namespace mtc
