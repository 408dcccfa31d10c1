// affine — the codec either side of the quantized matmuls: float tensor -> packed codes + per-group scale / bias, and back.
//
//   quantize   per group of G values:  scale = (max - min) / (2^b - 1)  (1 when below 1e-7),  bias = min,
//              q = trunc(clamp((v - bias) * (1 / scale) + 0.5, 0, 2^b - 1));  codes packed LSB-first, one bit-stream per
//              group; scale and bias stored in the activation type
//   dequantize out[i] = scale[i / G] * q_i + bias[i / G], rounded to the activation type
//
// Stands in for mt_affine_quantize_int{2,3,4,5,6,8} and mt_affine_dequantize_int{2,3,4,5,6,8}
// (crates/metaltile-std/src/mlx/quantized.rs:3575-4214; one template there too).  Every float operation is a separately
// rounded f32 operation (no fused multiply-add), so codes and values are those of the scalar CPU formula bit for bit.
// Both are passes over data that is touched once (weights are quantized at load time); the rate of memory is the bound, the
// instructions of each value come close to it.
#include "common.cuh"

namespace mtc {
namespace {

template <int BITS>
__device__ __forceinline__ uint32_t code_of(const uint32_t (&w)[BITS], int k) {      // k: compile-time after unrolling
    const int bit = k * BITS, word = bit >> 5, sh = bit & 31;
    uint32_t q = w[word] >> sh;
    if (sh + BITS > 32) q |= w[word + 1] << (32 - sh);
    return q & ((1u << BITS) - 1u);
}

// ---- units of 8 values -------------------------------------------------------------------------------------------
// The codec moves 2 bytes a value (16-bit types) plus b / 8 and touches each once, so it should run at the rate of memory.
// Two things kept the forms with 32 consecutive values per thread at 62 % of that: neighbouring lanes 64 bytes apart (every
// 16-byte access touches 32 half-used sectors), and a float <-> integer conversion per value (16 a clock and SM: 13 us of
// the 23 that 14336 x 4096 bf16 values take).  So here a lane owns 8 consecutive values = b whole bytes of codes and 16
// bytes of 16-bit values - a warp's accesses are contiguous - with kUnits such units per lane in flight, and the
// conversions go through the f32 binade [2^23, 2^24), where one unit in the last place is 1: 2^23 + q is 0x4B000000 | q
// exactly, and adding 2^23 with rounding toward zero truncates.  4-bit groups of 64, 14336 x 4096 bf16: quantize 39.1 -> 27.7 us,
// dequantize 38.9 -> 27.3 us (23 us at the copy rate).
constexpr int kUnits = 4;                              // units per lane: a warp covers 1024 consecutive values
constexpr uint32_t kTwo23 = 0x4B000000u;               // 2^23 as f32

// The b bytes of codes of unit i, first code in the low bits.  3 / 5 / 6-bit units start inside a word: two words and a shift
// (the second word only where the unit reaches it, so nothing past the last unit is read).
template <int BITS>
__device__ __forceinline__ uint64_t ld_codes(const uint32_t *w, uint32_t i) {
    if (BITS == 8) return w[2 * i] | static_cast<uint64_t>(w[2 * i + 1]) << 32;
    if (BITS == 4) return w[i];
    if (BITS == 2) return reinterpret_cast<const uint16_t *>(w)[i];
    const uint32_t at = i * BITS, sh = (at & 3) * 8;       // byte, bit of its word
    const uint32_t *p = w + (at >> 2);
    return (p[0] | static_cast<uint64_t>(p[sh + 8 * BITS > 32 ? 1 : 0]) << 32) >> sh;
}
// Eight codes of a unit in two words of four (lo, hi: code k at bit (k & 3) * BITS) to the b bytes of unit i.  Every lane of a
// warp calls it (3 / 5 / 6-bit: the four lanes of a quad hold b whole words, and a lane that stores one gets the other half of it from a neighbour);
// `on` is the same for the lanes of a quad.
template <int BITS>
__device__ __forceinline__ void st_codes(uint32_t *out, uint32_t i, uint32_t lo, uint32_t hi, bool on) {
    if (BITS == 8) {
        if (on) reinterpret_cast<uint2 *>(out)[i] = make_uint2(lo, hi);
    } else if (BITS == 4) {
        if (on) out[i] = lo | hi << 16;
    } else if (BITS == 2) {
        if (on) reinterpret_cast<uint16_t *>(out)[i] = static_cast<uint16_t>(lo | hi << 8);
    } else {
        const uint64_t v = lo | static_cast<uint64_t>(hi) << (4 * BITS);
        const uint32_t t = threadIdx.x & 3;
        uint32_t *q = out + (i >> 2) * BITS;
        if (BITS == 3) {                                               // word t: the rest of unit t, the start of unit t + 1
            const uint32_t nb = __shfl_down_sync(0xffffffffu, static_cast<uint32_t>(v), 1);
            if (on && t < 3) q[t] = (static_cast<uint32_t>(v) >> (8 * t)) | (nb << (24 - 8 * t));
        } else if (BITS == 5) {                                        // word t: the end of unit t - 1, the start of unit t; word 4: the end of unit 3
            const uint32_t end = static_cast<uint32_t>(v >> 8), nb = __shfl_up_sync(0xffffffffu, end, 1);
            if (on) q[t] = static_cast<uint32_t>(v << (8 * t)) | (t ? nb >> (32 - 8 * t) : 0u);
            if (on && t == 3) q[4] = end;
        } else {                                                       // a pair of lanes holds three words
            const uint32_t nb = __shfl_xor_sync(0xffffffffu, static_cast<uint32_t>(v), 1);
            uint32_t *q3 = q + (t >> 1) * 3;
            if (on && !(t & 1)) {
                q3[0] = static_cast<uint32_t>(v);
                q3[1] = static_cast<uint32_t>(v >> 32) | nb << 16;
            }
            if (on && (t & 1)) q3[2] = static_cast<uint32_t>(v >> 16);
        }
    }
}
// two f32 operations an instruction, each rounded on its own
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
    float2 r;
    asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tadd.rn.f32x2 z, x, y;\n\tmov.b64 {%0, %1}, z;\n\t}"
        : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return r;
}
__device__ __forceinline__ float2 add2_rz(float2 a, float2 b) {
    float2 r;
    asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tadd.rz.f32x2 z, x, y;\n\tmov.b64 {%0, %1}, z;\n\t}"
        : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return r;
}
// (products one at a time: the paired product and a paired sum behind it came out as one fused operation)
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return make_float2(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y)); }
// code k of a unit as the float 2^23 + q
template <int BITS>
__device__ __forceinline__ float code_2_23(uint64_t codes, int k) {          // k: compile-time after unrolling
    if (BITS == 8) return __uint_as_float(__byte_perm(static_cast<uint32_t>(codes >> (k < 4 ? 0 : 32)), kTwo23, 0x7440 | (k & 3)));
    if (BITS == 4) return __uint_as_float(__byte_perm(static_cast<uint32_t>(codes >> ((k & 1) * 4)) & 0x0F0F0F0Fu, kTwo23, 0x7440 | (k >> 1)));
    return __uint_as_float((static_cast<uint32_t>(codes >> (k * BITS)) & ((1u << BITS) - 1u)) | kTwo23);
}

// Group sizes that are multiples of 32.  upg_log2 >= 0: units per group as a power of two (a shift instead of a division).
template <int BITS, int DT>
__global__ void __launch_bounds__(256) affine_dequantize_kernel(const uint32_t *w, const void *scales, const void *biases, void *out,
                                                                size_t n_units, int units_per_group, int upg_log2, int vec_ok) {
    pdl_enter();
    const int lane = threadIdx.x & 31;
    const size_t nwarps = (static_cast<size_t>(gridDim.x) * blockDim.x) >> 5;
    for (size_t base = ((blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x) >> 5) * (32 * kUnits); base < n_units;
         base += nwarps * (32 * kUnits)) {
        uint64_t codes[kUnits];
        float s[kUnits], b[kUnits];
        // 32-bit offsets inside the warp's 128 units; those past the end read unit 0 of the tile
        const uint32_t rem = static_cast<uint32_t>(n_units - base < 32 * kUnits ? n_units - base : 32 * kUnits);
        const uint32_t *wt = w + base / 4 * BITS;
        const size_t g0 = upg_log2 >= 0 ? base >> upg_log2 : 0;
#pragma unroll
        for (int u = 0; u < kUnits; ++u) {
            const uint32_t off = u * 32 + lane, at = off < rem ? off : 0;
            // power of two: the tile starts on a group, or lies inside one
            const size_t g = upg_log2 >= 0 ? g0 + (at >> upg_log2) : (base + at) / units_per_group;
            codes[u] = ld_codes<BITS>(wt, at);
            s[u] = ld_written_as_f32(scales, g, DT);
            b[u] = ld_written_as_f32(biases, g, DT);
        }
#pragma unroll
        for (int u = 0; u < kUnits; ++u) {
            const uint32_t off = u * 32 + lane;
            const size_t i = base + off;
            float v[8];
#pragma unroll
            for (int k = 0; k < 8; k += 2) {
                const float2 q = add2(make_float2(code_2_23<BITS>(codes[u], k), code_2_23<BITS>(codes[u], k + 1)), make_float2(-8388608.0f, -8388608.0f));
                const float2 r = add2(mul2(make_float2(s[u], s[u]), q), make_float2(b[u], b[u]));
                v[k] = r.x;
                v[k + 1] = r.y;
            }
            if (off >= rem) break;
            if (DT == MTC_F32) {
                float *o = static_cast<float *>(out) + i * 8;
                if (vec_ok) {
                    reinterpret_cast<float4 *>(o)[0] = make_float4(v[0], v[1], v[2], v[3]);
                    reinterpret_cast<float4 *>(o)[1] = make_float4(v[4], v[5], v[6], v[7]);
                } else {
#pragma unroll
                    for (int k = 0; k < 8; ++k) o[k] = v[k];
                }
            } else {
                if (vec_ok) {
                    uint32_t h[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        if (DT == MTC_BF16) {
                            const __nv_bfloat162 p2 = __floats2bfloat162_rn(v[2 * q], v[2 * q + 1]);
                            h[q] = *reinterpret_cast<const uint32_t *>(&p2);
                        } else {
                            const __half2 p2 = __floats2half2_rn(v[2 * q], v[2 * q + 1]);
                            h[q] = *reinterpret_cast<const uint32_t *>(&p2);
                        }
                    }
                    reinterpret_cast<uint4 *>(out)[i] = make_uint4(h[0], h[1], h[2], h[3]);
                } else {
#pragma unroll
                    for (int k = 0; k < 8; ++k) st_from_f32(out, i * 8 + k, v[k], DT);
                }
            }
        }
    }
}

// One warp per group (group_size % 32 == 0): min / max by shuffles, then 32 codes at a time - lane L owns code L of the
// chunk, the chunk's BITS words are OR-reduced over the warp and written by lanes 0 .. BITS-1.
template <int BITS>
__global__ void __launch_bounds__(256) affine_quantize_kernel(const void *w, uint32_t *out, void *scales, void *biases, size_t n_groups,
                                                              int group_size, int dt) {
    const int lane = threadIdx.x & 31;
    const size_t warp0 = (blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x) >> 5;
    const size_t nwarps = (static_cast<size_t>(gridDim.x) * blockDim.x) >> 5;
    const float n_bins = static_cast<float>((1u << BITS) - 1u);
    const int chunks = group_size >> 5;
    for (size_t g = warp0; g < n_groups; g += nwarps) {
        const size_t base = g * group_size;
        float mn = INFINITY, mx = -INFINITY;
        for (int c = 0; c < chunks; ++c) {
            const float v = ld_as_f32(w, base + c * 32 + lane, dt);
            mn = fminf(mn, v);
            mx = fmaxf(mx, v);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        }
        const float raw = __fdiv_rn(__fsub_rn(mx, mn), n_bins);
        const float scale = raw < 1.0e-7f ? 1.0f : raw;
        const float inv = __fdiv_rn(1.0f, scale);
        if (lane == 0) {
            st_from_f32(scales, g, scale, dt);
            st_from_f32(biases, g, mn, dt);
        }
        uint32_t *og = out + g * (static_cast<size_t>(group_size) * BITS / 32);
        const int bit = lane * BITS, word = bit >> 5, sh = bit & 31;
        for (int c = 0; c < chunks; ++c) {
            const float v = ld_as_f32(w, base + c * 32 + lane, dt);
            float qf = __fadd_rn(__fmul_rn(__fsub_rn(v, mn), inv), 0.5f);
            qf = qf > n_bins ? n_bins : (qf < 0.0f ? 0.0f : qf);
            const uint32_t q = static_cast<uint32_t>(qf);
            uint32_t mine = 0u;
#pragma unroll
            for (int j = 0; j < BITS; ++j) {
                uint32_t part = 0u;
                if (word == j) part = q << sh;
                if (word + 1 == j && sh + BITS > 32) part = q >> (32 - sh);
                const uint32_t all = __reduce_or_sync(0xffffffffu, part);
                if (lane == j) mine = all;
            }
            if (lane < BITS) og[c * BITS + lane] = mine;
        }
    }
}

// Units of 8 values again; a group (32 .. 1024 values, a power of two) is 4 .. 32 lanes of one unit index, or 2 / 4 whole
// unit indexes.  Every lane needs the range of its four groups, but the two divisions behind a scale are 20 instructions
// each: the reduction over the lanes leaves unit index (lane & 3) in a lane (two exchanges that halve what is left, then
// plain xor steps), the lane divides for that one, and the four lanes of a quad hand out (minimum, 1 / scale).  Minimum and
// negated maximum travel as one pair, packed in one register for 16-bit types (both are exact there).  `w` 16-byte, 8-bit
// `out` 8-byte aligned.
//
// No upper clamp: d = v - mn <= D = mx - mn as rounded, scale = rn(D / n) and 1 / scale are within 2^-22 of exact (a
// subnormal reciprocal of a scale above 2^126 included), so d / scale <= n (1 + 2^-20) and + 0.5 stays below n + 1 for
// n <= 255.  max(t, 0) turns a NaN into code 0.
template <int DT>
struct QzRange {
    uint32_t a, b;                                     // 16-bit: a = (min, -max) packed; f32: a = min, b = -max (bits)
    static __device__ __forceinline__ uint32_t min16(uint32_t x, uint32_t y) {
        uint32_t r;
        if (DT == MTC_BF16) asm("min.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(x), "r"(y));
        else asm("min.f16x2 %0, %1, %2;" : "=r"(r) : "r"(x), "r"(y));
        return r;
    }
    static __device__ __forceinline__ uint32_t max16(uint32_t x, uint32_t y) {
        uint32_t r;
        if (DT == MTC_BF16) asm("max.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(x), "r"(y));
        else asm("max.f16x2 %0, %1, %2;" : "=r"(r) : "r"(x), "r"(y));
        return r;
    }
    __device__ __forceinline__ void merge(uint32_t oa, uint32_t ob) {
        if (DT == MTC_F32) {
            a = __float_as_uint(fminf(__uint_as_float(a), __uint_as_float(oa)));
            b = __float_as_uint(fminf(__uint_as_float(b), __uint_as_float(ob)));
        } else {
            a = min16(a, oa);
        }
    }
    __device__ __forceinline__ void merge_xor(int o) {
        const uint32_t oa = __shfl_xor_sync(0xffffffffu, a, o);
        merge(oa, DT == MTC_F32 ? __shfl_xor_sync(0xffffffffu, b, o) : 0u);
    }
    __device__ __forceinline__ float lo() const {
        if (DT == MTC_F32) return __uint_as_float(a);
        if (DT == MTC_BF16) return __uint_as_float(a << 16);
        return __low2float(*reinterpret_cast<const __half2 *>(&a));
    }
    __device__ __forceinline__ float hi() const {
        if (DT == MTC_F32) return -__uint_as_float(b);
        if (DT == MTC_BF16) return -__uint_as_float(a & 0xFFFF0000u);
        return -__high2float(*reinterpret_cast<const __half2 *>(&a));
    }
};

template <int BITS, int DT>
__global__ void __launch_bounds__(256) affine_quantize8_kernel(const void *w, uint32_t *out, void *scales, void *biases, size_t n_units,
                                                               int gs_log2) {
    constexpr int RW = DT == MTC_F32 ? 8 : 4;          // words of a unit's values
    constexpr float n_bins = static_cast<float>((1u << BITS) - 1u);
    using Range = QzRange<DT>;
    // launched while the previous kernel drains, but it does not let the next one start early: a product may request its
    // weights before the kernel in front of it is complete, and this kernel writes weights
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int lane = threadIdx.x & 31;
    const int lpg = gs_log2 >= 8 ? 32 : 1 << (gs_log2 - 3);        // lanes of one unit index that share a group: 4 .. 32
    const size_t nwarps = (static_cast<size_t>(gridDim.x) * blockDim.x) >> 5;
    // whole warps stay in the loop (the shuffles need every lane); lanes past the end work on unit 0 of the tile and store nothing
    for (size_t base = ((blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x) >> 5) * (32 * kUnits); base < n_units;
         base += nwarps * (32 * kUnits)) {
        uint32_t raw[kUnits][RW];
        // 32-bit offsets inside the warp's 128 units
        const uint32_t rem = static_cast<uint32_t>(n_units - base < 32 * kUnits ? n_units - base : 32 * kUnits);
        const uint4 *wt = static_cast<const uint4 *>(w) + base * (RW / 4);
        uint32_t *ot = out + base / 4 * BITS;
#pragma unroll
        for (int u = 0; u < kUnits; ++u) {
            const uint32_t off = u * 32 + lane, at = off < rem ? off : 0;
#pragma unroll
            for (int q = 0; q < RW / 4; ++q) {
                const uint4 t = wt[at * (RW / 4) + q];
                raw[u][4 * q] = t.x; raw[u][4 * q + 1] = t.y; raw[u][4 * q + 2] = t.z; raw[u][4 * q + 3] = t.w;
            }
        }
        Range r[kUnits];
#pragma unroll
        for (int u = 0; u < kUnits; ++u) {
            if (DT == MTC_F32) {
                float mn = __uint_as_float(raw[u][0]), mx = mn;
#pragma unroll
                for (int k = 1; k < RW; ++k) {
                    mn = fminf(mn, __uint_as_float(raw[u][k]));
                    mx = fmaxf(mx, __uint_as_float(raw[u][k]));
                }
                r[u].a = __float_as_uint(mn);
                r[u].b = __float_as_uint(-mx);
            } else {
                const uint32_t mn = Range::min16(Range::min16(raw[u][0], raw[u][1]), Range::min16(raw[u][2], raw[u][3]));
                const uint32_t mx = Range::max16(Range::max16(raw[u][0], raw[u][1]), Range::max16(raw[u][2], raw[u][3]));
                r[u].a = Range::min16(__byte_perm(mn, mx, 0x5410) ^ 0x80000000u, __byte_perm(mn, mx, 0x7632) ^ 0x80000000u);      // even values with odd ones
                r[u].b = 0u;
            }
        }
        // lanes with bit 0 set keep units 1 and 3, the others 0 and 2; then bit 1 decides between the pair
        const bool o1 = lane & 1, o2 = lane & 2;
        Range k0 = o1 ? r[1] : r[0], k1 = o1 ? r[3] : r[2];
        const Range s0 = o1 ? r[0] : r[1], s1 = o1 ? r[2] : r[3];
        k0.merge(__shfl_xor_sync(0xffffffffu, s0.a, 1), DT == MTC_F32 ? __shfl_xor_sync(0xffffffffu, s0.b, 1) : 0u);
        k1.merge(__shfl_xor_sync(0xffffffffu, s1.a, 1), DT == MTC_F32 ? __shfl_xor_sync(0xffffffffu, s1.b, 1) : 0u);
        Range m = o2 ? k1 : k0;
        const Range s2 = o2 ? k0 : k1;
        m.merge(__shfl_xor_sync(0xffffffffu, s2.a, 2), DT == MTC_F32 ? __shfl_xor_sync(0xffffffffu, s2.b, 2) : 0u);
        for (int o = 4; o < lpg; o <<= 1) m.merge_xor(o);
        if (gs_log2 >= 9) m.merge_xor(1);                          // 512 values: unit indexes 0 and 1, 2 and 3
        if (gs_log2 >= 10) m.merge_xor(2);                         // 1024: all four
        // the scalar formula starts from +inf and -inf, which is what a group of nothing but NaN keeps (scale 1, bias +inf)
        const float my_mn = fminf(m.lo(), INFINITY);
        const float div = __fdiv_rn(__fsub_rn(fmaxf(m.hi(), -INFINITY), my_mn), n_bins);
        const float scale = div < 1.0e-7f ? 1.0f : div;
        const float my_inv = __fdiv_rn(1.0f, scale);
        {   // the first lanes of a group hold its unit indexes: lane j of them stores the scale and bias of index j
            const int u = lane & 3;
            const size_t i = base + u * 32 + (lane & ~(lpg - 1));  // first unit of the group of index u
            const size_t v0 = i * 8;
            if ((lane & (lpg - 1)) == u && i < n_units && (v0 & ((size_t{1} << gs_log2) - 1)) == 0) {
                st_from_f32(scales, v0 >> gs_log2, scale, DT);
                st_from_f32(biases, v0 >> gs_log2, my_mn, DT);
            }
        }
#pragma unroll
        for (int u = 0; u < kUnits; ++u) {
            const float mn = __shfl_sync(0xffffffffu, my_mn, (lane & ~3) | u), inv = __shfl_sync(0xffffffffu, my_inv, (lane & ~3) | u);
            // the bits of 2^23 + q are summed as they are; what their exponents add to each word (mod 2^32) leaves once
            constexpr uint32_t exps = kTwo23 + (kTwo23 << BITS) + (kTwo23 << (2 * BITS)) + (kTwo23 << (3 * BITS));
            uint32_t half[2] = {0u - exps, 0u - exps};
#pragma unroll
            for (int k = 0; k < 8; k += 2) {
                float2 v;
                if (DT == MTC_F32) v = make_float2(__uint_as_float(raw[u][k & (RW - 1)]), __uint_as_float(raw[u][(k + 1) & (RW - 1)]));
                else if (DT == MTC_BF16) v = make_float2(__uint_as_float(raw[u][k >> 1] << 16), __uint_as_float(raw[u][k >> 1] & 0xFFFF0000u));
                else v = __half22float2(*reinterpret_cast<const __half2 *>(&raw[u][k >> 1]));
                float2 c = add2(mul2(add2(v, make_float2(-mn, -mn)), make_float2(inv, inv)), make_float2(0.5f, 0.5f));
                c = add2_rz(make_float2(fmaxf(c.x, 0.0f), fmaxf(c.y, 0.0f)), make_float2(8388608.0f, 8388608.0f));
                half[k >> 2] += (__float_as_uint(c.x) << ((k & 3) * BITS)) + (__float_as_uint(c.y) << (((k + 1) & 3) * BITS));
            }
            const uint32_t off = u * 32 + lane;
            st_codes<BITS>(ot, off, half[0], half[1], off < rem);
        }
    }
}

// dequant_gather_int* (crates/metaltile-std/src/ffai/dequant_gather.rs:44-94): rows indices[t] of a quantized table
// [vocab, hidden], dequantized into out [n_tokens, hidden].  One thread per 32 values of an output row (hidden and the
// group size are multiples of 32); an index outside the table reads row 0 and is reported (status 0x904).
template <int BITS>
__global__ void __launch_bounds__(256) dequant_gather_kernel(const uint32_t *w, const void *scales, const void *biases,
                                                             const uint32_t *indices, void *out, size_t n_tokens, int hidden,
                                                             int group_size, int vocab, int dt, int vec_ok, uint32_t *status) {
    const int cpr = hidden >> 5;                                   // chunks per row
    const size_t n_chunks = n_tokens * cpr;
    for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < n_chunks;
         i += static_cast<size_t>(gridDim.x) * blockDim.x) {
        const size_t tok = i / cpr;
        const int c = static_cast<int>(i - tok * cpr);
        uint32_t row = __ldg(indices + tok);
        if (row >= static_cast<uint32_t>(vocab)) {
            atomicCAS(status, 0u, 0x904u);
            row = 0;
        }
        const uint32_t *rw = w + (static_cast<size_t>(row) * cpr + c) * BITS;
        uint32_t words[BITS];
#pragma unroll
        for (int j = 0; j < BITS; ++j) words[j] = __ldg(rw + j);
        const size_t g = static_cast<size_t>(row) * (hidden / group_size) + (c * 32) / group_size;
        const float s = ld_as_f32(scales, g, dt), b = ld_as_f32(biases, g, dt);
        float v[32];
#pragma unroll
        for (int k = 0; k < 32; ++k) v[k] = __fadd_rn(__fmul_rn(static_cast<float>(code_of<BITS>(words, k)), s), b);
        const size_t o = tok * hidden + c * 32;
        if (dt == MTC_F32) {
#pragma unroll
            for (int k = 0; k < 32; ++k) static_cast<float *>(out)[o + k] = v[k];
        } else {
            uint32_t h[16];
#pragma unroll
            for (int q = 0; q < 16; ++q) {
                if (dt == MTC_BF16) {
                    const __nv_bfloat162 p2 = __floats2bfloat162_rn(v[2 * q], v[2 * q + 1]);
                    h[q] = *reinterpret_cast<const uint32_t *>(&p2);
                } else {
                    const __half2 p2 = __floats2half2_rn(v[2 * q], v[2 * q + 1]);
                    h[q] = *reinterpret_cast<const uint32_t *>(&p2);
                }
            }
            if (vec_ok) {
                uint4 *p = reinterpret_cast<uint4 *>(static_cast<uint16_t *>(out) + o);
#pragma unroll
                for (int q = 0; q < 4; ++q) p[q] = make_uint4(h[4 * q], h[4 * q + 1], h[4 * q + 2], h[4 * q + 3]);
            } else {
                uint16_t *p = static_cast<uint16_t *>(out) + o;
#pragma unroll
                for (int q = 0; q < 16; ++q) {
                    p[2 * q] = static_cast<uint16_t>(h[q] & 0xFFFFu);
                    p[2 * q + 1] = static_cast<uint16_t>(h[q] >> 16);
                }
            }
        }
    }
}

// any hidden / group size: one thread per output element
__global__ void __launch_bounds__(256) dequant_gather_generic(const uint32_t *w, const void *scales, const void *biases,
                                                              const uint32_t *indices, void *out, size_t n_tokens, int hidden,
                                                              int group_size, int vocab, int bits, int dt, uint32_t *status) {
    const size_t n = n_tokens * hidden;
    const size_t wpr = static_cast<size_t>(hidden) * bits / 32;
    for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < n; i += static_cast<size_t>(gridDim.x) * blockDim.x) {
        const size_t tok = i / hidden;
        const uint32_t d = static_cast<uint32_t>(i - tok * hidden);
        uint32_t row = __ldg(indices + tok);
        if (row >= static_cast<uint32_t>(vocab)) {
            atomicCAS(status, 0u, 0x904u);
            row = 0;
        }
        const float q = static_cast<float>(code_at(w + row * wpr, d, bits));
        const size_t g = static_cast<size_t>(row) * (hidden / group_size) + d / group_size;
        st_from_f32(out, i, __fadd_rn(__fmul_rn(q, ld_as_f32(scales, g, dt)), ld_as_f32(biases, g, dt)), dt);
    }
}

// any group size, any alignment: one thread per element (dequantize) / one thread per group (quantize)
__global__ void __launch_bounds__(256) affine_dequantize_generic(const uint32_t *w, const void *scales, const void *biases, void *out,
                                                                 size_t n_elem, int group_size, int bits, int dt) {
    for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < n_elem;
         i += static_cast<size_t>(gridDim.x) * blockDim.x) {
        const size_t g = i / group_size;
        // the stream restarts at every group: group_size * bits is a multiple of 32
        const uint32_t *gw = w + g * (static_cast<size_t>(group_size) * bits / 32);
        const float q = static_cast<float>(code_at(gw, static_cast<uint32_t>(i - g * group_size), bits));
        st_from_f32(out, i, __fadd_rn(__fmul_rn(ld_as_f32(scales, g, dt), q), ld_as_f32(biases, g, dt)), dt);
    }
}

__global__ void __launch_bounds__(128) affine_quantize_generic(const void *w, uint32_t *out, void *scales, void *biases, size_t n_groups,
                                                               int group_size, int bits, int dt) {
    const float n_bins = static_cast<float>((1u << bits) - 1u);
    for (size_t g = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; g < n_groups;
         g += static_cast<size_t>(gridDim.x) * blockDim.x) {
        const size_t base = g * group_size;
        float mn = INFINITY, mx = -INFINITY;
        for (int i = 0; i < group_size; ++i) {
            const float v = ld_as_f32(w, base + i, dt);
            mn = fminf(mn, v);
            mx = fmaxf(mx, v);
        }
        const float raw = __fdiv_rn(__fsub_rn(mx, mn), n_bins);
        const float scale = raw < 1.0e-7f ? 1.0f : raw;
        const float inv = __fdiv_rn(1.0f, scale);
        st_from_f32(scales, g, scale, dt);
        st_from_f32(biases, g, mn, dt);
        const size_t wpg = static_cast<size_t>(group_size) * bits / 32;
        uint32_t *og = out + g * wpg;
        uint32_t cur = 0u;
        for (int i = 0; i < group_size; ++i) {
            float qf = __fadd_rn(__fmul_rn(__fsub_rn(ld_as_f32(w, base + i, dt), mn), inv), 0.5f);
            qf = qf > n_bins ? n_bins : (qf < 0.0f ? 0.0f : qf);
            const uint32_t q = static_cast<uint32_t>(qf);
            const int bit = i * bits, sh = bit & 31;
            cur |= q << sh;
            if (sh + bits >= 32) {
                og[bit >> 5] = cur;
                cur = sh + bits > 32 ? q >> (32 - sh) : 0u;
            }
        }
    }
}

int grid_for(size_t work, int per_block, int sms) {
    size_t g = (work + per_block - 1) / per_block;
    const size_t cap = static_cast<size_t>(sms) * 16;
    if (g > cap) g = cap;
    return g < 1 ? 1 : static_cast<int>(g);
}

int pow2_log2(int v) {                                 // -1: not a power of two
    int l = 0;
    while ((1 << l) < v) ++l;
    return (1 << l) == v ? l : -1;
}

int unit_grid(size_t units) {                          // one pass of 8 warps per block; beyond 2^20 blocks the kernels loop
    const size_t g = (units + 256 * kUnits - 1) / (256 * kUnits);
    return static_cast<int>(g > (size_t{1} << 20) ? size_t{1} << 20 : g);
}

}  // namespace

cudaError_t launch_affine_dequantize(Ctx *ctx, cudaStream_t st, const void *w, const void *scales, const void *biases, void *out,
                                     size_t n_elem, int bits, int group_size, int dt) {
    if (n_elem == 0) return cudaSuccess;
    const uint32_t *ww = static_cast<const uint32_t *>(w);
    if (group_size % 32 != 0 || n_elem % 32 != 0) {
        affine_dequantize_generic<<<grid_for(n_elem, 256, ctx->sm_count), 256, 0, st>>>(ww, scales, biases, out, n_elem, group_size, bits, dt);
        return cudaGetLastError();
    }
    const size_t units = n_elem / 8;
    const int vec_ok = reinterpret_cast<uintptr_t>(out) % 16 == 0 ? 1 : 0;
    const int grid = unit_grid(units), upg = group_size / 8, lg = pow2_log2(upg);
    cudaError_t e = cudaSuccess;
#define MTC_DQ(B)                                                                                                              \
    e = launch_pdl(dt == MTC_F32 ? affine_dequantize_kernel<B, MTC_F32> : dt == MTC_F16 ? affine_dequantize_kernel<B, MTC_F16> \
                                                                                        : affine_dequantize_kernel<B, MTC_BF16>, \
                   grid, 256, 0, st, ww, scales, biases, out, units, upg, lg, vec_ok)
    switch (bits) {
        case 2: MTC_DQ(2); break;
        case 3: MTC_DQ(3); break;
        case 4: MTC_DQ(4); break;
        case 5: MTC_DQ(5); break;
        case 6: MTC_DQ(6); break;
        default: MTC_DQ(8); break;
    }
#undef MTC_DQ
    return e;
}

cudaError_t launch_dequant_gather(Ctx *ctx, cudaStream_t st, const void *w, const void *scales, const void *biases, const void *indices,
                                  void *out, size_t n_tokens, int hidden, int vocab, int bits, int group_size, int dt) {
    if (n_tokens == 0 || hidden == 0) return cudaSuccess;
    const uint32_t *ww = static_cast<const uint32_t *>(w), *ix = static_cast<const uint32_t *>(indices);
    if (hidden % 32 != 0 || group_size % 32 != 0) {
        dequant_gather_generic<<<grid_for(n_tokens * hidden, 256, ctx->sm_count), 256, 0, st>>>(ww, scales, biases, ix, out, n_tokens, hidden,
                                                                                              group_size, vocab, bits, dt, ctx->d_status);
        return cudaGetLastError();
    }
    const int vec_ok = reinterpret_cast<uintptr_t>(out) % 16 == 0 ? 1 : 0;
    const int grid = grid_for(n_tokens * (hidden / 32), 256, ctx->sm_count);
#define MTC_DG(B) dequant_gather_kernel<B><<<grid, 256, 0, st>>>(ww, scales, biases, ix, out, n_tokens, hidden, group_size, vocab, dt, vec_ok, ctx->d_status)
    switch (bits) {
        case 2: MTC_DG(2); break;
        case 3: MTC_DG(3); break;
        case 4: MTC_DG(4); break;
        case 5: MTC_DG(5); break;
        case 6: MTC_DG(6); break;
        default: MTC_DG(8); break;
    }
#undef MTC_DG
    return cudaGetLastError();
}

cudaError_t launch_affine_quantize(Ctx *ctx, cudaStream_t st, const void *w, void *out, void *scales, void *biases, size_t n_groups,
                                   int bits, int group_size, int dt) {
    if (n_groups == 0) return cudaSuccess;
    uint32_t *oo = static_cast<uint32_t *>(out);
    if (group_size % 32 != 0) {
        affine_quantize_generic<<<grid_for(n_groups, 128, ctx->sm_count), 128, 0, st>>>(w, oo, scales, biases, n_groups, group_size, bits, dt);
        return cudaGetLastError();
    }
    const int lg = pow2_log2(group_size);
    if (lg >= 5 && lg <= 10 && reinterpret_cast<uintptr_t>(w) % 16 == 0 && (bits != 8 || reinterpret_cast<uintptr_t>(out) % 8 == 0)) {
        const size_t units = n_groups * (group_size / 8);
        const int grid = unit_grid(units);
        cudaError_t e = cudaSuccess;
#define MTC_QZ(B)                                                                                                             \
    e = launch_pdl(dt == MTC_F32 ? affine_quantize8_kernel<B, MTC_F32> : dt == MTC_F16 ? affine_quantize8_kernel<B, MTC_F16>  \
                                                                                       : affine_quantize8_kernel<B, MTC_BF16>, \
                   grid, 256, 0, st, w, oo, scales, biases, units, lg)
        switch (bits) {
            case 2: MTC_QZ(2); break;
            case 3: MTC_QZ(3); break;
            case 4: MTC_QZ(4); break;
            case 5: MTC_QZ(5); break;
            case 6: MTC_QZ(6); break;
            default: MTC_QZ(8); break;
        }
#undef MTC_QZ
        return e;
    }
    const int grid = grid_for(n_groups, 8, ctx->sm_count);
    switch (bits) {
        case 2: affine_quantize_kernel<2><<<grid, 256, 0, st>>>(w, oo, scales, biases, n_groups, group_size, dt); break;
        case 3: affine_quantize_kernel<3><<<grid, 256, 0, st>>>(w, oo, scales, biases, n_groups, group_size, dt); break;
        case 4: affine_quantize_kernel<4><<<grid, 256, 0, st>>>(w, oo, scales, biases, n_groups, group_size, dt); break;
        case 5: affine_quantize_kernel<5><<<grid, 256, 0, st>>>(w, oo, scales, biases, n_groups, group_size, dt); break;
        case 6: affine_quantize_kernel<6><<<grid, 256, 0, st>>>(w, oo, scales, biases, n_groups, group_size, dt); break;
        default: affine_quantize_kernel<8><<<grid, 256, 0, st>>>(w, oo, scales, biases, n_groups, group_size, dt); break;
    }
    return cudaGetLastError();
}

}  // namespace mtc
