// qmv_frag — small-M quantized products of every width on the warp-level tensor cores, weights straight from global memory
// into MMA fragments.
//
//   out[m, n] = sum_k (q(n,k) * scale[n, k/G] + bias[n, k/G]) * x[m, k]      1 <= M <= 16, f32 accumulation
//
// The integer codes are the A operand without a conversion: a 16-bit float whose exponent field is 0 or 1 is linear in its
// low bits (bf16: bits 0-7, value bits * 2^-133; f16: bits 0-10, bits * 2^-24), so a mask (and a shift where the field lies
// higher) leaves two codes in place.  x is the B operand, staged in the matching order as bf16 times 2^64 (a field at bit p
// meets x * 2^-p: exact changes of exponent) or as f16 unchanged (fields shifted down to bit 0); f32 activations are
// staged as three bf16 pieces, which hold all of their 24 significant bits.  Products and sums therefore lose nothing
// before the f32 accumulators, and the power of two leaves once per output.
//
// What bounds it: bytes of weights per SM (22 B a clock at the copy rate) against issue slots.  The split:
//   * a warp owns a tile of 16 weight rows and a contiguous slice of K; the warps of a CTA share a tile K-wise (KS of them)
//     or own different tiles.  A step is 128 codes of each row: quad lane t loads chunk t (32 codes = BITS words) of rows g
//     and g + 8 with the widest loads the width allows.  Everything a run of steps needs is requested one run ahead, in
//     registers: no shared-memory ring, no copy iterator, nothing between a load and its use but the mask.
//   * the four chunks of a step are the k positions of one MMA, so they would have to share a scale.  Instead the idle
//     columns of the B operand separate them (the MMA has 8 columns, M is small): modes
//       S2  chunk t meets columns 2t, 2t+1 only (zero elsewhere): two tokens a tile, any group that is a multiple of 32;
//           lane t then holds exactly the sums of its own chunk and needs only that chunk's scale (S1: one token);
//       S4  chunks 0, 1 meet columns 0-3, chunks 2, 3 columns 4-7: four tokens a tile, groups that are multiples of 64;
//       G   (4- and 8-bit) lane t takes 16 codes of each 64-code half instead of 32 codes of the step: eight tokens a
//           tile, two accumulators a step, groups that are multiples of 64.
//   * every warp stages the activations of its own slice (fragment order, 256 bytes per step and token) and their sums, which
//     a lane adds up from the activations it stages (through MMAs against codes that are all one they were 0.6-1.1 us of a
//     decode launch: 4096 x 4096, M = 1, 4.46 -> 3.79 us; 4096 x 14336 10.7 -> 9.5 us): no CTA barrier before the products.
//   * the KS partial tiles are added in shared memory in warp order, once per launch where they fit: deterministic.
#pragma once

#include "common.cuh"

namespace mtc {

struct FragProj {
    const uint32_t *w;
    const void *scales, *biases;
    void *out;
    int N, tile0;                // rows; first tile of this projection in the launch
};

struct FragArgs {
    FragProj p[4];
    int n_proj, tiles;           // projections that share x; 16-row tiles of all of them
    const void *x;
    int M, K, gs_shift;
    int wpr, gpr;                // words and groups per weight row
    int steps;                   // 128-code steps of a row (the last may be partial)
    int ks, iters;               // warps per tile; tile iterations of every warp slot
    int blk_runs;                // runs whose activations fit the warp's part of shared memory
    int nred;                    // tiles whose partial sums fit the reduction buffer at once
    uint32_t off_sum, off_red, warp_bytes;   // shared memory: sums within a warp's part, partial sums, bytes of a warp's part
    int early;                   // weights may be read before the previous kernel of the stream is complete
};

namespace frag {

constexpr int kMaxWarps = 16;                  // 8 warps a CTA and two CTAs an SM, or 16 warps where there are few tiles
enum { S1 = 0, S2 = 1, S4 = 2, G8 = 3 };

template <int BITS>
constexpr int kRun = BITS <= 4 ? 4 : 2;       // steps requested at once (registers: 2 * BITS words a step)

// 3-bit codes in S1 and S2, where every chunk has its own columns: where rows start on 16 bytes, lane t takes RUN consecutive chunks
// of a run, one a step (else chunk t of every step), so that its words of the run are whole 16-byte loads, 6 a run and two
// rows instead of 24 (8192 x 8192, groups of 32, 4 tokens 18.3 -> 16.9 us, groups of 64, one token 14.7 -> 12.5).  Not for 6 bits,
// whose 8-byte loads are enough (18.7 -> 19.4), nor 5, whose runs of two are 40 bytes a lane.
template <int BITS, int MODE>
constexpr bool kLong = BITS == 3 && (MODE == S1 || MODE == S2);

template <int MODE>
constexpr int kCap = MODE == S1 ? 1 : MODE == S2 ? 2 : MODE == S4 ? 4 : 8;      // tokens of one tile of columns

template <int XT>
constexpr int kPieces = XT == MTC_F32 ? 3 : 1;

// ---- fields: register r (0..15) of a 32-code chunk holds codes lo(r) and hi(r) at bit pos(r) of its halves -----------
template <int BITS>
__host__ __device__ constexpr int code_lo(int r) {
    return BITS == 4 ? 8 * (r >> 2) + (r & 3) : BITS == 8 ? 4 * (r >> 1) + (r & 1) : BITS == 2 ? 16 * (r >> 3) + (r & 7) : r;
}
template <int BITS>
__host__ __device__ constexpr int code_hi(int r) {
    return code_lo<BITS>(r) + (BITS == 4 ? 4 : BITS == 8 ? 2 : BITS == 2 ? 8 : 16);
}
// bit of the 16-bit stream half at which the field of register r starts
template <int BITS>
__host__ __device__ constexpr int field_bit(int r) {
    return BITS == 4 ? 4 * (r & 3) : BITS == 8 ? 8 * (r & 1) : BITS == 2 ? 2 * (r & 7) : (BITS * r) % 16;
}
// how far the field is shifted down: bf16 fields may stay anywhere in bits 0-7 (one shift by 8 serves several), f16 fields
// go to bit 0, because x / 2^p could fall below the f16 range
template <int BITS, bool BF>
__host__ __device__ constexpr int field_shift(int r) {
    const int b = field_bit<BITS>(r);
    if (b + BITS > 16) return b;                              // straddles two halves: joined at bit 0
    if (!BF) return b;
    if (b + BITS <= 8) return 0;
    return b >= 8 ? 8 : b;
}
template <int BITS, bool BF>
__host__ __device__ constexpr int field_pos(int r) { return field_bit<BITS>(r) - field_shift<BITS, BF>(r); }

// planar form of the widths whose codes straddle words: half j of stream 0 (codes 0-15) and of stream 1 (codes 16-31)
template <int BITS>
struct Planes {
    static constexpr bool kPlanar = BITS == 3 || BITS == 5 || BITS == 6;
    uint32_t v[BITS];
    __device__ __forceinline__ explicit Planes(const uint32_t (&w)[BITS]) {
#pragma unroll
        for (int j = 0; j < BITS; ++j) {
            if (kPlanar) v[j] = __byte_perm(w[j / 2], w[(j + BITS) / 2], ((j & 1) ? 0x32 : 0x10) | (((j + BITS) & 1) ? 0x7600 : 0x5400));
            else v[j] = w[j];
        }
    }
};

template <int BITS, bool BF>
__device__ __forceinline__ uint32_t field(const Planes<BITS> &p, int r) {      // r is a constant where this is inlined
    constexpr uint32_t one = (1u << BITS) - 1u;
    const int b = field_bit<BITS>(r), s = field_shift<BITS, BF>(r);
    const int j = BITS == 4 ? r >> 2 : BITS == 8 ? r >> 1 : BITS == 2 ? r >> 3 : (BITS * r) / 16;
    if (b + BITS > 16) {
        const int n = 16 - b;                                 // bits of the code in this half
        const uint32_t lo = ((1u << n) - 1u) * 0x10001u, hi = (one ^ ((1u << n) - 1u)) * 0x10001u;
        return ((p.v[j] >> b) & lo) | ((p.v[j + 1] << n) & hi);
    }
    return (p.v[j] >> s) & ((one << (b - s)) * 0x10001u);
}

// ---- instructions -------------------------------------------------------------------------------------------------
template <bool BF>
__device__ __forceinline__ void mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1, bool first) {
    if (first) {
        if (BF)
            asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
                : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.0f));
        else
            asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
                : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.0f));
    } else {
        if (BF)
            asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
        else
            asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
    }
}

// Predicated loads: a lane outside the row (or a warp with nothing left to request) keeps what the registers hold - any
// bits are finite codes, and the activations there are zero.
__device__ __forceinline__ void ldg16(const void *p, uint32_t *v, bool on) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %5, 0;\n\t@p ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];\n\t}"
                 : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]) : "l"(p), "r"(static_cast<uint32_t>(on)));
}
__device__ __forceinline__ void ldg8(const void *p, uint32_t *v, bool on) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %3, 0;\n\t@p ld.global.nc.v2.u32 {%0,%1}, [%2];\n\t}"
                 : "+r"(v[0]), "+r"(v[1]) : "l"(p), "r"(static_cast<uint32_t>(on)));
}
__device__ __forceinline__ void ldg4(const void *p, uint32_t *v, bool on) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\t@p ld.global.nc.u32 %0, [%1];\n\t}"
                 : "+r"(v[0]) : "l"(p), "r"(static_cast<uint32_t>(on)));
}
// Scales and biases: zero outside the row.  What the run before left there need not be finite, and inf * 0 is not 0.
__device__ __forceinline__ void ldg4_or_zero(const void *p, uint32_t *v, bool on) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\tmov.u32 %0, 0;\n\t@p ld.global.nc.u32 %0, [%1];\n\t}"
                 : "=&r"(v[0]) : "l"(p), "r"(static_cast<uint32_t>(on)));
}
__device__ __forceinline__ void ldg2_or_zero(const void *p, uint32_t *v, bool on) {
    asm volatile("{\n\t.reg .pred p;\n\t.reg .u16 h;\n\tsetp.ne.b32 p, %2, 0;\n\tmov.u16 h, 0;\n\t@p ld.global.nc.u16 h, [%1];\n\tcvt.u32.u16 %0, h;\n\t}"
                 : "=r"(v[0]) : "l"(p), "r"(static_cast<uint32_t>(on)));
}

// ... and the plain ones, where the whole run lies inside the row
__device__ __forceinline__ void ldg16(const void *p, uint32_t *v) {
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "l"(p));
}
// 16 bytes whose sectors are shared with the lane's next load: kept in L1
__device__ __forceinline__ void ldg16_l1(const void *p, uint32_t *v) {
    asm volatile("ld.global.nc.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "l"(p));
}
__device__ __forceinline__ void ldg8(const void *p, uint32_t *v) {
    asm volatile("ld.global.nc.v2.u32 {%0,%1}, [%2];" : "=r"(v[0]), "=r"(v[1]) : "l"(p));
}
__device__ __forceinline__ void ldg4(const void *p, uint32_t *v) { asm volatile("ld.global.nc.u32 %0, [%1];" : "=r"(v[0]) : "l"(p)); }
__device__ __forceinline__ void ldg2(const void *p, uint32_t *v) {
    unsigned short h;
    asm volatile("ld.global.nc.u16 %0, [%1];" : "=h"(h) : "l"(p));
    v[0] = h;
}
template <int BITS, int MODE>
__device__ __forceinline__ void load_words(const char *p, uint32_t (&w)[BITS]) {
    if constexpr (MODE == G8 && BITS == 4) {
        ldg8(p, w);
        ldg8(p + 32, w + 2);
    } else if constexpr (MODE == G8) {
        ldg16(p, w);
        ldg16(p + 64, w + 4);
    } else if constexpr (BITS % 4 == 0) {
#pragma unroll
        for (int i = 0; i < BITS; i += 4) ldg16(p + 4 * i, w + i);
    } else if constexpr (BITS % 2 == 0) {
#pragma unroll
        for (int i = 0; i < BITS; i += 2) ldg8(p + 4 * i, w + i);
    } else {
#pragma unroll
        for (int i = 0; i < BITS; ++i) ldg4(p + 4 * i, w + i);
    }
}

// One row's packed words of one step for this lane.  p: the lane's words of the step in the row (S modes: chunk t; G8: its 16
// codes of the first half, the second half is HALF bytes further on); on0, on1: whether they lie inside the row.
template <int BITS, int MODE>
__device__ __forceinline__ void load_words(const char *p, uint32_t (&w)[BITS], bool on0, bool on1) {
    if constexpr (MODE == G8 && BITS == 4) {
        ldg8(p, w, on0);
        ldg8(p + 32, w + 2, on1);
    } else if constexpr (MODE == G8) {
        ldg16(p, w, on0);
        ldg16(p + 64, w + 4, on1);
    } else if constexpr (BITS % 4 == 0) {
#pragma unroll
        for (int i = 0; i < BITS; i += 4) ldg16(p + 4 * i, w + i, on0);
    } else if constexpr (BITS % 2 == 0) {
#pragma unroll
        for (int i = 0; i < BITS; i += 2) ldg8(p + 4 * i, w + i, on0);
    } else {
#pragma unroll
        for (int i = 0; i < BITS; ++i) ldg4(p + 4 * i, w + i, on0);
    }
}

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}
template <int XT>
__device__ __forceinline__ float scale_f32(uint32_t raw) {
    if (XT == MTC_F32) return __uint_as_float(raw);
    if (XT == MTC_BF16) return __uint_as_float(raw << 16);
    return __half2float(__ushort_as_half(static_cast<unsigned short>(raw)));
}
template <int XT>
__device__ __forceinline__ void ld_scale(const char *p, uint32_t *v, bool on) {
    if (XT == MTC_F32) ldg4_or_zero(p, v, on);
    else ldg2_or_zero(p, v, on);
}
template <int XT>
__device__ __forceinline__ void ld_scale(const char *p, uint32_t *v) {
    if (XT == MTC_F32) ldg4(p, v);
    else ldg2(p, v);
}

// The 32 activations of (step, token, quad lane t) as 16 B registers per piece: block (s*Mp + m)*4 + t of kPitch bytes (Mp = columns for tokens), 64
// bytes a piece.  The 16 bytes of padding put the eight blocks that a load phase reads (two tokens, four t) on eight different
// 16-byte columns of the banks.
template <int XT>
constexpr int kPitch = 64 * kPieces<XT> + 16;

// Returns the sum of the 32 activations (not for G8, whose two halves have sums of their own).
template <int BITS, int XT, int MODE, int UP = 64, typename A>              // bf16: x times 2^UP; A: x, K, M of the rows
__device__ __forceinline__ float stage_chunk(const A &a, int m, int k_lo, int k_hi, char *dst) {
    // k_lo: first activation of registers 0-7, k_hi: of registers 8-15 (16 values each; both inside or outside the row)
    constexpr bool BF = XT != MTC_F16;
    if constexpr (XT == MTC_F32) {
        float v[32];
        const float *x = static_cast<const float *>(a.x) + static_cast<size_t>(m) * a.K;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int k = (q < 4 ? k_lo : k_hi - 16) + 4 * q;
            const float4 f = k < a.K && m < a.M ? *reinterpret_cast<const float4 *>(x + k) : make_float4(0.f, 0.f, 0.f, 0.f);
            v[4 * q] = f.x; v[4 * q + 1] = f.y; v[4 * q + 2] = f.z; v[4 * q + 3] = f.w;
        }
        float sum[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        if (MODE != G8) {
#pragma unroll
            for (int q = 0; q < 32; ++q) sum[q & 3] += v[q];
        }
        uint32_t o[3][4];
#pragma unroll
        for (int r = 0; r < 16; ++r) {
            const float sc = __uint_as_float(static_cast<uint32_t>(127 + UP - field_pos<BITS, true>(r)) << 23);
            float lo = v[code_lo<BITS>(r)] * sc, hi = v[code_hi<BITS>(r)] * sc;
#pragma unroll
            for (int p = 0; p < 3; ++p) {
                const uint32_t b = pack_bf16(lo, hi);
                o[p][r & 3] = b;
                lo -= __uint_as_float(b << 16);
                hi -= __uint_as_float(b & 0xFFFF0000u);
                if (p == 0) {             // an infinity or a NaN is all in the first piece: inf - inf would make the others NaN
                    if ((b & 0x7F80u) == 0x7F80u) lo = 0.0f;
                    if ((b & 0x7F800000u) == 0x7F800000u) hi = 0.0f;
                }
            }
            if ((r & 3) == 3) {
#pragma unroll
                for (int p = 0; p < 3; ++p)
                    *reinterpret_cast<uint4 *>(dst + p * 64 + ((r >> 2) << 4)) = make_uint4(o[p][0], o[p][1], o[p][2], o[p][3]);
            }
        }
        return (sum[0] + sum[1]) + (sum[2] + sum[3]);
    } else {
        uint32_t u[16];
        const uint16_t *x = static_cast<const uint16_t *>(a.x) + static_cast<size_t>(m) * a.K;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int k = (q < 2 ? k_lo : k_hi - 16) + 8 * q;
            const uint4 f = k < a.K && m < a.M ? *reinterpret_cast<const uint4 *>(x + k) : make_uint4(0u, 0u, 0u, 0u);
            u[4 * q] = f.x; u[4 * q + 1] = f.y; u[4 * q + 2] = f.z; u[4 * q + 3] = f.w;
        }
        float sum[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        if (MODE != G8) {
#pragma unroll
            for (int q = 0; q < 16; ++q) {
                const float2 f = BF ? make_float2(__uint_as_float(u[q] << 16), __uint_as_float(u[q] & 0xFFFF0000u))
                                    : __half22float2(*reinterpret_cast<const __half2 *>(&u[q]));
                sum[2 * (q & 1)] += f.x;
                sum[2 * (q & 1) + 1] += f.y;
            }
        }
        uint32_t o[4];
#pragma unroll
        for (int r = 0; r < 16; ++r) {
            const int lo = code_lo<BITS>(r), hi = code_hi<BITS>(r);
            uint32_t b = __byte_perm(u[lo >> 1], u[hi >> 1], ((lo & 1) ? 0x32 : 0x10) | ((hi & 1) ? 0x7600 : 0x5400));
            if (BF) {                     // times 2^(UP - pos): exact, subnormals included (inf beyond 2^(127 - UP))
                const uint32_t e = static_cast<uint32_t>(127 + UP - field_pos<BITS, true>(r)) << 7;
                asm("mul.rn.bf16x2 %0, %0, %1;" : "+r"(b) : "r"(e * 0x10001u));
            }
            o[r & 3] = b;
            if ((r & 3) == 3) *reinterpret_cast<uint4 *>(dst + ((r >> 2) << 4)) = make_uint4(o[0], o[1], o[2], o[3]);
        }
        return (sum[0] + sum[1]) + (sum[2] + sum[3]);
    }
}

// B registers of a lane.  Lanes whose column belongs to another chunk never load, so theirs stay zero; tokens past M are
// staged as zeros.  Four rotating sets keep the loads ahead of the products.
struct BRegs {
    uint32_t v[4][4] = {};
};

// One step: registers of rows g (wl) and g + 8 (wh) against the fragments; at: shared address of the step's block of the lane's
// first token and t, on: the lane's column takes part.  G8: d[nt][0], d[nt][1] are the two halves.
template <int BITS, int XT, int MODE, int NT, bool ONES>
__device__ __forceinline__ void step_mma(const uint32_t (&wl)[BITS], const uint32_t (&wh)[BITS], uint32_t at, bool on, BRegs &br,
                                         float (&d)[NT][MODE == G8 ? 2 : 1][4]) {
    constexpr bool BF = XT != MTC_F16;
    constexpr int P = kPieces<XT>;
    // Chains of dependent MMAs.  16-bit activations and one tile of columns: two, for latency.  f32: the leading pieces in two
    // chains and the two lower pieces, 2^-8 and 2^-16 of them, in a third: the tensor core cuts its sums off instead of
    // rounding them, and three short chains of which one is small stay at the error of an FFMA chain (4e-7 against
    // 1-2e-6 in one chain of 24).
    constexpr bool kTwo = NT * P == 1;
    float e[P == 3 ? NT : 1][4], f[P == 3 ? NT : 1][4];
    const Planes<BITS> pl(wl), ph(wh);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        uint32_t al[4], ah[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int r = 4 * q + i;
            if (ONES) {                   // codes that are all one: sums of the activations
                al[i] = ah[i] = 0x10001u << field_pos<BITS, BF>(r);
            } else {
                al[i] = field<BITS, BF>(pl, r);
                ah[i] = field<BITS, BF>(ph, r);
            }
        }
        const int h = MODE == G8 ? q >> 1 : 0;
        const bool first = MODE == G8 ? (q & 1) == 0 : q == 0;
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int p = 0; p < P; ++p) {
                uint32_t (&b)[4] = br.v[(q * NT * P + nt * P + p) & 3];
                asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %5, 0;\n\t@p ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];\n\t}"
                             : "+r"(b[0]), "+r"(b[1]), "+r"(b[2]), "+r"(b[3])
                             : "r"(at + nt * (kCap<MODE> * 4 * kPitch<XT>) + p * 64 + q * 16), "r"(static_cast<uint32_t>(on)));
                if (P == 3 && p > 0) {
                    mma<BF>(f[nt], al[0], ah[0], al[1], ah[1], b[0], b[1], first && p == 1);
                    mma<BF>(f[nt], al[2], ah[2], al[3], ah[3], b[2], b[3], false);
                } else {
                    mma<BF>(d[nt][h], al[0], ah[0], al[1], ah[1], b[0], b[1], first);
                    mma<BF>(P == 3 ? e[nt] : kTwo ? e[0] : d[nt][h], al[2], ah[2], al[3], ah[3], b[2], b[3], (P == 3 || kTwo) && first);
                }
            }
        if (q == 3 || (MODE == G8 && q == 1)) {
#pragma unroll
            for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    if (P == 3) d[nt][h][j] = (d[nt][h][j] + e[nt][j]) + f[nt][j];
                    else if (kTwo) d[nt][h][j] += e[0][j];
                }
        }
    }
}

// ---- scales (or biases) of a run: rows g and g + 8 -----------------------------------------------------------------------
// VEC 6, 7 (log2 of the group; 16-bit types, whole runs of 512 codes, 16-byte aligned rows of scales): the eight (four) groups
// of a run are one load per row.  VEC 0: one element per row, step (and half).
template <int XT, int MODE, int RUN, int VEC>
struct Affine {
    static constexpr int H = MODE == G8 ? 2 : 1;
    static constexpr int W = VEC ? (VEC == 6 ? 4 : 2) : RUN * H;
    uint32_t r[2][W];

    // i: step of the run, h: half (G8), row: 0 = g, 1 = g + 8
    __device__ __forceinline__ float get(int i, int h, int row, int t) const {
        if constexpr (VEC == 0) {
            return scale_f32<XT>(r[row][i * H + h]);
        } else {
            const uint32_t w = VEC == 6 ? r[row][i] : r[row][i >> 1];
            if constexpr (XT == MTC_BF16) {
                if (VEC == 7) return __uint_as_float((i & 1) ? (w & 0xFFFF0000u) : (w << 16));
                if (MODE == G8) return __uint_as_float(h ? (w & 0xFFFF0000u) : (w << 16));
                return __uint_as_float(__byte_perm(w, 0u, t & 2 ? 0x3244 : 0x1044));
            } else {
                const bool hi = VEC == 7 ? (i & 1) != 0 : (MODE == G8 ? h != 0 : (t & 2) != 0);
                return __half2float(__ushort_as_half(static_cast<unsigned short>(hi ? w >> 16 : w & 0xFFFFu)));
            }
        }
    }
};

// ---- kernel ----------------------------------------------------------------------------------------------------------
template <int BITS, int XT, int MODE, int NT, int VEC>
__global__ void __launch_bounds__(32 * kMaxWarps, 1) qmv_frag_kernel(const __grid_constant__ FragArgs a) {
    constexpr int RUN = (MODE == G8 && !VEC) ? 2 : kRun<BITS>;
    constexpr int H = MODE == G8 ? 2 : 1;
    constexpr int CAP = kCap<MODE>, MP = CAP * NT;
    const bool lng = kLong<BITS, MODE> && a.wpr % 4 == 0;
    constexpr uint32_t STEP = MP * 4 * kPitch<XT>;                                 // fragments of one step
    constexpr uint32_t SUM = NT * H * 4 * (MODE == S1 ? 4 : 8);                    // activation sums of one step
    constexpr int ESZ = XT == MTC_F32 ? 4 : 2;
    extern __shared__ __align__(128) char smem[];
    const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0), lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int nwarps = blockDim.x >> 5, slots = nwarps / a.ks, slot = warp / a.ks, slice = warp - slot * a.ks;
    const int total_runs = (a.steps + RUN - 1) / RUN;
    const int r0 = slice * total_runs / a.ks, r1 = (slice + 1) * total_runs / a.ks;
    char *part = smem + warp * a.warp_bytes;
    float *red = reinterpret_cast<float *>(smem + a.off_red);
    const bool on = MODE == S1 ? g == 2 * t : MODE == S2 ? (g >> 1) == t : MODE == S4 ? (g >> 2) == (t >> 1) : true;
    if (!a.early) asm volatile("griddepcontrol.wait;" ::: "memory");

    // ---- requests: one run of steps in registers, one run ahead of the products ----
    uint32_t wl[RUN][BITS], wh[RUN][BITS];
    Affine<XT, MODE, RUN, VEC> sc, bi, sc_next;
#pragma unroll
    for (int i = 0; i < RUN; ++i)
#pragma unroll
        for (int j = 0; j < BITS; ++j) wl[i][j] = wh[i][j] = 0u;
#pragma unroll
    for (int j = 0; j < sc.W; ++j) sc.r[0][j] = sc.r[1][j] = bi.r[0][j] = bi.r[1][j] = 0u;
    const char *wbase = nullptr, *sbase = nullptr, *bbase = nullptr;               // of the projection of the tile being requested
    uint32_t wo[2] = {0u, 0u}, ao[2] = {0u, 0u};                                   // byte offsets of rows g, g + 8: words (with the lane's), scales
    int l_it = 0, l_run = r0, l_tile = blockIdx.x * slots + slot;
    auto open_tile = [&]() {
        int pi = 0;
#pragma unroll
        for (int i = 1; i < 4; ++i)
            if (i < a.n_proj && l_tile >= a.p[i].tile0) pi = i;
        const FragProj &pr = a.p[pi];
        wbase = reinterpret_cast<const char *>(pr.w);
        sbase = static_cast<const char *>(pr.scales);
        bbase = static_cast<const char *>(pr.biases);
        const int n = (l_tile - pr.tile0) * 16 + g;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const uint32_t row = min(n + 8 * j, pr.N - 1);
            wo[j] = row * static_cast<uint32_t>(a.wpr * 4) + (MODE == G8 ? t * (BITS * 2) : t * (BITS * 4) * (lng ? RUN : 1));
            ao[j] = row * static_cast<uint32_t>(a.gpr * ESZ);
        }
    };
    const int n_units = MODE == G8 ? a.K >> 6 : a.K >> 5;                          // halves (G8) or chunks of a row
    const char *pl = nullptr, *ph = nullptr, *ps[2] = {nullptr, nullptr}, *pb[2] = {nullptr, nullptr};    // of the run being requested
    bool whole = true;                        // the run being requested lies inside the row (VEC: all do)
    auto request_words = [&](int i, int limit) {
        if (limit == 0) return;               // nothing left for this warp (uniform)
        if (lng && whole) {
            if constexpr (kLong<BITS, MODE>) {
                static_assert((RUN * BITS) % 4 == 0, "whole 16-byte loads");
                // a load goes out with the last step whose words it replaces
#pragma unroll
                for (int v = 0; v < RUN * BITS / 4; ++v)
                    if ((4 * v + 3) / BITS == i) {
                        ldg16_l1(pl + 16 * v, &wl[0][0] + 4 * v);
                        ldg16_l1(ph + 16 * v, &wh[0][0] + 4 * v);
                    }
            }
        } else if (VEC != 0 || whole) {
            load_words<BITS, MODE>(pl + i * (16 * BITS), wl[i]);
            load_words<BITS, MODE>(ph + i * (16 * BITS), wh[i]);
        } else {
            const int s = l_run * RUN + i;
            const bool on0 = (MODE == G8 ? 2 * s : lng ? (4 * l_run + t) * RUN + i : 4 * s + t) < limit, on1 = 2 * s + 1 < limit;
            const int step_w = lng ? 4 * BITS : 16 * BITS;                         // bytes from a lane's words of a step to those of the next
            load_words<BITS, MODE>(pl + i * step_w, wl[i], on0, on1);
            load_words<BITS, MODE>(ph + i * step_w, wh[i], on0, on1);
        }
    };
    auto request_affine = [&](const char *const (&p)[2], Affine<XT, MODE, RUN, VEC> &f, int i, int limit) {   // VEC: the whole run, i unused
        if (limit == 0) return;
        if constexpr (VEC != 0) {
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                if constexpr (VEC == 6) ldg16(p[j], f.r[j]);
                else ldg8(p[j], f.r[j]);
            }
        } else {
#pragma unroll
            for (int h = 0; h < H; ++h) {
                const int s = l_run * RUN + i;
                const int k = MODE == G8 ? 128 * s + 64 * h : MODE == S4 ? 128 * s + 64 * (t >> 1) : lng ? ((4 * l_run + t) * RUN + i) * 32 : 128 * s + 32 * t;
                const uint32_t off = static_cast<uint32_t>(k >> a.gs_shift) * ESZ;
                if (whole) {
#pragma unroll
                    for (int j = 0; j < 2; ++j) ld_scale<XT>(p[j] + off, &f.r[j][i * H + h]);
                } else {
                    const bool in = (MODE == G8 ? 2 * s + h : MODE == S4 ? 4 * s + 2 * (t >> 1) : lng ? (4 * l_run + t) * RUN + i : 4 * s + t) < limit;
#pragma unroll
                    for (int j = 0; j < 2; ++j) ld_scale<XT>(p[j] + off, &f.r[j][i * H + h], in);
                }
            }
        }
    };
    auto open_run = [&]() {
        const uint32_t run_w = static_cast<uint32_t>(l_run) * (RUN * 16 * BITS);
        const uint32_t run_a = VEC ? static_cast<uint32_t>(l_run) * (VEC == 6 ? 16 : 8) : 0u;
        whole = (l_run + 1) * (RUN * 128) <= a.K;
        pl = wbase + (wo[0] + run_w);
        ph = wbase + (wo[1] + run_w);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            ps[j] = sbase + (ao[j] + run_a);
            pb[j] = bbase + (ao[j] + run_a);
        }
    };
    // to the next run of this warp; returns its row limit, 0: there is none
    auto advance = [&]() -> int {
        if (++l_run == r1) {
            l_run = r0;
            l_tile += gridDim.x * slots;
            if (++l_it >= a.iters || l_tile >= a.tiles) return 0;
            open_tile();
        }
        open_run();
        return n_units;
    };
    int limit = r0 < r1 && l_tile < a.tiles ? n_units : 0;
    if (limit) {
        open_tile();
        open_run();
#pragma unroll
        for (int i = 0; i < RUN; ++i) request_words(i, limit);
#pragma unroll
        for (int i = 0; i < (VEC ? 1 : RUN); ++i) {
            request_affine(ps, sc, i, limit);
            request_affine(pb, bi, i, limit);
        }
    }
    asm volatile("griddepcontrol.launch_dependents;");
    if (a.early) asm volatile("griddepcontrol.wait;" ::: "memory");

    // ---- activations of runs [from, to) of this warp's slice ----
    BRegs br;
    const int tok0 = MODE == S1 ? 0 : MODE == S2 ? g & 1 : MODE == S4 ? g & 3 : g;   // this lane's token in a tile of columns
    const uint32_t frag0 = static_cast<uint32_t>(__cvta_generic_to_shared(part)) + static_cast<uint32_t>((tok0 * 4 + t) * kPitch<XT>);
    char *sums = part + a.off_sum;
    auto stage = [&](int from, int to) {
        __syncwarp();
        const int n = (to - from) * RUN * 4 * MP;
        for (int e0 = 0; e0 < n; e0 += 32) {
            const int e = e0 + lane, et = e & 3, em = (e >> 2) % MP, es = (e >> 2) / MP;
            const int k = lng ? ((from + es / RUN) * 4 * RUN + es % RUN) * 32 + et * (32 * RUN - 32) : (from * RUN + es) * 128;
            float sum = 0.0f;
            if (e < n)
                sum = stage_chunk<BITS, XT, MODE>(a, em, MODE == G8 ? k + 16 * et : k + 32 * et, MODE == G8 ? k + 64 + 16 * et : k + 32 * et + 16,
                                                  part + static_cast<size_t>(e) * kPitch<XT>);
            if (MODE != G8) {
                // in the units of the products: x times 2^64 against codes times 2^-133, f16: codes times 2^-24
                constexpr uint32_t unit = (XT == MTC_F16 ? 127u - 24u : 127u - 69u) << 23;
                if (MODE == S4) sum += __shfl_xor_sync(0xffffffffu, sum, 1);             // chunks 0 and 1, 2 and 3
                // as the products leave the MMA: chunk t (S4: pair t >> 1) and token at the columns they meet
                const uint32_t at = MODE == S1 ? et * 4 : (em / CAP) * 32 + (MODE == S2 ? et * 8 : (et >> 1) * 16) + (em % CAP) * 4;
                if (e < n && (MODE != S4 || !(et & 1))) *reinterpret_cast<float *>(sums + es * SUM + at) = sum * __uint_as_float(unit);
            }
        }
        __syncwarp();
        // G8 adds over the quad and keeps its halves apart: the same MMAs against codes that are all one
#pragma unroll 2
        for (int s = 0; s < (MODE == G8 ? (to - from) * RUN : 0); ++s) {
            const uint32_t none[BITS] = {};
            float d[NT][H][4];
            step_mma<BITS, XT, MODE, NT, true>(none, none, frag0 + s * STEP, on, br, d);
            if (lane < 4) {
#pragma unroll
                for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                    for (int h = 0; h < H; ++h) {
                        char *q = sums + s * SUM + (nt * H + h) * 32;
                        reinterpret_cast<float2 *>(q)[t] = make_float2(d[nt][h][0], d[nt][h][1]);
                    }
            }
        }
        __syncwarp();
    };
    const bool resident = r1 - r0 <= a.blk_runs;
    if (resident && r0 < r1) stage(r0, r1);

    // ---- tiles ----
    const float post = XT == MTC_F16 ? __uint_as_float((127u + 24u) << 23) : __uint_as_float((127u + 69u) << 23);
    int tile = blockIdx.x * slots + slot, buf = 0;
    for (int it = 0; it < a.iters; ++it, tile += gridDim.x * slots) {
        if (tile < a.tiles) {
            float acc[NT][4];
#pragma unroll
            for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[nt][j] = 0.0f;
            int blk0 = r0;
            for (int run = r0; run < r1; ++run) {
                if (!resident && (run == r0 || run - blk0 == a.blk_runs)) {
                    blk0 = run;
                    stage(run, min(run + a.blk_runs, r1));
                }
                limit = limit ? advance() : 0;
                const uint32_t at = frag0 + (run - blk0) * (RUN * STEP);
                const char *sat = sums + (run - blk0) * (RUN * SUM) + t * (MODE == S1 ? 4 : 8);
                // the bias term of the run first: its registers are free for the next run's biases at once
#pragma unroll
                for (int i = 0; i < RUN; ++i)
#pragma unroll
                    for (int h = 0; h < H; ++h) {
                        const float b_l = bi.get(i, h, 0, t), b_h = bi.get(i, h, 1, t);
#pragma unroll
                        for (int nt = 0; nt < NT; ++nt) {
                            const char *q = sat + i * SUM + (nt * H + h) * (MODE == S1 ? 16 : 32);
                            if (MODE == S1) {
                                const float xs = *reinterpret_cast<const float *>(q);
                                acc[nt][0] = fmaf(b_l, xs, acc[nt][0]);
                                acc[nt][2] = fmaf(b_h, xs, acc[nt][2]);
                            } else {
                                const float2 xs = *reinterpret_cast<const float2 *>(q);
                                acc[nt][0] = fmaf(b_l, xs.x, acc[nt][0]);
                                acc[nt][1] = fmaf(b_l, xs.y, acc[nt][1]);
                                acc[nt][2] = fmaf(b_h, xs.x, acc[nt][2]);
                                acc[nt][3] = fmaf(b_h, xs.y, acc[nt][3]);
                            }
                        }
                    }
#pragma unroll
                for (int i = 0; i < (VEC ? 1 : RUN); ++i) request_affine(pb, bi, i, limit);
                if constexpr (VEC != 0) request_affine(ps, sc_next, 0, limit);
#pragma unroll
                for (int i = 0; i < RUN; ++i) {
                    float d[NT][H][4];
                    step_mma<BITS, XT, MODE, NT, false>(wl[i], wh[i], at + i * STEP, on, br, d);
                    request_words(i, limit);
#pragma unroll
                    for (int h = 0; h < H; ++h) {
                        const float s_l = sc.get(i, h, 0, t), s_h = sc.get(i, h, 1, t);
#pragma unroll
                        for (int nt = 0; nt < NT; ++nt) {
                            acc[nt][0] = fmaf(s_l, d[nt][h][0], acc[nt][0]);
                            acc[nt][2] = fmaf(s_h, d[nt][h][2], acc[nt][2]);
                            if (MODE != S1) {
                                acc[nt][1] = fmaf(s_l, d[nt][h][1], acc[nt][1]);
                                acc[nt][3] = fmaf(s_h, d[nt][h][3], acc[nt][3]);
                            }
                        }
                    }
                    if constexpr (VEC == 0) request_affine(ps, sc, i, limit);
                }
                if constexpr (VEC != 0) sc = sc_next;
            }
            // this warp's partial tile: [token][16 rows]
            float *mine = red + (buf * nwarps + warp) * (MP * 16);
#pragma unroll
            for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    if (MODE == S1 && (j & 1)) continue;
                    float v = acc[nt][j];
                    if (MODE == S1 || MODE == S2) v += __shfl_xor_sync(0xffffffffu, v, 1);
                    if (MODE != G8) v += __shfl_xor_sync(0xffffffffu, v, 2);
                    const bool holds = MODE == G8 ? true : MODE == S4 ? t < 2 : t == 0;
                    const int tok = nt * CAP + (MODE == G8 || MODE == S4 ? 2 * t : 0) + (j & 1);
                    if (holds) mine[tok * 16 + g + (j >> 1) * 8] = v;
                }
        }
        // After nred rounds (usually all of them): the sum over the warps of a tile in warp order, and the stores.  No flag or
        // fence per tile: a fence would also wait for the requests in flight.
        if (++buf == a.nred || it + 1 == a.iters) {
            __syncthreads();
            const int round0 = it + 1 - buf, n = buf * slots * MP * 16;
            for (int e = threadIdx.x; e < n; e += blockDim.x) {
                const int row = e & 15, tok = (e >> 4) % MP, ts = (e >> 4) / MP, rs = ts / slots, sl = ts - rs * slots;
                const int tl = ((round0 + rs) * static_cast<int>(gridDim.x) + static_cast<int>(blockIdx.x)) * slots + sl;
                if (tl >= a.tiles || tok >= a.M) continue;
                const float *base = red + (rs * nwarps + sl * a.ks) * (MP * 16) + tok * 16 + row;
                float v = base[0];
                for (int q = 1; q < a.ks; ++q) v += base[q * (MP * 16)];
                int pi = 0;
#pragma unroll
                for (int i = 1; i < 4; ++i)
                    if (i < a.n_proj && tl >= a.p[i].tile0) pi = i;
                const FragProj &pr = a.p[pi];
                const int nn = (tl - pr.tile0) * 16 + row;
                if (nn < pr.N) st_from_f32(pr.out, static_cast<size_t>(tok) * pr.N + nn, v * post, XT);
            }
            if (it + 1 < a.iters) __syncthreads();
            buf = 0;
        }
    }
}

// ---- host side -----------------------------------------------------------------------------------------------------
struct Shape {
    int mode, nt, vec, xt;
};

template <int BITS, int XT, int MODE, int NT, int VEC>
cudaError_t launch_one(cudaStream_t st, FragArgs a, int sms) {
    constexpr int RUN = (MODE == G8 && !VEC) ? 2 : kRun<BITS>;
    constexpr int P = kPieces<XT>;
    constexpr size_t kSmemMax = 226 * 1024, kSmemTwo = 112 * 1024;
    constexpr size_t kFrags = static_cast<size_t>(kCap<MODE>) * NT * 4 * kPitch<XT>, kSums = NT * (MODE == G8 ? 2 : 1) * 4 * (MODE == S1 ? 4 : 8);
    constexpr size_t step_bytes = kFrags + kSums;
    // one run of activations for each of eight warps fits whatever the shape: there is always a plan
    static_assert(RUN * step_bytes <= (kSmemMax - 8 * kCap<MODE> * NT * 64) / 8 / 128 * 128, "a run of activations fits a warp's part");
    const int total_runs = (a.steps + RUN - 1) / RUN;
    // Split of a CTA's eight warps: KS of them share a tile.  Cost of a split = tile rounds x (runs of a slice + the sum over
    // the warps, worth about half a run), plus the activations a warp stages: once when they fit, else with every tile.
    double best = 1e30;
    int best_grid = 0;
    size_t best_smem = 0;
    FragArgs pick = a;
    int best_warps = 8;
    for (int form = 0; form < 3; ++form) {                     // 8 warps and two CTAs an SM, 16 warps, 8 warps and one CTA
        const int nw = form == 1 ? 16 : 8, per_sm = form == 0 ? 2 : 1;
        for (int ks = nw; ks >= 1; ks >>= 1) {
            const int slots = nw / ks;
            const int want = (a.tiles + slots - 1) / slots;
            const int grid = want < sms * per_sm ? want : sms * per_sm;
            const int iters = (a.tiles + grid * slots - 1) / (grid * slots);
            const int runs = (total_runs + ks - 1) / ks;
            const size_t tile_red = static_cast<size_t>(nw) * kCap<MODE> * NT * 64;              // partial sums of one round
            int nred = static_cast<int>(24 * 1024 / tile_red);
            nred = nred < 1 ? 1 : nred > iters ? iters : nred;
            const size_t red = nred * tile_red;
            const size_t limit = per_sm == 2 ? kSmemTwo : kSmemMax;
            if (red >= limit) continue;
            int blk = static_cast<int>((limit - red) / nw / 128 * 128 / (RUN * step_bytes));
            if (blk < 1) continue;
            if (blk > runs) blk = runs;
            const bool resident = blk >= runs;
            // issue slots of the busiest SM, in steps: a step ~65 instructions, the sum over the warps ~60 a warp, staging
            // ~45 (f32: 260) per 32-code chunk over 32 lanes and the MMAs of the sums
            const int on_sm = (grid + sms - 1) / sms;
            const double staging = (4.0 * a.M * (P == 3 ? 260 : 45) / 32 + 20) / 65 * runs * RUN;
            const double warp_cost = iters * (runs * RUN + 1.0) + staging * (resident ? 1 : iters);
            // fewer than 16 warps on an SM have half as many to hide latency with
            const double cost = nw * warp_cost * on_sm * (nw * on_sm >= 16 ? 1.0 : 1.5);
            if (cost < best - 1e-9) {
                best = cost;
                best_grid = grid;
                best_warps = nw;
                pick.ks = ks;
                pick.iters = iters;
                pick.blk_runs = blk;
                pick.nred = nred;
                const size_t part = (blk * RUN * step_bytes + 127) / 128 * 128;
                pick.warp_bytes = static_cast<uint32_t>(part);
                pick.off_sum = static_cast<uint32_t>(blk * RUN * kFrags);
                pick.off_red = static_cast<uint32_t>(nw * part);
                best_smem = nw * part + red;
            }
        }
    }
    if (best_grid == 0) return cudaErrorInvalidConfiguration;
    auto kern = qmv_frag_kernel<BITS, XT, MODE, NT, VEC>;
    static PerDeviceAttr attr;
    cudaError_t e = attr.set(kern, kSmemMax);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(best_grid);
    cfg.blockDim = dim3(32 * best_warps);
    cfg.dynamicSmemBytes = best_smem;
    cfg.stream = st;
    cudaLaunchAttribute la[1];
    la[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    la[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = la;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, pick);
}

template <int BITS, int XT>
cudaError_t launch_type(cudaStream_t st, const FragArgs &a, const Shape &s, int sms) {
    if constexpr (BITS == 4 && XT != MTC_F32) {
        if (s.vec == 6) {
            if (s.mode == S1) return launch_one<BITS, XT, S1, 1, 6>(st, a, sms);
            if (s.mode == S2) return launch_one<BITS, XT, S2, 1, 6>(st, a, sms);
            if (s.mode == S4) return launch_one<BITS, XT, S4, 1, 6>(st, a, sms);
            if (s.nt == 1) return launch_one<BITS, XT, G8, 1, 6>(st, a, sms);
            return launch_one<BITS, XT, G8, 2, 6>(st, a, sms);
        }
        if (s.vec == 7) {
            if (s.mode == S1) return launch_one<BITS, XT, S1, 1, 7>(st, a, sms);
            if (s.mode == S2) return launch_one<BITS, XT, S2, 1, 7>(st, a, sms);
            if (s.mode == S4) return launch_one<BITS, XT, S4, 1, 7>(st, a, sms);
            if (s.nt == 1) return launch_one<BITS, XT, G8, 1, 7>(st, a, sms);
            return launch_one<BITS, XT, G8, 2, 7>(st, a, sms);
        }
    }
    if (s.mode == S1) return launch_one<BITS, XT, S1, 1, 0>(st, a, sms);
    if (s.mode == S2) {
        if (s.nt == 1) return launch_one<BITS, XT, S2, 1, 0>(st, a, sms);
        if (s.nt == 2) return launch_one<BITS, XT, S2, 2, 0>(st, a, sms);
        return launch_one<BITS, XT, S2, 4, 0>(st, a, sms);
    }
    if (s.mode == S4 && s.nt == 1) return launch_one<BITS, XT, S4, 1, 0>(st, a, sms);
    // f32 activations: eight token rows a launch at most (rows_per_launch)
    constexpr bool kMany = XT != MTC_F32;
    if constexpr (BITS == 4 || BITS == 8) {
        if (!kMany || s.nt == 1) return launch_one<BITS, XT, G8, 1, 0>(st, a, sms);
        if constexpr (kMany) return launch_one<BITS, XT, G8, 2, 0>(st, a, sms);
    } else {
        if (!kMany || s.nt == 2) return launch_one<BITS, XT, S4, 2, 0>(st, a, sms);
        if constexpr (kMany) return launch_one<BITS, XT, S4, 4, 0>(st, a, sms);
    }
}

template <int BITS>
cudaError_t launch_bits(cudaStream_t st, const FragArgs &a, const Shape &s, int sms) {
    if (s.xt == MTC_F32) return launch_type<BITS, MTC_F32>(st, a, s, sms);
    if (s.xt == MTC_F16) return launch_type<BITS, MTC_F16>(st, a, s, sms);
    return launch_type<BITS, MTC_BF16>(st, a, s, sms);
}

}  // namespace frag

// one translation unit per width (qmv_frag_b*.cu)
cudaError_t launch_frag_b2(cudaStream_t, const FragArgs &, const frag::Shape &, int);
cudaError_t launch_frag_b3(cudaStream_t, const FragArgs &, const frag::Shape &, int);
cudaError_t launch_frag_b4(cudaStream_t, const FragArgs &, const frag::Shape &, int);
cudaError_t launch_frag_b5(cudaStream_t, const FragArgs &, const frag::Shape &, int);
cudaError_t launch_frag_b6(cudaStream_t, const FragArgs &, const frag::Shape &, int);
cudaError_t launch_frag_b8(cudaStream_t, const FragArgs &, const frag::Shape &, int);

}  // namespace mtc
