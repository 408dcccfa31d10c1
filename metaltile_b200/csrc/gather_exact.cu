// gather_exact — the grouped (mixture-of-experts) 4-bit product of bf16 layers on tcgen05, with nothing rounded on the way:
//
//   out[r, n] = sum_k (q(e, n, k) * scale[e, n, k/G] + bias[e, n, k/G]) * x[r, k],   e = the expert that owns row r
//
// x rows are sorted by expert (expert_offsets, CSR).  Stands in for mt_moe_gather_qmm_int4{,_m8,_m16,_m32}
// (crates/metaltile-std/src/ffai/moe.rs:358-1363) where an expert sees some rows: then a layer is bound by reading every expert's packed
// matrix once, and by the instructions that make operands of its codes.
//
// Arithmetic.  With a bf16 scale (8 bits) and a 4-bit code, (q - 8) * scale has at most 11 bits: an f16 holds it.  So the operand is
// fma(q, scale, -8 * scale) in packed halves, where q is the masked word itself (a 16-bit float with exponent field 0 is linear in its low
// bits: q * 2^-24, or q * 2^-20 at bits 4..7) and the power of two sits in the factor: 9 instructions per 8 codes.  What is left, the sum over the
// groups of (bias + 8 * scale) * sum(x), is a short product of its own at the end of K: biases and 8 * scales against the sums of x, the sums cut
// into three bf16 pieces that hold their 24 bits.  Everything adds up in one f32 accumulator.  Powers of two keep the factors in f16's range: one for
// each weight row (its largest scale, or bias / 8, comes to [2^-9, 2^-8)), one for each row of x (its largest value to [2^14, 2^15)); the
// epilogue takes them out.  That holds every scale down to 2^-8 of its row's largest.  Where a row of the 32 of a warp has smaller ones, they come to
// [2^12, 2^13) instead and the operand is (1024 + q - 1032) * scale, 13 instructions, which holds them down to 2^-29 (the layer below 151 us
// before there was this form, 152.5 with it, 173 where every row takes it).  Rows with smaller ones yet or with
// an infinity, and infinite tokens, are added up from the definition.  Elements of x below 2^-31 of their row's largest are rounded, by 2^-40 of it at most, as every tcgen05 product of bf16 rows does.
//
// Work.  A PASS is (expert, up to TB of its rows); an item is a pass x 128 weight rows (64 of gate and 64 of up where one launch covers
// both), all of K.  One persistent CTA per SM walks the items; its roles meet at mbarriers and run ahead of each other across items:
//   warps 0-3    epilogue  the accumulator of an item: tcgen05.ld, factors, stores
//   warps 4-15   codes     three teams of 128 rows, every third stage: words out of shared memory, masked, multiplied, tcgen05.st
//   warp 16      producer  a stage at a time: 16 KB of packed words (128 bytes of each row) and the activations of the same codes; an item at a
//                          time: its scales and biases, which lie in one piece.  It also allocates and frees the tensor memory.
//   warp 17      MMA       four K = 16 steps a k block of 64 codes, A from tensor memory; two accumulators, items in turn
// Every wait is bounded: on expiry the kernel records a code in the status word, all roles leave, copies and MMAs in flight are awaited (bounded
// too) and the tensor memory is freed.
//
// What was measured on the way to this form (a layer of 512 tokens, 128 experts of 2048 x 768, top-8, us; the mma.sync kernel 257): the integer codes as
// operands, a group an accumulator that warps read back, scale and add: 367; every hand-off for four k blocks and by warp-uniform loops 294;
// polls of two instructions (a poll loop of eight took half of all issue slots), results out by loops, not unrolled code that is fetched anew for
// every item: 257; twice the warps at the accumulators 221.  A load of each lane's own row (scales) takes the load pipe ten cycles a lane, and
// is waited for together with the loads of tensor memory: 4 such loads a stage took 1000 cycles, hence the bulk copies.
#include <cstddef>

#include "far_tokens.cuh"
#include "tcgen05.cuh"

namespace mtc {
namespace {

constexpr int kRows = 128;                     // weight rows of an item: TMEM lanes, MMA M
constexpr int kBlk = 64;                       // codes of a k block: one 128-byte row of the activations' tile
constexpr int kChunk = 4;                      // k blocks of a stage: what one hand-off between the roles covers
constexpr int kWordBytes = kRows * 128;        // packed words of a stage
constexpr int kMaxStages = 8;
constexpr int kTeams = 3;                      // each with a place of its own for A: 4 k blocks of 32 columns
constexpr int kACols = kChunk * 32;
constexpr int kDCol0 = kTeams * kACols, kDCols = 64;
constexpr int kMaxTB = 64;
constexpr int kOutBytes = kMaxTB * kRows * 2;  // results of an item on their way out, [token][128 rows]
constexpr int kEpiWarps = 4, kCodeWarp0 = kEpiWarps, kCodeWarps = 4 * kTeams, kLoadWarp = kCodeWarp0 + kCodeWarps, kMmaWarp = kLoadWarp + 1;
constexpr int kThreads = (kMmaWarp + 1) * 32;
constexpr int kSmemBytes = 226 * 1024;         // of which the ring takes what the rest leaves
constexpr int kMaxPasses = 4096;
constexpr int kSlots = 8, kSegs = kBlk / kSlots;      // a segment of 64 codes in the last product: 8 elements of K; segments of a k block

struct EPass {
    int expert, tok0, ntok, pad;      // rows tok0 .. tok0 + ntok - 1 of the product
};
struct ETable {
    int n_pass, pad[3];
    EPass pass[kMaxPasses];
};

struct EArgs {
    const void *scales[2], *biases[2];        // of the matrix that owns rows 0..63 and 64..127 of an item
    void *outs[2];
    void *act;                       // not null: silu(rows 0..63) * rows 64..127 goes here, outs are not written
    const ETable *table;
    const float *tok_scale;          // powers of two that the rows of x were divided by; negative: an infinite row
    const uint32_t *w[2];            // for rows that are added up from the definition
    const __nv_bfloat16 *x;
    const uint32_t *row_src;
    int n_src_rows;
    uint32_t *status;
    int two;                         // 1: an item is 64 rows of each matrix; 0: 128 rows of the first
    int n_out, gpr, gs_shift;
    int tiles;                       // items of a pass
    int nkb, nlast;                  // k blocks of codes, then of biases and scales
    int nst;                         // stages of the ring
    uint32_t off_item, item_bytes;   // an item's scales, then its biases: 128 rows each, as they lie in memory; two such buffers
    uint32_t off_ring, stage;        // where the ring starts; bytes of a stage
};
struct EMaps {
    CUtensorMap x[4];                // boxes of 4 k blocks x 16, 32, 48 and 64 rows
    CUtensorMap w[2];                // boxes of 128 bytes x 64 rows
};

struct __align__(16) ECtrl {
    uint64_t full[kMaxStages], empty[kMaxStages];      // a stage has landed / its MMAs, and so all who read its words, are done
    uint64_t item_full[2], item_empty[2];              // an item's scales and biases
    uint64_t a_full[kTeams], a_empty[kTeams];          // a stage's A operand is complete / read
    uint64_t d_full[2], d_empty[2];                    // an item's accumulator is complete / read
    int4 head[2];                                      // the item's pass: expert, first row, rows
    uint32_t tmem_base;
    volatile uint32_t abort;
    uint32_t again_rows[2][kEpiWarps];                 // of an item's rows those that are added up from the definition for every token, and all that there are
    uint64_t drained;                                  // giving up: the MMAs are complete
    uint32_t stages_issued, items_issued;              // what the producer started
    alignas(16) float row_factor[2][kRows];            // negative: a row whose scales the operands do not hold
    alignas(16) float tok_factor[kEpiWarps][kMaxTB];
};
constexpr int kCtlBytes = (sizeof(ECtrl) + 1023) / 1024 * 1024;

// ---- preparation -----------------------------------------------------------------------------------------------------
// The activations row by row in the order of the product: f16 times a power of two of the row, the 8 elements that meet a word in the order of
// the word's operands (0 4 1 5 2 6 3 7), behind them the pieces of the sums of 64.  W warps share a row and hold it in registers between the maximum and
// the conversion, up to 2048 W elements; longer rows are read twice.  Row m of the product is row row_src[m] of x (the permutation of
// mt_moe_permute, moe.rs:222-281, without the copy), or row m where there is no row_src.
// Block 0 also walks expert_offsets: expert e with r rows gives ceil(r / TB) passes of nearly equal size.  Offsets that are not monotone or
// reach past m_total are clamped (the rows they would have named are left out) and reported in the status word (0x901).
__device__ void build_passes(const uint32_t *offsets, int n_experts, int m_total, int TB, ETable *table, uint32_t *status) {
    const int lane = threadIdx.x & 31;
    int n_pass = 0;
    bool bad = false, over = false;
    for (int e0 = 0; e0 < n_experts; e0 += 32) {
        const int e = e0 + lane;
        int lo = 0, hi = 0;
        if (e < n_experts) {
            const uint32_t a = offsets[e], b = offsets[e + 1], m = static_cast<uint32_t>(m_total);
            lo = static_cast<int>(min(a, m));
            hi = static_cast<int>(min(b, m));
            if (a > m || b > m || b < a) bad = true;
            if (hi < lo) hi = lo;
        }
        const int rows = hi - lo, np = (rows + TB - 1) / TB, per = np ? (rows + np - 1) / np : 0;
        int pp = np;                       // inclusive scan over these 32 experts
        for (int d = 1; d < 32; d <<= 1) {
            const int up = __shfl_up_sync(0xffffffffu, pp, d);
            if (lane >= d) pp += up;
        }
        const int p0 = n_pass + pp - np;
        for (int i = 0; i < np; ++i) {
            if (p0 + i < kMaxPasses) table->pass[p0 + i] = EPass{e, lo + i * per, min(per, rows - i * per), 0};
            else over = true;
        }
        n_pass += __shfl_sync(0xffffffffu, pp, 31);
    }
    bad = __any_sync(0xffffffffu, bad);
    over = __any_sync(0xffffffffu, over);
    if (lane == 0) {
        table->n_pass = over ? 0 : n_pass;         // a table that does not fit runs nothing: the caller is told
        if (bad) atomicCAS(status, 0u, 0x901u);
        if (over) atomicCAS(status, 0u, 0x902u);
    }
}

template <int W>
__global__ void __launch_bounds__(256) exact_prep_kernel(const __nv_bfloat16 *x, const uint32_t *row_src, int n_src_rows, const uint32_t *offsets, int n_experts,
                                                         int m_total, int K, int row_elems, int TB, unsigned short *xprep, float *tok_scale, ETable *table,
                                                         uint32_t *status) {
    pdl_enter();
    constexpr int ROWS = 8 / W, HELD = 8, STEP = 32 * W;
    __shared__ uint32_t part[8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (blockIdx.x == gridDim.x - 1) {             // a block of its own
        if (warp == 0) build_passes(offsets, n_experts, m_total, TB, table, status);
        return;
    }
    const int m = blockIdx.x * ROWS + warp / W, i0 = (warp % W) * 32 + lane;
    const bool on = m < m_total;
    const int nvec = on ? K / 8 : 0;
    size_t src = on ? m : 0;
    if (row_src && on) {
        const uint32_t r = row_src[m];
        if (r >= static_cast<uint32_t>(n_src_rows)) atomicCAS(status, 0u, 0x903u);     // not a row of x: row 0 is read instead
        src = r < static_cast<uint32_t>(n_src_rows) ? r : 0;
    }
    const uint4 *from = reinterpret_cast<const uint4 *>(x + src * K);
    unsigned short *const row = xprep + static_cast<size_t>(on ? m : 0) * row_elems;
    uint4 held[HELD];
#pragma unroll
    for (int q = 0; q < HELD; ++q) held[q] = i0 + q * STEP < nvec ? from[i0 + q * STEP] : make_uint4(0u, 0u, 0u, 0u);
    uint32_t amax = 0;                             // two maxima of |x| as bf16 bit patterns (monotone for finite values)
    auto fold = [&](const uint4 &v) {
        amax = __vmaxu2(amax, __vmaxu2(__vmaxu2(v.x & 0x7FFF7FFFu, v.y & 0x7FFF7FFFu), __vmaxu2(v.z & 0x7FFF7FFFu, v.w & 0x7FFF7FFFu)));
    };
#pragma unroll
    for (int q = 0; q < HELD; ++q) fold(held[q]);
    for (int i = i0 + HELD * STEP; i < nvec; i += STEP) fold(from[i]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) amax = __vmaxu2(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    if constexpr (W > 1) {
        if (lane == 0) part[warp] = amax;
        __syncthreads();
#pragma unroll
        for (int w = 0; w < W; ++w) amax = __vmaxu2(amax, part[warp / W * W + w]);
    }
    const int ex = static_cast<int>(max(amax & 0xFFFFu, amax >> 16) >> 7);      // biased exponent of the row maximum
    const int e = ex == 0 || ex == 0xFF ? 0 : max(ex - 127 - 14, -126);        // zero rows and inf / nan rows stay unscaled; 2^-e and 2^e both normal
    const float down = __uint_as_float(static_cast<uint32_t>(127 - e) << 23);
    // negative: an infinity and no NaN.  The products with such a token are added up from the definition.
    if (on && i0 == 0) tok_scale[m] = __uint_as_float(static_cast<uint32_t>(127 + e) << 23 | (max(amax & 0xFFFFu, amax >> 16) == 0x7F80u ? 0x80000000u : 0u));
    auto convert = [&](int i, const uint4 &v) {
        const bool here = i < nvec;
        const uint32_t u[4] = {v.x, v.y, v.z, v.w};
        uint32_t h[4];
        float sum = 0.0f;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float lo = __uint_as_float(u[j] << 16) * down, hi = __uint_as_float(u[j] & 0xFFFF0000u) * down;
            sum += lo + hi;
            const __half2 p = __floats2half2_rn(lo, hi);
            h[j] = *reinterpret_cast<const uint32_t *>(&p);
        }
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);       // eight lanes hold a segment
        if (!here) return;
        *reinterpret_cast<uint4 *>(row + static_cast<size_t>(i) * 8) = make_uint4(__byte_perm(h[0], h[2], 0x5410), __byte_perm(h[0], h[2], 0x7632),
                                                                                 __byte_perm(h[1], h[3], 0x5410), __byte_perm(h[1], h[3], 0x7632));
        if ((i & 7) != 0) return;
        // three bf16 pieces that hold the 24 bits; an infinity or a NaN is all in the first
        const uint32_t p1 = __float_as_uint(sum) & 0xFFFF0000u;
        const float r1 = (p1 & 0x7F800000u) != 0x7F800000u ? sum - __uint_as_float(p1) : 0.0f;
        const uint32_t p2 = __float_as_uint(r1) & 0xFFFF0000u, p3 = __float_as_uint(r1 - __uint_as_float(p2));
        const uint32_t top = sum != sum ? 0x7FC00000u : p1;      // a NaN whose bits are all in the lower half must not become an infinity
        // against (b b b t t t 0 0), t = 8 * scale
        const int seg = i >> 3;
        uint4 *const to = reinterpret_cast<uint4 *>(row + K + seg * kSlots);
        *to = make_uint4((top >> 16) | p2, (p3 >> 16) | top, (p2 >> 16) | (p3 & 0xFFFF0000u), 0u);
        if (seg == K / 64 - 1)                               // the end of the last block meets zeros, and must be finite
            for (uint4 *z = to + 1; z < reinterpret_cast<uint4 *>(row + row_elems); ++z) *z = make_uint4(0u, 0u, 0u, 0u);
    };
    const int rounds = (K / 8 + STEP - 1) / STEP;            // whole warps: the sums use shuffles
#pragma unroll
    for (int q = 0; q < HELD; ++q)
        if (q < rounds) convert(i0 + q * STEP, held[q]);
    for (int q = HELD; q < rounds; ++q) {
        const int i = i0 + q * STEP;
        convert(i, i < nvec ? from[i] : make_uint4(0u, 0u, 0u, 0u));
    }
}

// ---- the product -----------------------------------------------------------------------------------------------------
__device__ __forceinline__ bool epilogue_votes(bool ok) {
    uint32_t all;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.and.pred q, 1, 128, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
                 : "=r"(all) : "r"(static_cast<uint32_t>(ok)) : "memory");
    return all != 0;
}
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}
// silu(g) * u of two bf16 pairs, as mt_swiglu rounds it (crates/metaltile-std/src/mlx/swiglu.rs:45-57)
__device__ __forceinline__ uint32_t silu_mul(uint32_t g, uint32_t u) {
    const float g0 = __uint_as_float(g << 16), g1 = __uint_as_float(g & 0xFFFF0000u), u0 = __uint_as_float(u << 16), u1 = __uint_as_float(u & 0xFFFF0000u);
    return pack_bf16((g0 / (1.0f + expf(-g0))) * u0, (g1 / (1.0f + expf(-g1))) * u1);
}
__device__ __forceinline__ uint32_t hmul2(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ uint32_t hfma2(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t r;
    asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
    return r;
}

// q - 8 of the codes at bits 0..3 / 4..7 of either half: 1024 + q (1024 + 16 q) by an OR
__device__ __forceinline__ uint32_t low_code(uint32_t w) {
    uint32_t r;
    asm("add.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"((w & 0x000F000Fu) | 0x64006400u), "r"(0xE408E408u /* -1032 */));
    return r;
}
__device__ __forceinline__ uint32_t high_code(uint32_t w) {
    return hfma2((w & 0x00F000F0u) | 0x64006400u, 0x2C002C00u /* 2^-4 */, 0xD480D480u /* -72 */);
}

// Two 16-bit values from shared memory; WIDE: the address is a multiple of 4
template <bool WIDE>
__device__ __forceinline__ uint32_t lds4(uint32_t addr) {
    if constexpr (WIDE) {
        uint32_t v;
        asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr));
        return v;
    } else {
        unsigned short lo, hi;
        asm volatile("ld.shared.u16 %0, [%1];" : "=h"(lo) : "r"(addr));
        asm volatile("ld.shared.u16 %0, [%1];" : "=h"(hi) : "r"(addr + 2));
        return lo | static_cast<uint32_t>(hi) << 16;
    }
}
// Eight of them; ALIGN: what the address is a multiple of, 16, 4 or 2
template <int ALIGN>
__device__ __forceinline__ uint4 lds16(uint32_t addr) {
    uint4 v;
    if constexpr (ALIGN == 16) {
        asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
    } else {
        v = make_uint4(lds4<ALIGN == 4>(addr), lds4<ALIGN == 4>(addr + 4), lds4<ALIGN == 4>(addr + 8), lds4<ALIGN == 4>(addr + 12));
    }
    return v;
}
__device__ __forceinline__ uint32_t max4(const uint4 &v) {          // of |bf16| pairs
    return __vmaxu2(__vmaxu2(v.x & 0x7FFF7FFFu, v.y & 0x7FFF7FFFu), __vmaxu2(v.z & 0x7FFF7FFFu, v.w & 0x7FFF7FFFu));
}
__device__ __forceinline__ uint32_t min4(const uint4 &v) {
    return __vminu2(__vminu2(v.x & 0x7FFF7FFFu, v.y & 0x7FFF7FFFu), __vminu2(v.z & 0x7FFF7FFFu, v.w & 0x7FFF7FFFu));
}
// the least |bf16| of a row of `rb` bytes that is not zero; 0x7FFF without one
__device__ __noinline__ uint32_t least_nonzero(uint32_t row, uint32_t rb) {
    uint32_t low = 0x7FFFu;
    for (uint32_t g = 0; g < rb; g += 2) {
        unsigned short v;
        asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(row + g));
        if (v & 0x7FFF) low = min(low, v & 0x7FFFu);
    }
    return low;
}

// A stage's k blocks in the form for scales far apart: pair, later: the scales of its groups.  Not inlined, so that the other form's loop stays in one piece.
__device__ __noinline__ void wide_blocks(uint32_t words, int r, uint32_t dst, int blocks, uint32_t pair, uint32_t later, bool groups64, float f) {
#pragma unroll 1
    for (int j = 0; j < blocks; ++j) {
        uint32_t v[32];
        const __half2 s2 = __float2half2_rn(__uint_as_float(pair << 16) * f);
        const uint32_t s = *reinterpret_cast<const uint32_t *>(&s2);
        if (groups64 || (j & 1)) pair = (j & 1) && groups64 ? later : pair >> 16;
#pragma unroll
        for (int p = 0; p < 2; ++p) {
            const uint4 q = lds16<16>(words + (((2 * j + p) ^ (r & 7)) << 4));
            const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const uint32_t u = w[k] >> 8;
                v[16 * p + 4 * k] = hmul2(low_code(w[k]), s);
                v[16 * p + 4 * k + 1] = hmul2(high_code(w[k]), s);
                v[16 * p + 4 * k + 2] = hmul2(low_code(u), s);
                v[16 * p + 4 * k + 3] = hmul2(high_code(u), s);
            }
        }
        tmem_st32(dst + j * 32, v);
    }
}

// Results of an item that its operands do not hold, in the buffer of results, by the definition, a warp an output: those of the marked weight rows (`row`:
// that of the calling thread of the epilogue is), and those of infinite tokens, where the infinity has met zeros and values of the other sign on
// the way.
__device__ __noinline__ void from_definition(const EArgs &a, ECtrl *ctl, const int4 pass, const int n0, const bool row) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, K = a.gpr << a.gs_shift;
    const bool exists = n0 + (a.two ? threadIdx.x & 63 : threadIdx.x) < static_cast<uint32_t>(a.n_out);
    const uint32_t marked = __ballot_sync(0xffffffffu, row && exists), all = __ballot_sync(0xffffffffu, exists);
    if (lane == 0) {
        ctl->again_rows[0][warp] = marked;
        ctl->again_rows[1][warp] = all;
    }
    asm volatile("bar.sync 1, 128;" ::: "memory");
    unsigned short *const staged = reinterpret_cast<unsigned short *>(reinterpret_cast<uint8_t *>(ctl) + kCtlBytes);
    for (int t = warp; t < pass.z; t += kEpiWarps) {         // the tokens that this warp stores
        size_t src = pass.y + t;
        if (a.row_src) src = a.row_src[src] < static_cast<uint32_t>(a.n_src_rows) ? a.row_src[src] : 0;
        const __nv_bfloat16 *const x = a.x + src * K;
        const int which = ctl->tok_factor[warp][t] < 0.0f;
        for (int q = 0; q < kRows / 32; ++q)
            for (uint32_t todo = ctl->again_rows[which][q]; todo != 0; todo &= todo - 1) {
                const int at = q * 32 + __ffs(todo) - 1, m = a.two ? at >> 6 : 0;
                const size_t n = static_cast<size_t>(pass.x) * a.n_out + n0 + (a.two ? at & 63 : at);
                const float v = far_tokens::sum<4, MTC_BF16>(a.w[m] + n * (K / 8), static_cast<const __nv_bfloat16 *>(a.scales[m]) + n * a.gpr,
                                                             static_cast<const __nv_bfloat16 *>(a.biases[m]) + n * a.gpr, x, K, a.gs_shift);
                if (lane == 0) staged[t * kRows + at] = static_cast<unsigned short>(pack_bf16(v, 0.0f));
            }
        __syncwarp();
    }
}

// A launch that gave up, once every role has ended: lets what is on its way arrive before the CTA tears down.
__device__ __noinline__ void rest(ECtrl *ctl, int nst) {
    const int warp = threadIdx.x >> 5;
    if (warp == kMmaWarp && elect_one()) {
        umma_commit(&ctl->drained);
        drain_ring(&ctl->drained, 1, 1);
    } else if (warp == kLoadWarp && (threadIdx.x & 31) == 0) {
        drain_ring(ctl->full, ctl->stages_issued, nst);
        drain_ring(ctl->item_full, ctl->items_issued, 2);
    }
    __syncthreads();
}

__global__ void __launch_bounds__(kThreads, 1) gather_exact_kernel(const __grid_constant__ EMaps maps, const __grid_constant__ EArgs a) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    ECtrl *ctl = reinterpret_cast<ECtrl *>(smem);      // then the results, two items' scales and biases, the ring
    uint8_t *const staged = smem + kCtlBytes;
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;       // known to be uniform
    const int nst = a.nst;
    const uint32_t stage = a.stage, bars = __shfl_sync(0xffffffffu, smem_u32(smem), 0), ring = bars + a.off_ring, items = bars + a.off_item;
    if (threadIdx.x == 0) {
        for (int s = 0; s < kMaxStages; ++s) {
            mbar_init(&ctl->full[s], 1);
            mbar_init(&ctl->empty[s], 1);
        }
        for (int s = 0; s < kTeams; ++s) {
            mbar_init(&ctl->a_full[s], 4);
            mbar_init(&ctl->a_empty[s], 1);
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(&ctl->item_full[s], 1);
            mbar_init(&ctl->item_empty[s], kEpiWarps + kCodeWarps + 1);
            mbar_init(&ctl->d_full[s], 1);
            mbar_init(&ctl->d_empty[s], kEpiWarps);
        }
        mbar_init(&ctl->drained, 1);
        ctl->abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kLoadWarp) tmem_alloc_all(&ctl->tmem_base);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, ctl->tmem_base, 0);
    pdl_enter();                                        // the table and the activations; nothing is stored before
    const uint32_t full = bars + offsetof(ECtrl, full), empty = bars + offsetof(ECtrl, empty), a_full = bars + offsetof(ECtrl, a_full),
                   a_empty = bars + offsetof(ECtrl, a_empty), d_full = bars + offsetof(ECtrl, d_full), d_empty = bars + offsetof(ECtrl, d_empty),
                   item_full = bars + offsetof(ECtrl, item_full), item_empty = bars + offsetof(ECtrl, item_empty), abort = bars + offsetof(ECtrl, abort);
    const int n_items = a.table->n_pass * a.tiles;
    const int ncc = (a.nkb + kChunk - 1) / kChunk, nch = ncc + (a.nlast + kChunk - 1) / kChunk;       // stages of codes, and with the last ones
    const int tile_rows = a.two ? 64 : 128;
    auto wait = [&](uint32_t bar, uint32_t parity, uint32_t code) { return mbar_wait(bar, parity, abort, a.status, code); };

    if (warp == kLoadWarp) {
        // ---------------- producer ----------------
        if (lane == 0) {
            auto pass_of = [&](int i) { return i < n_items ? *reinterpret_cast<const int4 *>(&a.table->pass[i / a.tiles]) : make_int4(0, 0, 0, 0); };
            int s = 0;
            uint32_t ph = 0, e = 0, eph = 0, laps = 0, started = 0;
            bool ok = true;
            int4 next = pass_of(blockIdx.x);
            for (int i = blockIdx.x; i < n_items && ok; i += gridDim.x) {
                const int4 pass = next;
                next = pass_of(i + gridDim.x);
                const int n0 = i % a.tiles * tile_rows, cols = (pass.z + 15) & ~15;
                if (!(ok = wait(item_empty + e * 8, eph ^ 1, 0xa01))) break;
                ctl->head[e] = pass;
                {
                    // rows of the first and of the second half that exist
                    const int left0 = min(64, a.n_out - n0), left1 = a.two ? left0 : min(64, max(a.n_out - n0 - 64, 0));
                    const uint32_t rb = a.gpr * 2, dst = items + e * a.item_bytes;
                    const size_t at = (static_cast<size_t>(pass.x) * a.n_out + n0) * rb;
                    mbar_expect_tx(&ctl->item_full[e], 2 * (left0 + left1) * rb);
#pragma unroll
                    for (int k = 0; k < 2; ++k) {
                        const char *const first = static_cast<const char *>(k ? a.biases[0] : a.scales[0]), *const second = static_cast<const char *>(k ? a.biases[1] : a.scales[1]);
                        bulk_load(dst + k * (kRows * rb), first + at, left0 * rb, &ctl->item_full[e]);
                        if (left1 > 0) bulk_load(dst + k * (kRows * rb) + 64 * rb, second + at + (a.two ? 0 : 64 * rb), left1 * rb, &ctl->item_full[e]);
                    }
                    eph ^= e;
                    e ^= 1;
                    ++started;
                }
                const CUtensorMap *const map_x = &maps.x[(cols >> 4) - 1];
                const int row0 = pass.x * a.n_out + n0, row1 = a.two ? row0 : row0 + 64;
                for (int c = 0; c < nch; ++c) {
                    if (!(ok = wait(empty + s * 8, ph ^ 1, 0xa02))) break;
                    const uint32_t dst = ring + s * stage;
                    uint64_t *const bar = &ctl->full[s];
                    const bool codes = c < ncc;
                    mbar_expect_tx(bar, (codes ? kWordBytes : 0) + kChunk * cols * 128);
                    if (codes) {                        // rows past the array and words past the row arrive as zeros; rows past n_out are never stored
                        tma_load_2d(dst, &maps.w[0], c * (kChunk * 8), row0, bar);
                        tma_load_2d(dst + kWordBytes / 2, &maps.w[a.two], c * (kChunk * 8), row1, bar);
                    }
                    tma_load_3d(dst + kWordBytes, map_x, 0, pass.y, codes ? c * kChunk : a.nkb + (c - ncc) * kChunk, bar);       // blocks past the row too
                    if (++s == nst) { s = 0; ph ^= 1; ++laps; }
                }
            }
            ctl->stages_issued = laps * nst + s;
            ctl->items_issued = started;
        }
    } else if (warp == kMmaWarp) {
        // ---------------- MMA ----------------
        // A wait costs its warp some 75 cycles even where the barrier is complete, four MMAs with addresses that are known to be uniform 60, others
        // 190: the whole warp runs the loop, its control flow depends on votes alone, one elected lane issues.
        const bool leader = elect_one();
        const uint64_t bdesc0 = make_desc_sw128(ring + kWordBytes);
        auto uniform = [&](bool ok) { return __all_sync(0xffffffffu, ok); };
        auto role = [&]() {
            int s = 0;
            uint32_t ph = 0, team = 0, aph = 0, e = 0, eph = 0;           // e, eph: the item's scales, and its accumulator
            for (int i = blockIdx.x; i < n_items; i += gridDim.x) {
                if (!uniform(wait(item_full + e * 8, eph, 0xa03))) return;
                const uint32_t cols = __shfl_sync(0xffffffffu, (ctl->head[e].z + 15) & ~15, 0), blk = cols * 8;
                if (lane == 0) mbar_arrive(item_empty + e * 8);
                __syncwarp();
                const uint32_t f16 = (1u << 4) | ((cols >> 3) << 17) | (static_cast<uint32_t>(kRows >> 4) << 24), bf16 = f16 | (1u << 7) | (1u << 10);
                const uint32_t dd = tmem + kDCol0 + e * kDCols;
                if (!uniform(wait(d_empty + e * 8, eph ^ 1, 0xa04))) return;
                for (int c = 0; c < nch; ++c) {
                    const bool codes = c < ncc;
                    const int blocks = codes ? a.nkb - c * kChunk : a.nlast - (c - ncc) * kChunk;      // at least 4 but in the last stage of a kind
                    const uint32_t idesc = codes ? f16 : bf16, aa = tmem + team * kACols;
                    const uint64_t bd = bdesc0 + static_cast<uint64_t>((s * stage) >> 4);
                    if (!uniform(wait(full + s * 8, ph, 0xa05))) return;
                    if (!uniform(wait(a_full + team * 8, aph, 0xa06))) return;
                    tc_fence_after();
                    if (leader) {
#pragma unroll
                        for (int j = 0; j < kChunk; ++j)
                            if (j < blocks) {
#pragma unroll
                                for (int k = 0; k < 4; ++k) umma_f16_ts(dd, aa + j * 32 + 8 * k, bd + static_cast<uint64_t>(j * blk + 2 * k), idesc, (c | j | k) ? 1u : 0u);
                            }
                        umma_commit(a_empty + team * 8);
                        umma_commit(empty + s * 8);
                        if (c + 1 == nch) umma_commit(d_full + e * 8);
                    }
                    __syncwarp();
                    if (++team == kTeams) { team = 0; aph ^= 1; }
                    if (++s == nst) { s = 0; ph ^= 1; }
                }
                eph ^= e;
                e ^= 1;
            }
        };
        role();
    } else if (warp >= kCodeWarp0) {
        // ---------------- codes: packed words -> A operand ----------------
        const int q = warp & 3, team = (warp - kCodeWarp0) >> 2, r = q * 32 + lane;
        const uint32_t dst = tmem + (static_cast<uint32_t>(q * 32) << 16) + team * kACols, words0 = ring + r * 128;
        const uint32_t rb = a.gpr * 2;
        const int align = rb % 16 == 0 ? 16 : rb % 4 == 0 ? 4 : 2;
        auto role = [&]() {
            int s = 0, turn = 0;                        // stage of the ring; whose stage it is
            uint32_t ph = 0, aph = 0, e = 0, eph = 0;
            for (int i = blockIdx.x; i < n_items; i += gridDim.x) {
                if (!wait(item_full + e * 8, eph, 0xa07)) return;
                __syncwarp();
                const uint32_t row = items + e * a.item_bytes + r * rb, brow = row + kRows * rb;
                // the power of two of the row, by its largest scale or bias / 8, and its least scale.  (Loops that run once an item are not unrolled, here and in the
                // epilogue: straight-line code is fetched anew, a line of it some 250 cycles.  512 tokens of 128 experts 154.7 -> 152.0 us.)
                uint32_t top = 0, btop = 0, low = 0x7FFF7FFFu;
                if (align == 16) {                      // lanes start at different pieces: rows lie 64 bytes apart, or some such number
                    uint32_t at = (lane >> 1) * 16 % rb;
#pragma unroll 1
                    for (uint32_t g = 0; g < rb; g += 16) {
                        const uint4 sv = lds16<16>(row + at);
                        top = __vmaxu2(top, max4(sv));
                        low = __vminu2(low, min4(sv));
                        btop = __vmaxu2(btop, max4(lds16<16>(brow + at)));
                        at = at + 16 == rb ? 0 : at + 16;
                    }
                } else if (align == 4) {
#pragma unroll 1
                    for (uint32_t g = 0; g < rb; g += 4) {
                        const uint32_t sv = lds4<true>(row + g) & 0x7FFF7FFFu;
                        top = __vmaxu2(top, sv);
                        low = __vminu2(low, sv);
                        btop = __vmaxu2(btop, lds4<true>(brow + g) & 0x7FFF7FFFu);
                    }
                } else {                                // an odd number: the last one with the one before it
#pragma unroll 1
                    for (uint32_t g = 0; g < rb; g += 4) {
                        const uint32_t at = min(g, rb - min(rb, 4u));
                        const uint32_t sv = lds4<false>(row + at), bv = lds4<false>(brow + at), keep = rb == 2 ? 0x7FFFu : 0x7FFF7FFFu;
                        top = __vmaxu2(top, sv & keep);
                        low = __vminu2(low, (sv & keep) | (0x7FFF7FFFu & ~keep));
                        btop = __vmaxu2(btop, bv & keep);
                    }
                }
                const int es = static_cast<int>(max(top & 0xFFFFu, top >> 16) >> 7), eb = static_cast<int>(max(btop & 0xFFFFu, btop >> 16) >> 7);
                const int ex = max(es, eb - 3);
                uint32_t least = min(low & 0xFFFFu, low >> 16);
                if (least == 0) least = least_nonzero(row, rb);
                // the biased exponent of the factor: 2^(118 - ex), or 2^(139 - ex) where that leaves a scale of these rows less than 2^-17, whose last bit f16 does
                // not hold.  Rows that this leaves one, too, are marked, and those with an infinity.
                int up = max(245 - ex, 1);
                const bool far = static_cast<int>(least >> 7) + up < 237 || ex >= 252;
                bool wide = __any_sync(0xffffffffu, far), mark = false;
                if (wide) {                             // rows past n_out hold what an item before left in the buffer, or nothing yet
                    const bool exists = i % a.tiles * tile_rows + (a.two ? r & 63 : r) < a.n_out;
                    wide = __any_sync(0xffffffffu, far && exists);
                    if (wide) up = min(max(266 - ex, 1), 253);
                    mark = exists && (static_cast<int>(least >> 7) + up < 237 || ex >= 252);
                }
                const float f = __uint_as_float(static_cast<uint32_t>(up) << 23);
                for (int c = 0; c < nch; ++c) {
                    if (turn == team) {
                        if (c == 0) ctl->row_factor[e][r] = __uint_as_float(static_cast<uint32_t>(254 - up) << 23 | (mark ? 0x80000000u : 0u));
                        // in this order: with the MMAs of this team's stage before complete, the pass of the ring before this one is, and
                        // its phase cannot be taken for this one's
                        if (!wait(a_empty + team * 8, aph ^ 1, 0xa09)) return;
                        if (!wait(full + s * 8, ph, 0xa08)) return;
                        __syncwarp();
                        tc_fence_after();
                        aph ^= 1;
                        if (c < ncc) {
                            const int blocks = min(kChunk, a.nkb - c * kChunk);
                            const uint32_t words = words0 + s * stage;
                            uint32_t pair, later = 0;        // the stage's scales
                            const uint32_t at = row + (a.gs_shift == 7 ? c * 4 : c * 8);
                            if (a.gs_shift == 6 && a.gpr % 4 == 0) {
                                asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(pair), "=r"(later) : "r"(at));
                            } else {
                                pair = align == 2 ? lds4<false>(at) : lds4<true>(at);
                                if (a.gs_shift == 6) later = align == 2 ? lds4<false>(at + 4) : lds4<true>(at + 4);
                            }
                            if (wide) wide_blocks(words, r, dst, blocks, pair, later, a.gs_shift == 6, f);
#pragma unroll 1
                            for (int j = wide ? blocks : 0; j < blocks; ++j) {
                                uint32_t w[8], v[32];
#pragma unroll
                                for (int p = 0; p < 2; ++p)
                                    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(w[4 * p]), "=r"(w[4 * p + 1]), "=r"(w[4 * p + 2]), "=r"(w[4 * p + 3])
                                                 : "r"(words + (((2 * j + p) ^ (r & 7)) << 4)));
                                const __half2 s24 = __float2half2_rn(__uint_as_float(pair << 16) * f * 16777216.0f);       // 2^24: the codes are q * 2^-24
                                if (a.gs_shift == 6 || (j & 1)) {        // on to the next group
                                    pair = (j & 1) && a.gs_shift == 6 ? later : pair >> 16;
                                }
                                const uint32_t s0 = *reinterpret_cast<const uint32_t *>(&s24);
                                const uint32_t s1 = hmul2(s0, 0x2C002C00u /* 2^-4 */), off = hmul2(s0, 0x80088008u /* -2^-21 */);
#pragma unroll
                                for (int k = 0; k < 8; ++k) {
                                    const uint32_t u = w[k] >> 8;
                                    v[4 * k] = hfma2(w[k] & 0x000F000Fu, s0, off);
                                    v[4 * k + 1] = hfma2(w[k] & 0x00F000F0u, s1, off);
                                    v[4 * k + 2] = hfma2(u & 0x000F000Fu, s0, off);
                                    v[4 * k + 3] = hfma2(u & 0x00F000F0u, s1, off);
                                }
                                tmem_st32(dst + j * 32, v);
                            }
                        } else {
                            // biases and 8 * scales of the segments, three times each against the pieces of their sums
                            const int b0 = (c - ncc) * kChunk, blocks = min(kChunk, a.nlast - b0);
#pragma unroll 1
                            for (int j = 0; j < blocks; ++j) {
                                const int seg0 = (b0 + j) * kSegs;
                                const uint32_t at = (seg0 << 6 >> a.gs_shift) << 1;      // 8 groups of 64, or 4 of 128; past the row's end they are not used
                                uint4 sv, bv;
                                if (align == 16 && a.gs_shift == 6) {
                                    sv = lds16<16>(row + at);
                                    bv = lds16<16>(brow + at);
                                } else if (align != 2) {
                                    sv = lds16<4>(row + at);
                                    bv = lds16<4>(brow + at);
                                } else {
                                    sv = lds16<2>(row + at);
                                    bv = lds16<2>(brow + at);
                                }
                                const uint32_t sw[4] = {sv.x, sv.y, sv.z, sv.w}, bw[4] = {bv.x, bv.y, bv.z, bv.w};
                                uint32_t v[32];
#pragma unroll
                                for (int k = 0; k < kSegs; ++k) {
                                    const uint32_t s16 = a.gs_shift == 6 ? sw[k >> 1] >> (16 * (k & 1)) : sw[k >> 2] >> (16 * ((k >> 1) & 1));
                                    const uint32_t b16 = a.gs_shift == 6 ? bw[k >> 1] >> (16 * (k & 1)) : bw[k >> 2] >> (16 * ((k >> 1) & 1));
                                    const bool in = seg0 + k < a.nkb;
                                    const uint32_t b = in ? __float_as_uint(__uint_as_float(b16 << 16) * f) >> 16 : 0u;
                                    const uint32_t t = in ? __float_as_uint(__uint_as_float(s16 << 16) * f * 8.0f) >> 16 : 0u;
                                    v[4 * k] = b | b << 16;
                                    v[4 * k + 1] = b | t << 16;
                                    v[4 * k + 2] = t | t << 16;
                                    v[4 * k + 3] = 0u;
                                }
                                tmem_st32(dst + j * 32, v);
                            }
                        }
                        tmem_wait_st();
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(a_full + team * 8);
                    }
                    if (++turn == kTeams) turn = 0;
                    if (++s == nst) { s = 0; ph ^= 1; }
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(item_empty + e * 8);
                eph ^= e;
                e ^= 1;
            }
        };
        role();
    } else {
        // ---------------- epilogue ----------------
        const int r = warp * 32 + lane;
        const uint32_t d0 = tmem + (static_cast<uint32_t>(warp * 32) << 16) + kDCol0;
        float *const tf = ctl->tok_factor[warp];
        uint32_t e = 0, eph = 0;
        for (int i = blockIdx.x; i < n_items; i += gridDim.x) {
            bool ok = wait(item_full + e * 8, eph, 0xa0a);
            __syncwarp();
            const int4 pass = ctl->head[e];
            bool infinite = false;                  // a token is
            if (ok) {
#pragma unroll
                for (int p = 0; p < kMaxTB; p += 32) {
                    const float f = p + lane < pass.z ? a.tok_scale[pass.y + p + lane] : 0.0f;
                    infinite = infinite || f < 0.0f;
                    tf[p + lane] = f;
                }
                ok = wait(d_full + e * 8, eph, 0xa0b);
            }
            __syncwarp();
            // The warps share the buffer and named barriers, so they give up together; by this vote the item before has left the buffer.
            // Items with results that the operands do not hold are found by the same vote.
            const float rf = ok ? ctl->row_factor[e][r] : 0.0f;
            bool again = false;
            if (!epilogue_votes(ok && rf >= 0.0f && !infinite)) {
                if (!epilogue_votes(ok)) break;
                again = true;
            }
            tc_fence_after();
            unsigned short *const to = reinterpret_cast<unsigned short *>(staged) + r;
#pragma unroll 1
            for (int t0 = 0; t0 < pass.z; t0 += 16) {
                uint32_t v[16];
                tmem_ld<16>(d0 + e * kDCols + t0, v);
                tmem_wait_ld();
#pragma unroll
                for (int t = 0; t < 16; t += 4) {
                    const float4 ts = *reinterpret_cast<const float4 *>(tf + t0 + t);
                    const uint32_t lo = pack_bf16(__uint_as_float(v[t]) * rf * ts.x, __uint_as_float(v[t + 1]) * rf * ts.y);
                    const uint32_t hi = pack_bf16(__uint_as_float(v[t + 2]) * rf * ts.z, __uint_as_float(v[t + 3]) * rf * ts.w);
                    to[(t0 + t) * kRows] = static_cast<unsigned short>(lo);
                    to[(t0 + t + 1) * kRows] = static_cast<unsigned short>(lo >> 16);
                    to[(t0 + t + 2) * kRows] = static_cast<unsigned short>(hi);
                    to[(t0 + t + 3) * kRows] = static_cast<unsigned short>(hi >> 16);
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(d_empty + e * 8);
                mbar_arrive(item_empty + e * 8);
            }
            eph ^= e;
            e ^= 1;
            asm volatile("bar.sync 1, 128;" ::: "memory");
            const int n0 = i % a.tiles * tile_rows;
            if (again) from_definition(a, ctl, pass, n0, rf < 0.0f);
            // out of shared memory, a token a warp
            if (a.act) {
                const int n = n0 + 2 * lane;
                const bool pairs = (a.n_out & 1) == 0 && (reinterpret_cast<uintptr_t>(a.act) & 3) == 0;
                unsigned short *const o = static_cast<unsigned short *>(a.act) + static_cast<size_t>(pass.y) * a.n_out + n;
#pragma unroll 1
                for (int t = warp; t < pass.z; t += kEpiWarps) {
                    const uint32_t *const from = reinterpret_cast<const uint32_t *>(staged + t * (kRows * 2)) + lane;
                    const uint32_t v = silu_mul(from[0], from[32]);
                    unsigned short *const p = o + static_cast<size_t>(t) * a.n_out;
                    if (pairs && n < a.n_out) {
                        *reinterpret_cast<uint32_t *>(p) = v;
                    } else {
                        if (n < a.n_out) p[0] = static_cast<unsigned short>(v);
                        if (n + 1 < a.n_out) p[1] = static_cast<unsigned short>(v >> 16);
                    }
                }
            } else {
                const int m = a.two ? lane >> 4 : 0, n = n0 + (a.two ? lane & 15 : lane) * 4;
                const bool vec = (a.n_out & 3) == 0 && (reinterpret_cast<uintptr_t>(a.outs[m]) & 7) == 0;
                unsigned short *const o = static_cast<unsigned short *>(a.outs[m]) + static_cast<size_t>(pass.y) * a.n_out + n;
#pragma unroll 1
                for (int t = warp; t < pass.z; t += kEpiWarps) {
                    const uint2 v = *reinterpret_cast<const uint2 *>(staged + t * (kRows * 2) + lane * 8);
                    unsigned short *const p = o + static_cast<size_t>(t) * a.n_out;
                    if (vec && n < a.n_out) {
                        *reinterpret_cast<uint2 *>(p) = v;
                    } else {
                        if (n < a.n_out) p[0] = static_cast<unsigned short>(v.x);
                        if (n + 1 < a.n_out) p[1] = static_cast<unsigned short>(v.x >> 16);
                        if (n + 2 < a.n_out) p[2] = static_cast<unsigned short>(v.y);
                        if (n + 3 < a.n_out) p[3] = static_cast<unsigned short>(v.y >> 16);
                    }
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (ctl->abort) rest(ctl, nst);
    if (warp == kLoadWarp) {
        tc_fence_after();
        tmem_free_all(tmem);
    }
}

inline size_t up256(size_t v) { return (v + 255) / 256 * 256; }
// 16-bit elements of a prepared row: the activations, then whole blocks of pieces of their sums
int row_elems(int K) { return K + (K / 64 + kSegs - 1) / kSegs * kBlk; }
// Scales and biases of an item as they lie in memory: 128 rows; the ring starts behind two of them.
int item_bytes(int gpr) { return 2 * kRows * gpr * 2; }
int ring_offset(int gpr) { return (kCtlBytes + kOutBytes + 2 * item_bytes(gpr) + 1023) / 1024 * 1024; }
// Three stages have to fit beside the rows of scales.
bool passes_fit(int TB, int gpr) { return ring_offset(gpr) + 3 * (kWordBytes + kChunk * TB * 128) <= kSmemBytes; }
// Rows of a pass at most: 32, 48 or 64 columns are stages of 32, 40 or 48 KB.  Room for nearly all of the experts of an even router, or fewer where
// rows of scales are long: 64 columns fit beside 63 groups, 48 beside 87, 32 beside 111.  0: none do.  (8 experts of 4096 x 1536, groups of 64, where 64
// columns do not fit, 40 / 60 / 300 rows an expert: 74 / 89 / 203 us; the other kernels 130 / 159 / 285 at that time.)
int pass_rows(int m_total, int n_experts, int gpr) {
    const long long rows = m_total, e = n_experts;
    int TB = rows <= 16 * e ? 32 : rows <= 34 * e ? 48 : 64;
    while (TB > 0 && !passes_fit(TB, gpr)) TB = TB > 32 ? TB - 16 : 0;
    return TB;
}

}  // namespace

bool gather_exact_supported(int m_total, int n_out, int K, int n_experts, int bits, int group_size, int dtype, const void *w, const void *scales,
                            const void *biases, const void *x) {
    if (bits != 4 || dtype != MTC_BF16 || (group_size != 64 && group_size != 128)) return false;
    if (m_total <= 0 || n_out <= 0 || K <= 0 || K % group_size != 0 || n_experts <= 0) return false;
    if (static_cast<long long>(n_experts) + m_total / 32 > kMaxPasses) return false;
    if (static_cast<long long>(n_experts) * n_out > 0x7FFF0000ll || static_cast<long long>(m_total) * K > (1ll << 40)) return false;
    const int gpr = K / group_size;
    // scales and biases of an item are copied in one piece
    if (static_cast<long long>(n_out) * gpr % 8 != 0 || gpr > kSmemBytes / (2 * kRows * 4) || pass_rows(m_total, n_experts, gpr) == 0) return false;
    const auto al = [](const void *q, uintptr_t n) { return q == nullptr || reinterpret_cast<uintptr_t>(q) % n == 0; };
    return al(w, 16) && al(x, 16) && al(scales, 16) && al(biases, 16);
}

size_t gather_exact_scratch_bytes(int m_total, int K) {
    return up256(static_cast<size_t>(m_total) * row_elems(K) * 2) + up256(static_cast<size_t>(m_total) * sizeof(float)) + up256(sizeof(ETable));
}

// x rows sorted by expert (expert_offsets [n_experts + 1]) -> mats[i].out [m_total, n_out] for one matrix set, or for two that read the same
// rows (gate and up); with `act`, silu(first) * second goes there instead.  `scratch` holds gather_exact_scratch_bytes(m_total, K) bytes and is used by
// the two launches only (stream order).  row_src: row m of the product reads x[row_src[m]] (x has n_src_rows rows).
cudaError_t launch_gather_exact(Ctx *ctx, cudaStream_t st, const void *x, const uint32_t *row_src, int n_src_rows, const GatherMats *mats, int n_mats,
                                void *act, const uint32_t *expert_offsets, int m_total, int n_out, int K, int n_experts, int group_size, void *scratch,
                                std::string *why) {
    if (n_mats < 1 || n_mats > 2 || (act && n_mats != 2)) return cudaErrorInvalidValue;
    const int elems = row_elems(K), TB = pass_rows(m_total, n_experts, K / group_size);
    unsigned short *xprep = static_cast<unsigned short *>(scratch);
    float *tok_scale = reinterpret_cast<float *>(static_cast<char *>(scratch) + up256(static_cast<size_t>(m_total) * elems * 2));
    ETable *table = reinterpret_cast<ETable *>(reinterpret_cast<char *>(tok_scale) + up256(static_cast<size_t>(m_total) * sizeof(float)));
    const int per = K <= 2048 ? 1 : K <= 4096 ? 2 : K <= 8192 ? 4 : 8;                 // warps per row: eight vectors a lane
    const auto prep = per == 1 ? exact_prep_kernel<1> : per == 2 ? exact_prep_kernel<2> : per == 4 ? exact_prep_kernel<4> : exact_prep_kernel<8>;
    cudaError_t e = launch_pdl(prep, (m_total + 8 / per - 1) / (8 / per) + 1, 256, 0, st, static_cast<const __nv_bfloat16 *>(x), row_src, n_src_rows, expert_offsets,
                               n_experts, m_total, K, elems, TB, xprep, tok_scale, table, ctx->d_status);
    if (e != cudaSuccess) return e;
    EMaps maps;
    for (int i = 0; i < 4; ++i)
        if ((e = make_map_blocks(&maps.x[i], xprep, m_total, elems, 16 * (i + 1), kChunk, why)) != cudaSuccess) return e;
    for (int i = 0; i < 2; ++i)
        if ((e = make_map_2d(&maps.w[i], CU_TENSOR_MAP_DATA_TYPE_UINT32, 4, mats[n_mats == 2 ? i : 0].w, static_cast<long long>(n_experts) * n_out, K / 8, 64, 32,
                             why)) != cudaSuccess) return e;
    EArgs a{};
    for (int i = 0; i < 2; ++i) {
        const GatherMats &m = mats[n_mats == 2 ? i : 0];
        a.scales[i] = m.scales;
        a.biases[i] = m.biases;
        a.outs[i] = m.out;
    }
    for (int i = 0; i < 2; ++i) a.w[i] = static_cast<const uint32_t *>(mats[n_mats == 2 ? i : 0].w);
    a.x = static_cast<const __nv_bfloat16 *>(x);
    a.row_src = row_src;
    a.n_src_rows = n_src_rows;
    a.act = act;
    a.table = table;
    a.tok_scale = tok_scale;
    a.status = ctx->d_status;
    a.two = n_mats == 2;
    a.n_out = n_out;
    a.gpr = K / group_size;
    a.gs_shift = group_size == 64 ? 6 : 7;
    a.tiles = (n_out + (a.two ? 63 : 127)) / (a.two ? 64 : 128);
    a.nkb = K / kBlk;
    a.nlast = (elems - K) / kBlk;
    a.item_bytes = static_cast<uint32_t>(item_bytes(a.gpr));
    a.off_item = kCtlBytes + kOutBytes;
    a.off_ring = static_cast<uint32_t>(ring_offset(a.gpr));
    a.stage = kWordBytes + kChunk * TB * 128;
    a.nst = std::min(kMaxStages, (kSmemBytes - static_cast<int>(a.off_ring)) / static_cast<int>(a.stage));
    constexpr size_t smem = kSmemBytes + 1024;
    static_assert(smem <= 227 * 1024, "shared memory per CTA");
    static PerDeviceAttr attr;
    if ((e = attr.set(gather_exact_kernel, smem)) != cudaSuccess) return e;
    return launch_pdl(gather_exact_kernel, ctx->sm_count, kThreads, smem, st, maps, a);
}

}  // namespace mtc
