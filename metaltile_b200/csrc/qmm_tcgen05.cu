// qmm / gather_qmm — prefill and MoE matmuls on the sm_100a tensor cores.
//
//   dense : out[m, n]  = sum_k x[m, k] * w(n, k)                      (mt_qmm_mma family)
//   gather: out[t, n]  = sum_k x[t, k] * w(E(t), n, k), rows sorted by expert (mt_moe_gather_qmm_*)
//
// Stands in for mt_qmm_mma and its int8/int2/bit-stream variants
// (crates/metaltile-std/src/mlx/quantized.rs:2106-2362,2731,3330,4720-5012) and for the MoE gather
// kernels (crates/metaltile-std/src/ffai/moe.rs:358-605,2256-2835).  Like the reference's MMA kernels
// the weight tile is dequantised to the activation type on chip and fed to the matrix unit with f32
// accumulation (quantized.rs:2245-2252); unlike them neither M nor the rows of an expert need padding.
//
// The product is computed transposed: D^T[n, t] = W_tile[128 x K] * X_chunk[TN x K]^T, so the
// dequantised weights are the A operand (always a full 128-row MMA, however few tokens there are) and
// the activations are the B operand (TN = 16..256 token rows, straight from TMA).
//
// One persistent CTA per SM, 640 threads, warp-specialised:
//   warp 0      producer   one lane issues TMA (cp.async.bulk.tensor, 128B swizzle) loads of the X
//                          chunk [TN x 64] into a shared-memory ring (one or two k blocks a stage)
//   warp 1      MMA        one lane issues tcgen05.mma (M=128, N=TN, K=16, kind::f16), A and the accumulators in TMEM, two
//                          accumulators in turn where they leave A four k blocks
//   warps 2-3   copies     packed words a super-block of 4 k blocks at a time (4 and 8 bits: one TMA box), scales and biases 64 bytes
//                          of a row at a time; warp 2 also allocates and frees the TMEM
//   warps 4-7   epilogue   tcgen05.ld of the finished accumulator, f32 -> T, transposed through shared memory, 256-byte
//                          rows to out (K slices: f32 partial sums)
//   warps 8-19  dequant    three teams of 128 weight rows, every third stage: codes out of the raw buffers (straight from global memory where a
//                          shape has no raw form), w = q*scale + bias rounded to the operand type, tcgen05.st as the A operand
// Stage hand-off uses mbarriers; tcgen05.commit releases a stage when its MMAs have read it.  Every
// wait is bounded: on expiry the kernel records a code in the context's status word, all roles leave
// their loops, copies and MMAs in flight are awaited (bounded too), TMEM is released and the kernel returns.
//
// Why A lies in tensor memory: shared memory moves 128 bytes a cycle, and a k block with A there costs it 16 KB stored and 16 KB read by each chunk's
// MMAs beside the 2 x 128 TN of X: 128 + TN cycles for the MMAs alone (measured), 2.9 cycles a token row in all at 2 x 256 rows where the tensor
// cores need 2.  With A in tensor memory X and the packed words are all there is: 2 TN cycles, as the tensor cores.  What bounds it: at 240 and 256
// rows the tensor cores at the clocks that the power leaves (2048 x 4096 x 4096, 4-bit 76 -> 67 us with the conversion of x), below some 200 rows the
// instructions of the dequant warps (256 x 4096 x 4096 23.2 -> 15.5 us, 8-bit 333 x 7616 x 2880 36 -> 22); 3200 other products 0.87
// to 2.1 times as fast, 1.25 in the mean, eleven of them below 0.97.
//
// Work items (weight-row tile, expert, first token row, token count) are enumerated arithmetically
// for the dense case and read from a list in scratch memory for the gather case; that list is built
// on the device from expert_offsets by build_items_kernel.
#include <cstddef>

#include "ring.cuh"
#include "tcgen05.cuh"

namespace mtc {
namespace {

constexpr int BMW = 128;         // weight rows per tile (TMEM lanes, MMA M)
constexpr int BK = 64;           // k per stage: 64 x 16-bit = one 128B swizzle row
constexpr int TN_MAX = 256;      // token rows per tile (TMEM columns of one accumulator, MMA N)
constexpr int MAX_STAGES = 8;    // ring depth: as many stages as fit in RING_BYTES and in the columns of A, at most this
constexpr int RING_BYTES = 216 * 1024;      // stages of the ring, the raw buffers, the scales
constexpr int EPI_TOK = 16;                 // token rows of one epilogue block: 128 outputs each, two buffers; SmemCtrl follows
constexpr int EPI_PITCH = BMW * 2 + 16;     // bytes of a row: eight consecutive rows start on different banks
constexpr int EPI_BYTES = 2 * EPI_TOK * EPI_PITCH;
constexpr int SB_PER_RAW = 4;               // k blocks per super-block, what K slices are whole multiples of
constexpr int MAX_RAW = 4;
constexpr int TMEM_COLS = 512, A_COLS = BK / 2;     // columns of A per k block
constexpr int TEAMS = 3;                    // of dequant warps
constexpr int EPI_WARP0 = 4;
constexpr int COPY_WARP0 = 2, COPY_THREADS = ring::kCopyWarps * 32;
constexpr int DEQ_WARP0 = 8, DEQ_WARPS = 4 * TEAMS;
constexpr int NUM_THREADS = (DEQ_WARP0 + DEQ_WARPS) * 32;
struct QmmParams {
    const uint32_t *w;
    const void *scales, *biases;
    void *out;
    void *outs[8];               // destinations of the result block (outs[0] == out); further ones may be peers' memory
    int n_outs;
    long long out_ld;            // elements between consecutive token rows of a destination (N, or the width of a wider matrix)
    uint32_t *status;
    const int4 *items;           // gather: {n_tile, expert, row_start, row_count}; dense: nullptr
    const int *item_count;       // gather: device counter; dense: nullptr
    int dense_items;             // dense: number of items = n_tiles * m_chunks
    int m_chunks;                // dense: token chunks per weight-row tile
    int M;                       // dense: rows of x; gather: total rows of x
    int N, K, gs_shift;          // N: weight rows per expert (output columns)
    int op_f16;                  // MMA operand format: 1 = f16, 0 = bf16 (dequantised W and the X tensor map)
    int sb_dt;                   // element type of scales / biases (MTC_F16 or MTC_BF16)
    int out_dt;                  // element type of out
    int out_vec;                 // 1: eight outputs of a row are one aligned 16-byte store (N, out_ld and the pointers allow it)
    const float *tok_scale;      // per-token power-of-two factor applied in the epilogue, or nullptr
    int wpr, gpr;                // words / groups per weight row
    int TN;                      // token rows per item (TMA box rows, MMA N)
    int nst;                     // ring depth
    int kps;                     // k blocks per stage: 1 or 2 (one chunk of few token rows)
    uint32_t hint_ns;            // base suspend-time hint of the waits (0: plain polling)
    int raw;                     // 1: packed words reach the dequant warps through shared memory (cp.async, whole lines)
    uint32_t raw_off, raw_tile;  // byte offset of the raw buffers in shared memory; bytes of one buffer
    int nraw, raw_blk;           // raw: number of buffers; k blocks of one (4; 2 at 8 bits beside two chunks, so that the ring keeps two stages)
    int raw8;                    // raw: 1 = rows of packed words start on 8-byte boundaries only (3 / 5 bits, K an odd multiple of 64)
    // raw: scales (and biases) of the tile, a span of sp_kb k blocks (sp_bytes of a row) at a time, two buffers.  Spans begin at multiples of sp_kb, and with
    // a K slice
    int sp_kb, sp_bytes;
    int sp_copy;                 // 2: TMA boxes (rows are whole 16-byte pieces); 1: 16-byte copies from the boundary below a row's first one on; 0: the
                                 //    arrays start on 4-byte boundaries only, words
    uint32_t sp_off;             // byte offset of the buffers
    long long sb_total;          // elements of the scale (and bias) array
    int wide_items;              // wide: items [0, wide_items) cover two token chunks, each later pair of items one such unit
    int wide;                    // 1: a dense item covers up to 2 TN token rows: one dequantised W stage meets two X chunks, both
                                 //    accumulators belong to the item (the dequant work per flop halves; no epilogue overlap)
    int nacc;                    // accumulators that items take in turn: 2, or 1 (wide: one pair)
    uint32_t a_col0;             // first column of A, behind the accumulators
    int n_tiles;                 // dense: weight-row tiles
    int ksplit;                  // dense: K slices per (weight-row tile, token rows) unit, each an item of its own; 1 = none
    float *partial;              // ksplit > 1: f32 partial sums [ksplit][M][N], added by ksplit_sum_kernel
    int cluster;                 // 1: the slices of a unit are the CTAs of a cluster (an item each) and add up through distributed shared memory
    int pdl_roles;               // programmatic dependent launch: 1 = only the roles that touch what an earlier kernel of the
                                 //    stream may have written (producer: x; epilogue: token factors, out) wait for it, the
                                 //    dequant warps start on the weights at once; 0 = every thread waits first
    uint32_t idesc;
};

struct QmmMaps {
    CUtensorMap x, w, scales, biases;     // the last three only where they travel by TMA
};

struct __align__(8) SmemCtrl {
    uint64_t full[MAX_STAGES];   // the X stage has landed (TMA transaction bytes) and the dequant warps finished the W stage
    uint64_t empty[MAX_STAGES];  // MMAs that read the stage have completed
    uint64_t acc_full[2];        // accumulator buffer complete
    uint64_t acc_empty[2];       // epilogue drained the accumulator buffer
    uint64_t raw_full[MAX_RAW];  // the copies of a raw super-block have landed
    uint64_t raw_empty[MAX_RAW]; // every dequant warp has read it
    uint64_t sp_full[2], sp_empty[2];   // the same for a span of scales
    uint32_t tmem_base;
    volatile uint32_t abort;
    uint64_t drained;                   // giving up: the MMAs are complete
    uint32_t stages_issued, raw_issued, sp_issued, converted[DEQ_WARPS];      // what was started; stages that a dequant warp which gave up has converted
};

// ---- PTX wrappers -------------------------------------------------------------------------------
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
// 32 TMEM lanes x 16 columns in the layout of an MMA accumulator: thread t holds, for the 8 lanes of block k (0..3) and the 8
// columns of half g, lane t / 4 and columns 2 (t % 4), 2 (t % 4) + 1: v[k >> 1][4 g + 2 (k & 1)], + 1.
__device__ __forceinline__ void tmem_ld_frag(uint32_t taddr, uint32_t (&v)[2][8]) {
#pragma unroll
    for (int i = 0; i < 2; ++i)
        asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                     : "=r"(v[i][0]), "=r"(v[i][1]), "=r"(v[i][2]), "=r"(v[i][3]), "=r"(v[i][4]), "=r"(v[i][5]), "=r"(v[i][6]), "=r"(v[i][7])
                     : "r"(taddr + (static_cast<uint32_t>(16 * i) << 16)));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t pack_out(float lo, float hi, bool f16) {
    uint32_t r;
    if (f16) asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    else asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}
// four 8 x 8 blocks, each stored transposed: lane i gives the address of row i % 8 of block i / 8
__device__ __forceinline__ void stmatrix_x4_trans(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

__device__ __forceinline__ uint32_t pack_f16x2(float lo, float hi) {
    uint32_t r;
    asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));   // first source -> upper half
    return r;
}
// (win & mask) | 1.0f in one LOP3: the constant 1.0f sits in a register, the mask is an immediate
__device__ __forceinline__ float code_plus_one(uint32_t win, uint32_t mask, uint32_t one) {
    uint32_t r;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(r) : "r"(win), "r"(mask), "r"(one));
    return __uint_as_float(r);
}
__device__ __forceinline__ void cp_async_16(uint32_t dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
// the first `n` bytes of 16, zeros behind them
__device__ __forceinline__ void cp_async_16_of(uint32_t dst, const void *src, uint32_t n) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}
template <int BYTES>
__device__ __forceinline__ void cp_async_small(uint32_t dst, const void *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(dst), "l"(src), "n"(BYTES) : "memory");
}
// BITS consecutive words from shared memory, with the widest loads the 4*BITS-byte pieces are aligned for
template <int BITS>
__device__ __forceinline__ void lds_words(uint32_t addr, uint32_t (&w)[BITS]) {
    if constexpr (BITS % 4 == 0) {
#pragma unroll
        for (int i = 0; i < BITS / 4; ++i)
            asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(w[4 * i]), "=r"(w[4 * i + 1]), "=r"(w[4 * i + 2]), "=r"(w[4 * i + 3]) : "r"(addr + 16 * i));
    } else if constexpr (BITS % 2 == 0) {
#pragma unroll
        for (int i = 0; i < BITS / 2; ++i)
            asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(w[2 * i]), "=r"(w[2 * i + 1]) : "r"(addr + 8 * i));
    } else {
#pragma unroll
        for (int i = 0; i < BITS; ++i) asm volatile("ld.shared.u32 %0, [%1];" : "=r"(w[i]) : "r"(addr + 4 * i));
    }
}

// ---- dequantisation: windows of codes that a f32 fraction holds, for the general form ----------------
template <int BITS>
struct QPack {
    static constexpr int CPW = 23 / BITS;       // codes per window: a window must fit the 23 mantissa bits
    static constexpr uint32_t MASK = (1u << BITS) - 1u;
};

// 32 codes (BITS words) of one weight row, straight from global memory
template <int BITS>
__device__ __forceinline__ void load_half_words(const uint32_t *p, uint32_t (&w)[BITS], bool valid) {
    if (!valid) {
#pragma unroll
        for (int i = 0; i < BITS; ++i) w[i] = 0u;
        return;
    }
    if constexpr (BITS % 4 == 0) {          // 4-, 8-bit: 16-byte pieces
#pragma unroll
        for (int i = 0; i < BITS / 4; ++i) {
            const uint4 v = __ldg(reinterpret_cast<const uint4 *>(p) + i);
            w[4 * i] = v.x; w[4 * i + 1] = v.y; w[4 * i + 2] = v.z; w[4 * i + 3] = v.w;
        }
    } else if constexpr (BITS % 2 == 0) {   // 2-, 6-bit: 8-byte pieces
#pragma unroll
        for (int i = 0; i < BITS / 2; ++i) {
            const uint2 v = __ldg(reinterpret_cast<const uint2 *>(p) + i);
            w[2 * i] = v.x; w[2 * i + 1] = v.y;
        }
    } else {                                // 3-, 5-bit: single words
#pragma unroll
        for (int i = 0; i < BITS; ++i) w[i] = __ldg(p + i);
    }
}

__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
    uint32_t r;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
    return r;
}
// 32 codes of a row -> 16 registers of two operands each, in the order of K: the general form, by way of f32
template <int BITS>
__device__ __forceinline__ void dequant_half(const uint32_t (&w)[BITS], float s, float b, uint32_t *v) {
    using Q = QPack<BITS>;
    // a code at bit p of a window becomes q * 2^(p-23) after the magic subtract: fold 2^(23-p) into the scale
    float sp[Q::CPW];
#pragma unroll
    for (int c = 0; c < Q::CPW; ++c) sp[c] = s * __uint_as_float(static_cast<uint32_t>(23 - c * BITS + 127) << 23);
    uint32_t one = 0x3F800000u;
    asm volatile("" : "+r"(one));            // keep 1.0f in a register so the extraction is a single LOP3
    float even = 0.0f;
#pragma unroll
    for (int i = 0; i < 32; ++i) {
        const int wi = i / Q::CPW, c = i % Q::CPW;
        const int sbit = wi * Q::CPW * BITS, word = sbit / 32, sh = sbit % 32;
        uint32_t win;
        if (sh == 0) win = w[word];
        else if (word + 1 < BITS) win = __funnelshift_r(w[word], w[word + 1], sh);
        else win = w[word] >> sh;
        const float r = fmaf(code_plus_one(win, Q::MASK << (c * BITS), one) - 1.0f, sp[c], b);
        if (i & 1) v[i >> 1] = pack_f16x2(even, r);
        else even = r;
    }
}
// A k block of a row, 64 codes (words(h, w): those of half h) with one scale (ONE: groups of 64 and more) or two, in packed halves with no conversion: a 16-bit float with exponent
// field 0 is linear in its low bits, so a code at bit P of its half is q * 2^(P - 24), and fma(that, scale * 2^(24 - P), bias) is
// round_f16(q * scale + bias), the value the general form rounds to (4 and 8 bits: with the bias an f16 of its own first).  4-bit codes get there by bytes (bit 7 is 0 where the nibble
// is at bits 3..6, so the sign-replicating form of the byte permute fills the upper byte with zeros): 12 instructions per eight codes; 8-bit ones by a
// byte permute, 8; others by two shifts and two masks a pair, 20 to 22 (32 by way of f32).
// That takes scales up to 65472 / 2^(24 - P): 0.031 (4 bits), 0.0039 (8 bits).  Where a row of the warp has larger ones, its codes become 1024 + q * 2^P by
// an OR of the exponent, an exact subtraction takes the 1024 away, and the factor is scale * 2^-P, one instruction a pair more; a warp whose scales are too far apart for
// either form takes the general one.  The choice is the warp's: lanes that go different ways take the time of both.
template <int BITS, bool ONE, typename Get>
__device__ __forceinline__ void dequant_block(Get words, float s0, float b0, float s1, float b1, uint32_t (&v)[32]) {
    // where a code lies in its half of a register: bit 3 (4 bits), 0 (8 bits), at the top of the ten bits of a fraction (others)
    constexpr int P = BITS == 4 ? 3 : BITS == 8 ? 0 : 10 - BITS;
    constexpr float kUp = static_cast<float>(1 << (24 - P)), kMost = 65472.0f / kUp, kDown = 1.0f / (1 << P);
    auto f16_holds = [](float f) { return __half2float(__float2half_rn(f)) == f; };
    // a bias that is no f16 (a bf16 below 2^-17) would be rounded by itself first
    auto fits = [&](float b) { return BITS == 4 || BITS == 8 ? fabsf(b) <= 65504.0f : f16_holds(b); };
    auto packed = [&](auto form) {
        constexpr bool LARGE = decltype(form)::value;
        constexpr float kFactor = LARGE ? kDown : kUp;
        __half2 s2 = __float2half2_rn(s0 * kFactor), b2 = __float2half2_rn(b0);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            if (!ONE && h == 1) {
                s2 = __float2half2_rn(s1 * kFactor);
                b2 = __float2half2_rn(b1);
            }
            uint32_t w[BITS];
            words(h, w);
            const uint32_t s = *reinterpret_cast<const uint32_t *>(&s2), b = *reinterpret_cast<const uint32_t *>(&b2);
            auto put = [&](int i, uint32_t q) {          // LARGE: 1024 + q * 2^P
                if (LARGE) asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(q) : "r"(q), "r"(0x64006400u));
                asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(v[16 * h + i]) : "r"(q), "r"(s), "r"(b));
            };
            [[maybe_unused]] constexpr uint32_t kOne = LARGE ? 0x64006400u : 0u, kTop = LARGE ? 0x64646464u : 0u;
            if constexpr (BITS == 4) {
#pragma unroll
                for (int i = 0; i < 4; ++i) {    // byte j of lo / hi: code 2j / 2j+1 at bits 3..6
                    const uint32_t lo = (w[i] << 3) & 0x78787878u, hi = (w[i] >> 1) & 0x78787878u;
#pragma unroll
                    for (int j = 0; j < 4; ++j) put(4 * i + j, prmt(lo, hi, ((0xC + j) << 12) | ((4 + j) << 8) | ((8 + j) << 4) | j) | kOne);
                }
            } else if constexpr (BITS == 8) {
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    put(2 * i, prmt(w[i], kTop, 0x4140));
                    put(2 * i + 1, prmt(w[i], kTop, 0x4342));
                }
            } else {
                constexpr uint32_t kLow = ((1u << BITS) - 1u) << P, kHigh = kLow << 16;
#pragma unroll
                for (int i = 0; i < 16; ++i) {   // codes 2i, 2i+1: bits 2i * BITS and on
                    const int at = 2 * i * BITS, word = at / 32;
                    int sh = at % 32;
                    uint32_t t = w[word];
                    if (sh + 2 * BITS > 32) {
                        t = __funnelshift_r(t, w[word + 1 < BITS ? word + 1 : word], sh);
                        sh = 0;
                    }
                    const int up0 = P - sh, up1 = 16 + P - sh - BITS;
                    const uint32_t lo = up0 >= 0 ? t << (up0 & 31) : t >> (-up0 & 31), hi = up1 >= 0 ? t << (up1 & 31) : t >> (-up1 & 31);
                    put(i, ((lo & kLow) | kOne) | (hi & kHigh));
                }
            }
        }
    };
    const bool small = fabsf(s0) <= kMost && fits(b0) && (ONE || (fabsf(s1) <= kMost && fits(b1)));
    if (__all_sync(0xffffffffu, small)) {
        packed(std::false_type{});
    } else if (__all_sync(0xffffffffu, f16_holds(s0 * kDown) && fits(b0) && (ONE || (f16_holds(s1 * kDown) && fits(b1))))) {
        packed(std::true_type{});
    } else {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            uint32_t w[BITS];
            words(h, w);
            dequant_half<BITS>(w, ONE || h == 0 ? s0 : s1, ONE || h == 0 ? b0 : b1, v + 16 * h);
        }
    }
}
__device__ __forceinline__ float sb_value(uint32_t bits, int dt) {
    return dt == MTC_F16 ? __half2float(__ushort_as_half(static_cast<unsigned short>(bits))) : __uint_as_float(bits << 16);
}
__device__ __forceinline__ uint32_t lds_u16(uint32_t addr) {
    unsigned short v;
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(addr));
    return v;
}

// The packed words of some k blocks of a weight tile as they lie in a raw buffer.
// 4 and 8 bits: TMA boxes of 128 bytes x 128 rows with the 128-byte swizzle; other widths: rows padded by 16 bytes.
template <int BITS>
struct RawTile {
    static constexpr bool TMA = BITS == 4 || BITS == 8;
    static constexpr int BLK_BYTES = 8 * BITS, PITCH = SB_PER_RAW * BLK_BYTES + 16;
    // the 32 codes of k block j, half h of row r
    static __device__ __forceinline__ void read(uint32_t base, int r, int j, int h, uint32_t (&w)[BITS]) {
        if constexpr (TMA) {
#pragma unroll
            for (int q = 0; q < BITS / 4; ++q) {
                const int c = (2 * j + h) * (BITS / 4) + q;          // 16-byte chunk of the row
                const uint32_t a = base + (c >> 3) * (BMW * 128) + r * 128 + (((c & 7) ^ (r & 7)) << 4);
                asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(w[4 * q]), "=r"(w[4 * q + 1]), "=r"(w[4 * q + 2]), "=r"(w[4 * q + 3]) : "r"(a));
            }
        } else {
            lds_words<BITS>(base + r * PITCH + (2 * j + h) * (4 * BITS), w);
        }
    }
};
int raw_bytes(int bits, int blocks) { return BMW * (8 * bits * blocks + (bits == 4 || bits == 8 ? 0 : 16)); }
// Rows of a span lie 16 bytes further apart than they are long: eight of them start on different banks, and words that cover them fit
__host__ __device__ constexpr int sp_pitch(int sp_bytes) { return sp_bytes + 16; }
__host__ __device__ constexpr int sp_buffer(int sp_bytes) { return 2 * BMW * sp_pitch(sp_bytes); }

// up to eight 16-bit outputs one by one
__device__ __noinline__ void store_row8(char *o, uint4 v, int n) {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int e = 0; e < 8; ++e)
        if (e < n) reinterpret_cast<unsigned short *>(o)[e] = static_cast<unsigned short>(w[e >> 1] >> (16 * (e & 1)));
}

// The epilogue warps' vote: true when all 128 threads say so (named barrier 1, which their blocks of rows use too)
__device__ __forceinline__ bool epilogue_agrees(bool ok) {
    uint32_t all;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.and.pred q, 1, 128, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
                 : "=r"(all) : "r"(static_cast<uint32_t>(ok)) : "memory");
    return all != 0;
}

struct Item {
    int n_tile, expert, row0, rows;
    int nc;                                 // token chunks of TN rows covered (1 or 2): one accumulator each
    int kb0, nkb, ks;                       // first k block, k blocks and index of the K slice (0, all, 0 unless the launch splits K)
};

template <bool KSPLIT>
__device__ __forceinline__ Item get_item(const QmmParams &p, int i) {
    Item it;
    it.kb0 = 0;
    it.nkb = p.K / BK;
    it.ks = 0;
    if (KSPLIT) {
        // K slices of a (tile, token rows) unit are adjacent items: whole super-blocks, as even as they come
        const int u = i / p.ksplit, unit = u / p.m_chunks, span = p.wide ? 2 * p.TN : p.TN;
        it.n_tile = unit;
        it.ks = i - u * p.ksplit;
        const int nsb = (it.nkb + SB_PER_RAW - 1) / SB_PER_RAW;
        const int sb0 = it.ks * nsb / p.ksplit, sb1 = (it.ks + 1) * nsb / p.ksplit;
        it.kb0 = sb0 * SB_PER_RAW;
        it.nkb = min(sb1 * SB_PER_RAW, it.nkb) - it.kb0;
        it.expert = 0;
        it.row0 = (u - unit * p.m_chunks) * span;
        it.rows = min(span, p.M - it.row0);
        it.nc = it.rows > p.TN ? 2 : 1;
        return it;
    }
    if (p.items) {
        const int4 v = p.items[i];               // written by the kernel before this one: no read-only load
        it.n_tile = v.x; it.expert = v.y & 0xFFFFFF; it.row0 = v.z; it.rows = v.w;
        it.nc = 1;
    } else if (p.wide) {
        // dense, wide: m_chunks items of up to 2 TN token rows per weight-row tile, adjacent so that CTAs running at
        // the same time share the tile's packed words in L2
        // the wide items that do not fill a whole round of the grid (items >= wide_items) run as two single-chunk
        // items each, so that the last round is a short one
        const int u = i < p.wide_items ? i : p.wide_items + ((i - p.wide_items) >> 1);
        const int half = i < p.wide_items ? 0 : ((i - p.wide_items) & 1);
        const int unit = u / p.m_chunks, chunk = u - unit * p.m_chunks;
        it.expert = 0;
        it.n_tile = unit;
        it.row0 = chunk * 2 * p.TN + half * p.TN;
        it.rows = i < p.wide_items ? min(2 * p.TN, p.M - it.row0) : min(p.TN, p.M - it.row0);
        it.nc = it.rows > p.TN ? 2 : 1;
    } else {
        // dense: the token chunks of one weight-row tile are adjacent, so CTAs running at the same time share its
        // packed words in L2
        const int unit = i / p.m_chunks, chunk = i - unit * p.m_chunks;
        it.nc = 1;
        it.expert = 0;
        it.n_tile = unit;
        it.row0 = chunk * p.TN;
        it.rows = min(p.TN, p.M - it.row0);
    }
    return it;
}

// A launch that gave up, once every role has ended: lets what is on its way arrive before the CTA tears down.
__device__ __noinline__ void rest(SmemCtrl *ctl, int nst, int nraw) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (warp >= DEQ_WARP0 && lane == 0) {            // the phases that an X copy completes take these arrivals too
        for (uint32_t u = ctl->converted[warp - DEQ_WARP0]; u < ctl->stages_issued; ++u)
            if (ring::owed(u, min(TEAMS, nst), (warp - DEQ_WARP0) >> 2)) mbar_arrive(&ctl->full[u % nst]);
    } else if (warp == 1 && elect_one()) {
        umma_commit(&ctl->drained);
        drain_ring(&ctl->drained, 1, 1);
    } else if (warp == 0 && lane == 0) {
        drain_ring(ctl->full, ctl->stages_issued, nst);
        if (nraw) {
            drain_ring(ctl->raw_full, ctl->raw_issued, nraw);
            drain_ring(ctl->sp_full, ctl->sp_issued, 2);
        }
    }
    __syncthreads();
}

// KSPLIT: the launch cuts K into slices (items carry a first k block, the epilogue writes f32 partial sums); a
// separate instantiation, so that the code of every other launch is what it was without the feature.
template <int BITS, bool KSPLIT, int KPS>
__global__ void __launch_bounds__(NUM_THREADS, 1)
qmm_tcgen05_kernel(const __grid_constant__ QmmMaps maps, const QmmParams p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    const int nst = p.nst;
    const uint32_t x_stage = static_cast<uint32_t>(p.TN) * BK * 2;      // one X chunk; multiple of 2 KB
    const uint32_t x_slot = KPS == 2 || p.wide ? 2 * x_stage : x_stage;  // two X chunks, or one per k block, per stage (KPS is 1 when wide)
    uint8_t *sX = smem;                                  // nst x x_slot: activations (B operand)
    SmemCtrl *ctl = reinterpret_cast<SmemCtrl *>(smem + RING_BYTES + EPI_BYTES);

    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;       // known to be uniform
    const uint32_t x_bytes = static_cast<uint32_t>(p.TN) * BK * 2;

    if (threadIdx.x == 0) {
        for (int s = 0; s < MAX_STAGES; ++s) {
            mbar_init(&ctl->full[s], 1 + 4);
            mbar_init(&ctl->empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&ctl->acc_full[b], 1);
            mbar_init(&ctl->acc_empty[b], 4);
        }
        for (int b = 0; b < MAX_RAW; ++b) {
            mbar_init(&ctl->raw_full[b], ring::fill_arrivals(RawTile<BITS>::TMA));
            mbar_init(&ctl->raw_empty[b], DEQ_WARPS);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&ctl->sp_full[b], ring::fill_arrivals(p.sp_copy == 2));
            mbar_init(&ctl->sp_empty[b], DEQ_WARPS);
        }
        mbar_init(&ctl->drained, 1);
        ctl->abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 2) {
        tmem_alloc_all(&ctl->tmem_base);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, ctl->tmem_base, 0);
    if (!p.pdl_roles) asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;");
    // a list of work items comes from an earlier kernel of the stream (pdl_roles is 0 then): its length after the wait
    const int num_items = p.items ? *p.item_count : p.dense_items;

    if (warp == 0) {
        // ---------------- producer: TMA loads of the X chunk ----------------
        if (lane == 0) {
            int s = 0;
            uint32_t ph = 0, laps = 0;                    // stage and ring-pass parity, advanced without a division
            bool ok = true;
            if (p.pdl_roles) asm volatile("griddepcontrol.wait;" ::: "memory");      // x may come from the previous kernel
            for (int i = blockIdx.x; i < num_items && ok; i += gridDim.x) {
                const Item item = get_item<KSPLIT>(p, i);
                for (int kb = 0; kb < item.nkb; kb += KPS) {
                    if (!(ok = mbar_wait(&ctl->empty[s], ph ^ 1, &ctl->abort, p.status, 0x101, p.hint_ns))) break;
                    const int k0 = ((KSPLIT ? item.kb0 : 0) + kb) * BK;
                    if constexpr (KPS == 2) {
                        const int nb = min(2, item.nkb - kb);                 // k blocks of this stage
                        mbar_expect_tx(&ctl->full[s], x_bytes * nb);
                        for (int c = 0; c < nb; ++c) tma_load_2d(smem_u32(sX) + s * x_slot + c * x_stage, &maps.x, k0 + c * BK, item.row0, &ctl->full[s]);
                    } else {
                        mbar_expect_tx(&ctl->full[s], x_bytes * item.nc);
                        for (int c = 0; c < item.nc; ++c) tma_load_2d(smem_u32(sX) + s * x_slot + c * x_stage, &maps.x, k0, item.row0 + c * p.TN, &ctl->full[s]);
                    }
                    if (++s == nst) {
                        s = 0;
                        ph ^= 1;
                        ++laps;
                    }
                }
            }
            ctl->stages_issued = laps * nst + s;
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer ----------------
        // The whole warp runs the loop so that stage counters, descriptors and accumulator addresses are
        // warp-uniform values; its control flow depends on votes alone; one elected lane issues.  (With operands that are not known to be
        // uniform four MMAs take 190 cycles to issue instead of 60; under `if (lane == 0)` a k block took 1100.)
        uint32_t tile_i = 0;
        int s = 0;
        uint32_t ph = 0;
        bool ok = true;
        const bool leader = elect_one();
        const uint64_t bdesc0 = make_desc_sw128(__shfl_sync(0xffffffffu, smem_u32(sX), 0));
        const uint32_t b_step = x_slot >> 4, c_step = x_stage >> 4;       // descriptor address units per stage, per chunk
        for (int i = blockIdx.x; i < num_items && ok; i += gridDim.x, ++tile_i) {
            const Item item = get_item<KSPLIT>(p, i);
            // items take the accumulators in turn, so that the epilogue overlaps the next one where there are two
            const int buf = p.nacc == 2 ? tile_i & 1 : 0;
            const uint32_t acc_ph = (p.nacc == 2 ? tile_i >> 1 : tile_i) & 1;
            if (!(ok = mbar_wait_vote(&ctl->acc_empty[buf], acc_ph ^ 1, &ctl->abort, p.status, 0x201))) break;
            tc_fence_after();
            const uint32_t tmem_d = tmem_base + buf * p.TN;
            for (int kb = 0; kb < item.nkb; kb += KPS) {
                if (!(ok = mbar_wait_vote(&ctl->full[s], ph, &ctl->abort, p.status, 0x202))) break;
                tc_fence_after();
                if (leader) {
                    const uint64_t bdesc = bdesc0 + static_cast<uint64_t>(s * b_step);
                    const uint32_t ta = tmem_base + p.a_col0 + s * (KPS * A_COLS);
                    if constexpr (KPS == 2) {                    // two k blocks, one accumulator
                        const int nb = min(2, item.nkb - kb);
#pragma unroll
                        for (int c = 0; c < 2; ++c)
                            if (c < nb) {
#pragma unroll
                                for (int k = 0; k < BK / 16; ++k)
                                    umma_f16_ts(tmem_d, ta + c * A_COLS + 8 * k, bdesc + static_cast<uint64_t>(c * c_step + 2 * k), p.idesc, (kb | c | k) ? 1u : 0u);
                            }
                    } else {
                        for (int c = 0; c < item.nc; ++c) {      // token chunk c accumulates in accumulator c
#pragma unroll
                            for (int k = 0; k < BK / 16; ++k)   // 16 elements = 32 bytes further along the swizzled row
                                umma_f16_ts(tmem_d + c * p.TN, ta + 8 * k, bdesc + static_cast<uint64_t>(c * c_step + 2 * k), p.idesc, (kb | k) ? 1u : 0u);
                        }
                    }
                    umma_commit(&ctl->empty[s]);         // frees the stage when these MMAs have read it
                }
                __syncwarp();
                if (++s == nst) {
                    s = 0;
                    ph ^= 1;
                }
            }
            if (ok && leader) umma_commit(&ctl->acc_full[buf]);
            __syncwarp();
        }
    } else if (warp >= COPY_WARP0 && warp < COPY_WARP0 + COPY_THREADS / 32) {
        // ---------------- copies: packed words, scales -> shared memory ----------------
        // Words: a super-block of 4 k blocks of the tile at a time, up to nraw ahead of the dequant warps and across items.  4- and
        // 8-bit words are one or two TMA boxes (128 bytes x 128 rows, swizzled so that the rows' reads do not conflict);
        // other widths are cp.async copies of these two warps.
        // Scales and biases: rows lie apart, and a cp.async takes the load pipe some ten cycles a lane, so 64 bytes of a row are copied at a time, and where rows are
        // whole 16-byte pieces by TMA.  (A bulk copy a row was slower than eight lanes: 333 x 7616 x 2880 28 -> 40 us.)
        // A warp waits only for buffers that it helps to fill (ring.cuh): what TMA copies is the first warp's alone.
        using R = RawTile<BITS>;
        const bool words_here = ring::fills(R::TMA, warp - COPY_WARP0), scales_here = ring::fills(p.sp_copy == 2, warp - COPY_WARP0);
        if (p.raw && (words_here || scales_here)) {
            const int t = threadIdx.x - COPY_WARP0 * 32;
            const uint32_t raw0 = smem_u32(smem) + p.raw_off, sp0 = smem_u32(smem) + p.sp_off;
            const int pitch = sp_pitch(p.sp_bytes);
            int buf = 0, sp = 0;
            uint32_t ph = 0, sph = 0, laps = 0, spans = 0;
            bool ok = true;
            for (int i = blockIdx.x; i < num_items && ok; i += gridDim.x) {
                const Item im = get_item<KSPLIT>(p, i);
                const int n0 = im.n_tile * BMW;
                const size_t erow = static_cast<size_t>(im.expert) * p.N;
                const int kb_first = KSPLIT ? im.kb0 : 0;
                int sp_next = 0;                         // where the next span starts
                for (int kb0 = 0; kb0 < im.nkb; kb0 += p.raw_blk) {
                    const bool start = kb0 == sp_next;
                    if (start) sp_next += p.sp_kb - (kb_first + kb0) % p.sp_kb;
                    if (start && scales_here) {
                        if (!(ok = mbar_wait_warp(&ctl->sp_empty[sp], sph ^ 1, &ctl->abort, p.status, 0x502, p.hint_ns))) break;
                        const int g0 = ((kb_first + kb0) * BK) >> p.gs_shift, n = ((min(sp_next, im.nkb) - kb0) * BK + (1 << p.gs_shift) - 1) >> p.gs_shift;
                        const uint32_t dst0 = sp0 + sp * sp_buffer(p.sp_bytes), dsts = dst0 + (warp == COPY_WARP0 ? 0 : BMW * pitch);
                        const unsigned short *const arr = static_cast<const unsigned short *>(warp == COPY_WARP0 ? p.scales : p.biases);
                        if (p.sp_copy == 2) {
                            if (t == 0) {                // rows past the array and groups past the row arrive as zeros
                                const int first = g0 & ~(p.sp_bytes / 2 - 1), row = static_cast<int>(erow) + n0;
                                mbar_expect_tx(&ctl->sp_full[sp], 2 * BMW * p.sp_bytes);
                                tma_load_2d(dst0, &maps.scales, first, row, &ctl->sp_full[sp]);
                                tma_load_2d(dst0 + BMW * pitch, &maps.biases, first, row, &ctl->sp_full[sp]);
                            }
                        } else {
                            if (p.sp_copy == 1) {
                                // one warp the scales, the other the biases, eight lanes a row (four: 32 bytes of a row)
                                const unsigned long long b0 = reinterpret_cast<unsigned long long>(arr + (static_cast<size_t>(erow) + n0) * p.gpr + g0);
                                const char *const from = reinterpret_cast<const char *>(b0 & ~15ull);
                                const long long behind = reinterpret_cast<const char *>(arr + p.sb_total) - from;       // to the array's end: nothing past it is read
                                const int left = static_cast<int>(min(behind, 0x7FFFFFFFll)), last = p.N - 1 - n0, low = static_cast<int>(b0 & 15), rb = p.gpr * 2;
                                auto rows = [&](auto lanes) {
                                    constexpr int L = decltype(lanes)::value, STEP = 32 / L;
                                    const int c = (lane % L) * 16;
                                    uint32_t dd = dsts + (lane / L) * pitch + c;
#pragma unroll 4
                                    for (int row = lane / L; row < BMW; row += STEP, dd += STEP * pitch) {
                                        const int at = low + min(row, last) * rb, piece = (at & ~15) + c;       // rows past N copy the last row; never stored
                                        if (piece < at + 2 * n) cp_async_16_of(dd, from + piece, min(16, left - piece));
                                    }
                                };
                                if (p.sp_bytes == 64) rows(std::integral_constant<int, 8>{});
                                else rows(std::integral_constant<int, 4>{});
                            } else {
                                // the words that cover them; the element that ends the array alone in its word is copied by itself
                                for (int row = 0; row < BMW; ++row) {
                                    const size_t el0 = (erow + min(n0 + row, p.N - 1)) * p.gpr + g0;
                                    const long long el = static_cast<long long>(el0 & ~static_cast<size_t>(1)) + 2 * lane;
                                    const uint32_t dd = dsts + row * pitch + lane * 4;
                                    if (lane <= n / 2) {
                                        if (el + 1 < p.sb_total) {
                                            cp_async_small<4>(dd, arr + el);
                                        } else if (el < p.sb_total) {
                                            asm volatile("st.shared.u16 [%0], %1;" ::"r"(dd), "h"(__ldg(arr + el)) : "memory");
                                            __threadfence_block();
                                        }
                                    }
                                }
                            }
                            asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(&ctl->sp_full[sp])) : "memory");
                        }
                        sph ^= sp;
                        sp ^= 1;
                        ++spans;
                    }
                    if (!words_here) continue;
                    if (!(ok = mbar_wait_warp(&ctl->raw_empty[buf], ph ^ 1, &ctl->abort, p.status, 0x501, p.hint_ns))) break;
                    const uint32_t dstt = raw0 + buf * p.raw_tile;
                    if constexpr (R::TMA) {
                        if (t == 0) {
                            mbar_expect_tx(&ctl->raw_full[buf], BMW * R::BLK_BYTES * p.raw_blk);
                            // rows past the array and words past the row arrive as zeros; rows past N are never stored
                            for (int q = 0; q < p.raw_blk * R::BLK_BYTES / 128; ++q)
                                tma_load_2d(dstt + q * (BMW * 128), &maps.w, (kb_first + kb0) * (2 * BITS) + q * 32, static_cast<int>(erow) + n0, &ctl->raw_full[buf]);
                        }
                    } else {
                        const int bytes = min(p.raw_blk, p.K / BK - kb_first - kb0) * (8 * BITS);   // the last one of a row may be short
                        const char *src = reinterpret_cast<const char *>(p.w) + static_cast<size_t>(kb_first + kb0) * (8 * BITS);
                        if (!p.raw8) {
                            constexpr int CPR = 2 * BITS;
#pragma unroll 4
                            for (int ch = t; ch < BMW * CPR; ch += COPY_THREADS) {
                                const int row = ch / CPR, col = ch - row * CPR;
                                const size_t grow = erow + min(n0 + row, p.N - 1);
                                if (col * 16 < bytes) cp_async_16(dstt + row * R::PITCH + col * 16, src + grow * (p.wpr * 4) + col * 16);
                            }
                        } else {
                            constexpr int CPR = 4 * BITS;
#pragma unroll 4
                            for (int ch = t; ch < BMW * CPR; ch += COPY_THREADS) {
                                const int row = ch / CPR, col = ch - row * CPR;
                                const size_t grow = erow + min(n0 + row, p.N - 1);
                                if (col * 8 < bytes) cp_async_small<8>(dstt + row * R::PITCH + col * 8, src + grow * (p.wpr * 4) + col * 8);
                            }
                        }
                        asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(&ctl->raw_full[buf])) : "memory");
                    }
                    if (++buf == p.nraw) {
                        buf = 0;
                        ph ^= 1;
                        ++laps;
                    }
                }
            }
            asm volatile("cp.async.wait_all;" ::: "memory");
            if (t == 0) {          // what TMA copies: the others' copies have landed
                ctl->raw_issued = R::TMA ? laps * p.nraw + buf : 0;
                ctl->sp_issued = p.sp_copy == 2 ? spans : 0;
            }
        }
    } else if (warp >= EPI_WARP0 && warp < EPI_WARP0 + 4) {
        // ---------------- epilogue: TMEM -> registers -> out (transposed) ----------------
        const int q = warp - EPI_WARP0;          // == warp % 4: the TMEM lane quarter this warp may read
        uint32_t epi_buf = 0;
        // what the loop below reads of the parameters, kept in registers: read again for every row the constant bank costs
        // ~200 cycles each time
        uint64_t out0 = reinterpret_cast<uint64_t>(p.outs[0]), ld2 = static_cast<uint64_t>(p.out_ld) * 2, tokp = reinterpret_cast<uint64_t>(p.tok_scale);
        uint32_t more_outs = p.n_outs - 1, out_f16 = p.out_dt == MTC_F16, out_vec = p.out_vec;
        int pN = p.N;
        asm volatile("" : "+l"(out0), "+l"(ld2), "+l"(tokp), "+r"(more_outs), "+r"(out_f16), "+r"(out_vec), "+r"(pN));
        const float *tok_scale = reinterpret_cast<const float *>(tokp);
        const int tok_last = p.M - 1;
        const uint32_t epi0 = smem_u32(smem + RING_BYTES);
        uint32_t tile_i = 0;
        bool ok = true;
        if (p.pdl_roles) asm volatile("griddepcontrol.wait;" ::: "memory");          // token factors; nothing is stored before this
        // slices that add up in a cluster leave the accumulators through all warps, below
        for (int i = KSPLIT && p.cluster ? num_items : blockIdx.x; i < num_items && ok; i += gridDim.x, ++tile_i) {
            const int buf = p.nacc == 2 ? tile_i & 1 : 0;
            const uint32_t acc_ph = (p.nacc == 2 ? tile_i >> 1 : tile_i) & 1;
            const Item item = get_item<KSPLIT>(p, i);
            ok = mbar_wait_warp(&ctl->acc_full[buf], acc_ph, &ctl->abort, p.status, 0x301, p.hint_ns);
            // The four warps share named barriers below, so they give up together: a warp that gave up while another saw the
            // barrier complete would leave that one waiting for good.
            if constexpr (!KSPLIT) ok = epilogue_agrees(ok);
            if (!ok) break;
            tc_fence_after();
            const int n = item.n_tile * BMW + q * 32 + lane;     // output column owned by this thread
            const bool n_ok = n < p.N;
            for (int hh = 0; hh < item.nc; ++hh) {               // accumulators of this item: 1 or 2
                const int c = hh;
                const int row_base = item.row0 + c * p.TN;
                const int rows_h = item.nc == 2 ? min(p.TN, item.rows - c * p.TN) : item.rows;
                if constexpr (KSPLIT) {
                    // a K slice: f32 partial sums, 32 token rows at a time in 128-byte segments per warp and row
                    for (int c0 = 0; c0 < rows_h; c0 += 32) {
                        uint32_t v[32];
                        tmem_ld<32>(tmem_base + (static_cast<uint32_t>(q * 32) << 16) + (buf + hh) * p.TN + c0, v);
                        tmem_wait_ld();
                        if (!n_ok) continue;
                        float *o = p.partial + (static_cast<size_t>(item.ks) * p.M + row_base + c0) * p.N + n;
#pragma unroll
                        for (int j = 0; j < 32; ++j) {
                            if (c0 + j < rows_h) *o = __uint_as_float(v[j]);       // the sum kernel applies the token factors
                            o += p.N;
                        }
                    }
                    continue;
                }
                // 16 token rows at a time through shared memory, transposed on the way ([row][128 outputs]), then whole rows of
                // 256 bytes.  Kept to ~45 instructions a block: the four warps have nobody to hide instruction fetches
                // behind, and a block of 16 conversions and 16 stores a thread took 600 cycles.
                const int n8 = item.n_tile * BMW + (lane & 15) * 8;
                char *row_out = reinterpret_cast<char *>(out0) + static_cast<uint64_t>(row_base + 2 * q + (lane >> 4)) * ld2 + static_cast<uint64_t>(n8) * 2;
                for (int c0 = 0; c0 < rows_h; c0 += EPI_TOK) {
                    float2 ts[2] = {{1.0f, 1.0f}, {1.0f, 1.0f}};       // this lane's token factors
                    if (tok_scale) {
#pragma unroll
                        for (int g = 0; g < 2; ++g) {
                            const int j = row_base + c0 + 8 * g + 2 * (lane & 3);
                            ts[g].x = tok_scale[min(j, tok_last)];
                            ts[g].y = tok_scale[min(j + 1, tok_last)];
                        }
                    }
                    uint32_t v[2][8];
                    tmem_ld_frag(tmem_base + (static_cast<uint32_t>(q * 32) << 16) + (buf + hh) * p.TN + c0, v);
                    const uint32_t sb = epi0 + (epi_buf & 1) * (EPI_TOK * EPI_PITCH);
                    ++epi_buf;
#pragma unroll
                    for (int g = 0; g < 2; ++g) {
                        uint32_t o[4];
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            o[k] = pack_out(__uint_as_float(v[k >> 1][4 * g + 2 * (k & 1)]) * ts[g].x, __uint_as_float(v[k >> 1][4 * g + 2 * (k & 1) + 1]) * ts[g].y, out_f16);
                        stmatrix_x4_trans(sb + (8 * g + (lane & 7)) * EPI_PITCH + q * 64 + (lane >> 3) * 16, o[0], o[1], o[2], o[3]);
                    }
                    asm volatile("bar.sync 1, 128;" ::: "memory");     // the four epilogue warps; two buffers: one barrier a block
#pragma unroll
                    for (int rr = 0; rr < EPI_TOK / 8; ++rr) {          // two rows per warp and step, 16 lanes each
                        const int j = rr * 8 + 2 * q + (lane >> 4);
                        if (c0 + j < rows_h && n8 < pN) {
                            uint4 o4;
                            asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(o4.x), "=r"(o4.y), "=r"(o4.z), "=r"(o4.w) : "r"(sb + j * EPI_PITCH + (lane & 15) * 16));
                            if (out_vec) *reinterpret_cast<uint4 *>(row_out) = o4;
                            else store_row8(row_out, o4, pN - n8);
                            for (uint32_t d = 0; d < more_outs; ++d) {  // the peers' copies of a column block
                                char *o = static_cast<char *>(p.outs[d + 1]) + static_cast<uint64_t>(row_base + c0 + j) * ld2 + static_cast<uint64_t>(n8) * 2;
                                if (out_vec) *reinterpret_cast<uint4 *>(o) = o4;
                                else store_row8(o, o4, pN - n8);
                            }
                        }
                        row_out += 8 * ld2;
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&ctl->acc_empty[buf]);
        }
    } else if (warp >= DEQ_WARP0) {
        // ---------------- dequant: packed W rows -> A operand ----------------
        const int q = warp & 3, team = (warp - DEQ_WARP0) >> 2, r = q * 32 + lane;      // row of the W tile; q: the TMEM lanes this warp may write
        const uint32_t ta0 = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + p.a_col0;
        // A team that comes to a stage has waited for the one that it had before, `teams` stages back: no further back than the ring is deep, or a phase of
        // the barrier two passes old would look like the one it waits for.
        const int teams = min(TEAMS, nst);
        int s = 0, turn = 0;                              // stage, and the team whose stage it is
        uint32_t ph = 0;                                  // ring-pass parity, advanced without a division
        int gave_up = num_items, gave_up_kb = 0;          // item and k block where a wait ran out
        const bool second = p.gs_shift == 5;              // groups of 32: two scales a k block
        auto convert = [&](auto words, uint32_t s0, uint32_t s1, uint32_t b0, uint32_t b1, uint32_t at) {
            uint32_t v[32];
            if (second) dequant_block<BITS, false>(words, sb_value(s0, p.sb_dt), sb_value(b0, p.sb_dt), sb_value(s1, p.sb_dt), sb_value(b1, p.sb_dt), v);
            else dequant_block<BITS, true>(words, sb_value(s0, p.sb_dt), sb_value(b0, p.sb_dt), 0.0f, 0.0f, v);
            tmem_st32(at, v);
        };
        const uint32_t bars = __shfl_sync(0xffffffffu, smem_u32(ctl), 0), abort = bars + offsetof(SmemCtrl, abort);
        auto wait = [&](uint32_t bar, uint32_t parity, uint32_t code) {
            const bool done = mbar_wait(bars + bar, parity, abort, p.status, code);
            __syncwarp();
            return done;
        };
        auto stage_free = [&]() {
            const bool done = wait(offsetof(SmemCtrl, empty) + s * 8, ph ^ 1, 0x401);
            tc_fence_after();
            return done;
        };
        auto stage_done = [&]() {
            tmem_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bars + static_cast<uint32_t>(offsetof(SmemCtrl, full)) + s * 8);
        };
        auto next_stage = [&]() {
            if (++turn == teams) turn = 0;
            if (++s == nst) {
                s = 0;
                ph ^= 1;
            }
        };
        // packed words and scales through the buffers that the copy warps fill
        auto through_buffers = [&]() {
            using R = RawTile<BITS>;
            const int nraw = p.nraw, gsh = p.gs_shift;
            const uint32_t raw0 = smem_u32(smem) + p.raw_off, sp0 = smem_u32(smem) + p.sp_off, bias_off = BMW * sp_pitch(p.sp_bytes);
            // a box's rows are sp_bytes apart, their 16-byte pieces swizzled as TMA does for that width
            const bool by_tma = p.sp_copy == 2;
            const uint32_t piece_of = p.sp_bytes == 64 ? (r >> 1) & 3 : (r >> 2) & 1, in_row = p.sp_bytes - 1;
            int buf = 0;
            uint32_t buf_ph = 0, sp = 0, sph = 0;
            for (int i = blockIdx.x; i < num_items; i += gridDim.x) {
                const Item item = get_item<KSPLIT>(p, i);
                const int kb_first = KSPLIT ? item.kb0 : 0;
                // the row's first scale, modulo 2^32: its place in a buffer, since copies start on boundaries of 16 (or 4) bytes
                const uint32_t el0 = (static_cast<uint32_t>(item.expert) * p.N + min(item.n_tile * BMW + r, p.N - 1)) * p.gpr;
                uint32_t scales = 0;                     // where those of the span lie, less the groups before it
                int sp_next = 0;                         // where the next span starts
                for (int kb0 = 0; kb0 < item.nkb; kb0 += p.raw_blk) {
                    if (kb0 == sp_next) {
                        if (!wait(offsetof(SmemCtrl, sp_full) + sp * 8, sph, 0x403)) {
                            gave_up = i, gave_up_kb = kb0;
                            return;
                        }
                        const uint32_t g = ((kb_first + kb0) * BK) >> gsh, buffer = sp0 + sp * sp_buffer(p.sp_bytes);
                        scales = by_tma ? buffer + r * p.sp_bytes : buffer + r * sp_pitch(p.sp_bytes) + ((el0 + g) & (p.sp_copy ? 7 : 1)) * 2 - 2 * g;
                        sp_next += p.sp_kb - (kb_first + kb0) % p.sp_kb;
                    }
                    if (!wait(offsetof(SmemCtrl, raw_full) + buf * 8, buf_ph, 0x402)) {
                        gave_up = i, gave_up_kb = kb0;
                        return;
                    }
                    const uint32_t base = raw0 + buf * p.raw_tile;
                    const int end = min(p.raw_blk, item.nkb - kb0);
#pragma unroll 1
                    for (int j = 0; j < end; j += KPS) {
                        if (turn == team) {
                            if (!stage_free()) {
                                gave_up = i, gave_up_kb = kb0 + j;
                                return;
                            }
#pragma unroll 1
                            for (int c = 0; c < KPS; ++c) {
                                if (KPS > 1 && j + c >= end) break;
                                const uint32_t at = (((kb_first + kb0 + j + c) * BK) >> gsh) << 1;          // of the row
                                const uint32_t sa = scales + (by_tma ? (at & in_row) ^ (piece_of << 4) : at), sb = sa + bias_off;
                                convert([&](int h, uint32_t (&w)[BITS]) { R::read(base, r, j + c, h, w); }, lds_u16(sa), second ? lds_u16(sa + 2) : 0u, lds_u16(sb), second ? lds_u16(sb + 2) : 0u, ta0 + (s * KPS + c) * A_COLS);
                            }
                            stage_done();
                        }
                        next_stage();
                    }
                    const bool sp_done = kb0 + p.raw_blk == sp_next || kb0 + p.raw_blk >= item.nkb;
                    __syncwarp();
                    if (lane == 0) {
                        mbar_arrive(bars + static_cast<uint32_t>(offsetof(SmemCtrl, raw_empty)) + buf * 8);
                        if (sp_done) mbar_arrive(bars + static_cast<uint32_t>(offsetof(SmemCtrl, sp_empty)) + sp * 8);
                    }
                    if (++buf == nraw) {
                        buf = 0;
                        buf_ph ^= 1;
                    }
                    if (sp_done) {
                        sph ^= sp;
                        sp ^= 1;
                    }
                }
            }
        };
        // straight from global memory
        auto from_memory = [&]() {
            for (int i = blockIdx.x; i < num_items; i += gridDim.x) {
                const Item item = get_item<KSPLIT>(p, i);
                const int n = item.n_tile * BMW + r;
                const bool valid = n < p.N;
                const size_t grow = static_cast<size_t>(item.expert) * p.N + (valid ? n : 0);
                const uint32_t *wrow = p.w + grow * p.wpr;
                const unsigned short *sc16 = static_cast<const unsigned short *>(p.scales) + grow * p.gpr;
                const unsigned short *bi16 = static_cast<const unsigned short *>(p.biases) + grow * p.gpr;
                const int kb0 = KSPLIT ? item.kb0 : 0;
                uint32_t w[2][BITS];
                uint32_t sv[2] = {0, 0}, bv[2] = {0, 0};      // raw 16-bit scales / biases, converted when used
                auto request = [&](int kb) {                  // a k block of this team's, asked for a turn ahead
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        load_half_words<BITS>(wrow + static_cast<size_t>(kb0 + kb) * (2 * BITS) + h * BITS, w[h], valid);
                        const int g = ((kb0 + kb) * BK + h * 32) >> p.gs_shift;
                        sv[h] = valid ? __ldg(sc16 + g) : 0u;
                        bv[h] = valid ? __ldg(bi16 + g) : 0u;
                    }
                };
                const int mine = team >= turn ? team - turn : team - turn + teams;        // this team's first k block of the item
                if (team < teams && mine < item.nkb) request(mine);
                for (int kb = 0; kb < item.nkb; ++kb) {
                    if (turn == team) {
                        if (!stage_free()) {
                            gave_up = i, gave_up_kb = kb;
                            return;
                        }
                        convert([&](int h, uint32_t (&to)[BITS]) {
#pragma unroll
                            for (int e = 0; e < BITS; ++e) to[e] = w[h][e];
                        }, sv[0], sv[1], bv[0], bv[1], ta0 + s * A_COLS);
                        if (kb + teams < item.nkb) request(kb + teams);
                        stage_done();
                    }
                    next_stage();
                }
            }
        };
        if (p.raw) through_buffers();
        else from_memory();
        uint32_t stages = 0xFFFFFFFFu;
        if (gave_up < num_items) {                       // those before that
            stages = gave_up_kb / KPS;
            for (int i = blockIdx.x; i < gave_up; i += gridDim.x) stages += (get_item<KSPLIT>(p, i).nkb + KPS - 1) / KPS;
        }
        if (lane == 0) ctl->converted[warp - DEQ_WARP0] = stages;
    }

    if constexpr (KSPLIT) {
        if (p.cluster) {
            // The sum over the slices in slice order, the token factors, the stores: a CTA takes its share of the blocks of 16 token rows.  The others
            // push theirs of it into its ring, which is free when all MMAs of the cluster are complete: stores to another SM are not waited for, loads
            // from it were 2 us of a product (and sums left to the four epilogue warps 6).  Every role of every CTA comes here, also one that gave up.
            asm volatile("griddepcontrol.wait;" ::: "memory");
            __syncwarp();
            const Item item = get_item<KSPLIT>(p, blockIdx.x);
            const int S = p.ksplit, me = item.ks, blocks = item.nc * p.TN / 16, most = (blocks + S - 1) / S;
            const int first = blocks * me / S, own = blocks * (me + 1) / S - first;
            constexpr uint32_t BLOCK = 16 * BMW * 4;                       // a block of sums: [16 token rows][128 outputs] of f32
            const uint32_t mine = smem_u32(smem) + ((warp & 3) * 32 + lane) * 4, lanes = tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16);
            const bool ok = mbar_wait_warp(&ctl->acc_full[0], 0, &ctl->abort, p.status, 0x302, p.hint_ns);
            tc_fence_after();
            cluster_sync();
            if (ok) {
#pragma unroll 1
                for (int c = warp >> 2; c < blocks; c += NUM_THREADS / 128) {
                    const int to = ((c + 1) * S - 1) / blocks;             // blocks * to / S <= c < blocks * (to + 1) / S
                    if (to == me) continue;
                    uint32_t v[16], a;
                    tmem_ld<16>(lanes + c * 16, v);
                    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(mine + ((me < to ? me : me - 1) * most + c - blocks * to / S) * BLOCK), "r"(to));
                    tmem_wait_ld();
#pragma unroll
                    for (int j = 0; j < 16; ++j) asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(a + j * (BMW * 4)), "r"(v[j]) : "memory");
                }
            }
            cluster_sync();
            if (ok) {
#pragma unroll 1
                for (int c = warp >> 2; c < own; c += NUM_THREADS / 128) {
                    uint32_t v[16];
                    tmem_ld<16>(lanes + (first + c) * 16, v);
                    tmem_wait_ld();
                    float sum[16];
#pragma unroll 1
                    for (int r = 0; r < S; ++r) {
                        const uint32_t a = mine + ((r < me ? r : r - 1) * most + c) * BLOCK;
#pragma unroll
                        for (int j = 0; j < 16; ++j) {
                            float t = __uint_as_float(v[j]);
                            if (r != me) asm volatile("ld.shared.f32 %0, [%1];" : "=f"(t) : "r"(a + j * (BMW * 4)) : "memory");
                            sum[j] = r == 0 ? t : sum[j] + t;
                        }
                    }
#pragma unroll
                    for (int j = 0; j < 16; ++j) asm volatile("st.shared.f32 [%0], %1;" ::"r"(mine + c * BLOCK + j * (BMW * 4)), "f"(sum[j]) : "memory");
                }
            }
            __syncthreads();
            // a warp a row, a lane four outputs
            const int n = item.n_tile * BMW + lane * 4, left = p.N - n;
            for (int j = warp; j < own * 16; j += NUM_THREADS / 32) {
                if (left <= 0 || first * 16 + j >= item.rows) continue;
                float4 v;
                asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(smem_u32(smem) + j * (BMW * 4) + lane * 16) : "memory");
                const int m = item.row0 + first * 16 + j;
                if (p.tok_scale) {
                    const float f = p.tok_scale[m];
                    v.x *= f; v.y *= f; v.z *= f; v.w *= f;
                }
                const uint32_t lo = pack_out(v.x, v.y, p.out_dt == MTC_F16), hi = pack_out(v.z, v.w, p.out_dt == MTC_F16);
                for (int d = 0; d < p.n_outs; ++d) {
                    unsigned short *const o = static_cast<unsigned short *>(p.outs[d]) + static_cast<size_t>(m) * p.out_ld + n;
                    if (left >= 4 && p.out_ld % 4 == 0 && reinterpret_cast<uintptr_t>(p.outs[d]) % 8 == 0) {
                        *reinterpret_cast<uint2 *>(o) = make_uint2(lo, hi);
                    } else {
                        const unsigned short e[4] = {static_cast<unsigned short>(lo), static_cast<unsigned short>(lo >> 16), static_cast<unsigned short>(hi),
                                                     static_cast<unsigned short>(hi >> 16)};
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            if (k < left) o[k] = e[k];
                    }
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (ctl->abort) rest(ctl, nst, p.raw ? p.nraw : 0);
    if (warp == 2) {
        tc_fence_after();
        tmem_free_all(tmem_base);
    }
}

// bf16 activations -> f16 with one power-of-two factor per row.  bf16 keeps 8 significant bits, so
// x * 2^-e is exact in f16 (11 bits) once the row maximum is brought to [2^14, 2^15); elements more than
// 2^31 below the row maximum lose bits (2^-40 of it at most), which changes nothing measurable.  The MMA then runs on f16
// operands, whose 3 extra mantissa bits keep the dequantised weights 8x closer to the f32 oracle than
// bf16 weights would be; the epilogue multiplies the accumulator by 2^e again.
// W warps share a row and hold it in registers between the maximum and the conversion (one read of x instead of two), eight
// 16-byte loads a lane in flight: 2048 x 4096 10.1 -> 5 us, which every bf16 product waits for.  Longer rows are read twice.
template <int W>
__global__ void __launch_bounds__(256) rows_to_f16_kernel(const __nv_bfloat16 *x, __half *y, float *row_scale, int rows, int K) {
    asm volatile("griddepcontrol.launch_dependents;");      // the product kernel may start on the weights meanwhile
    asm volatile("griddepcontrol.wait;" ::: "memory");       // x may come from the previous kernel, which may read the last y
    constexpr int ROWS = 8 / W, HELD = 8, STEP = 32 * W;
    __shared__ uint32_t part[8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int row = blockIdx.x * ROWS + warp / W, i0 = (warp % W) * 32 + lane;
    const bool on = row < rows;
    const int nvec = on ? K / 8 : 0;
    const uint4 *src = reinterpret_cast<const uint4 *>(x + static_cast<size_t>(on ? row : 0) * K);
    uint4 *dst = reinterpret_cast<uint4 *>(y + static_cast<size_t>(on ? row : 0) * K);
    uint4 held[HELD];
#pragma unroll
    for (int q = 0; q < HELD; ++q) held[q] = i0 + q * STEP < nvec ? src[i0 + q * STEP] : make_uint4(0u, 0u, 0u, 0u);
    uint32_t amax = 0;                       // max of |x| as bf16 bit patterns (monotone for finite values)
    auto fold = [&](const uint4 &v) {
        const uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            amax = max(amax, u[j] & 0x7FFFu);
            amax = max(amax, (u[j] >> 16) & 0x7FFFu);
        }
    };
#pragma unroll
    for (int q = 0; q < HELD; ++q) fold(held[q]);
    for (int i = i0 + HELD * STEP; i < nvec; i += STEP) fold(src[i]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) amax = max(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    if constexpr (W > 1) {
        if (lane == 0) part[warp] = amax;
        __syncthreads();
#pragma unroll
        for (int w = 0; w < W; ++w) amax = max(amax, part[warp / W * W + w]);
    }
    const int ex = static_cast<int>(amax >> 7);                    // biased exponent of the row maximum
    int e = (ex == 0 || ex == 0xFF) ? 0 : ex - 127 - 14;           // zero rows and inf/nan rows stay unscaled
    e = max(e, -126);                                              // 2^-e and 2^e must both be normal f32 numbers
    const float down = __uint_as_float(static_cast<uint32_t>(127 - e) << 23);
    if (on && i0 == 0) row_scale[row] = __uint_as_float(static_cast<uint32_t>(127 + e) << 23);
    auto convert = [&](const uint4 &v) {
        const uint32_t u[4] = {v.x, v.y, v.z, v.w};
        uint32_t o[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const __half2 h = __floats2half2_rn(__uint_as_float(u[j] << 16) * down, __uint_as_float(u[j] & 0xFFFF0000u) * down);
            o[j] = *reinterpret_cast<const uint32_t *>(&h);
        }
        return make_uint4(o[0], o[1], o[2], o[3]);
    };
#pragma unroll
    for (int q = 0; q < HELD; ++q)
        if (i0 + q * STEP < nvec) dst[i0 + q * STEP] = convert(held[q]);
    for (int i = i0 + HELD * STEP; i < nvec; i += STEP) dst[i] = convert(src[i]);
}
cudaError_t launch_rows_to_f16(cudaStream_t st, const void *x, __half *y, float *row_scale, int rows, int K) {
    const __nv_bfloat16 *xb = static_cast<const __nv_bfloat16 *>(x);
    const int per = K <= 2048 ? 1 : K <= 4096 ? 2 : K <= 8192 ? 4 : 8;                 // warps per row: eight vectors a lane
    const int grid = (rows + 8 / per - 1) / (8 / per);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(256);
    cfg.stream = st;
    cudaLaunchAttribute la[1];
    la[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    la[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = la;
    cfg.numAttrs = 1;
    const auto kern = per == 1 ? rows_to_f16_kernel<1> : per == 2 ? rows_to_f16_kernel<2> : per == 4 ? rows_to_f16_kernel<4> : rows_to_f16_kernel<8>;
    return cudaLaunchKernelEx(&cfg, kern, xb, y, row_scale, rows, K);
}

// Work list of the gather case, built on the device from the CSR expert_offsets (or, when only the
// per-row expert ids are given, from those: rows are sorted by expert, so offsets[e] is the first
// row whose id is >= e).  Layout of the scratch block: int count; int pad[3]; int4 items[].
// Expert-major order: the token chunks and weight-row tiles of one expert are adjacent, so the
// CTAs working at the same time share that expert's X rows in L2.
// Offsets that reach past total_rows are clamped to it (the rows they would have named do not exist: nothing is read or
// written for them) and reported in the status word, 0x901, like offsets that run backwards (those experts get no rows).
__global__ void build_items_kernel(const uint32_t *expert_offsets, const uint32_t *indices, int total_rows, int n_experts,
                                   int n_tiles, int TN, int *count_out, int4 *items, int max_items, uint32_t *status) {
    extern __shared__ int sh[];          // [n_experts + 1] offsets, then [n_experts + 1] item bases
    int *off = sh, *base = sh + n_experts + 1;
    for (int e = threadIdx.x; e <= n_experts; e += blockDim.x) {
        if (expert_offsets) {
            const uint32_t o = expert_offsets[e];
            if (o > static_cast<uint32_t>(total_rows) || (e > 0 && o < expert_offsets[e - 1])) atomicCAS(status, 0u, 0x901u);
            off[e] = static_cast<int>(min(o, static_cast<uint32_t>(total_rows)));
        } else {                          // lower bound of e in the sorted per-row ids
            int lo = 0, hi = total_rows;
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (indices[mid] < static_cast<uint32_t>(e)) lo = mid + 1; else hi = mid;
            }
            off[e] = lo;
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int acc = 0;
        for (int e = 0; e < n_experts; ++e) {
            base[e] = acc;
            const int rows = max(off[e + 1] - off[e], 0);
            acc += ((rows + TN - 1) / TN) * n_tiles;
        }
        base[n_experts] = acc;
        *count_out = acc < max_items ? acc : max_items;
    }
    __syncthreads();
    for (int e = threadIdx.x; e < n_experts; e += blockDim.x) {
        const int rows = max(off[e + 1] - off[e], 0);
        const int chunks = (rows + TN - 1) / TN;
        int idx = base[e];
        for (int c = 0; c < chunks; ++c)
            for (int nt = 0; nt < n_tiles; ++nt, ++idx)
                if (idx < max_items) items[idx] = make_int4(nt, e, off[e] + c * TN, min(TN, rows - c * TN));
    }
}

// ---- host side ----------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn get_encode_fn() {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void *ptr = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) == cudaSuccess &&
            qres == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(ptr);
    }
    return fn;
}

template <int BITS>
constexpr size_t qmm_smem_bytes() {
    return RING_BYTES + EPI_BYTES + sizeof(SmemCtrl) + 1024;
}

template <int BITS>
cudaError_t launch_bits(cudaStream_t st, const QmmMaps &maps, const QmmParams &p, int grid) {
    constexpr size_t smem = qmm_smem_bytes<BITS>();
    static_assert(smem <= 227 * 1024, "shared memory per CTA");
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(NUM_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute la[2];
    la[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    la[0].val.programmaticStreamSerializationAllowed = 1;
    la[1].id = cudaLaunchAttributeClusterDimension;
    la[1].val.clusterDim.x = p.cluster ? p.ksplit : 1;
    la[1].val.clusterDim.y = 1;
    la[1].val.clusterDim.z = 1;
    cfg.attrs = la;
    cfg.numAttrs = p.cluster ? 2 : 1;
    auto go = [&](auto kern, PerDeviceAttr &attr) {
        cudaError_t e = attr.set(kern, smem);
        return e != cudaSuccess ? e : cudaLaunchKernelEx(&cfg, kern, maps, p);
    };
    static PerDeviceAttr attr[4];
    if (p.kps == 2) return p.ksplit > 1 ? go(qmm_tcgen05_kernel<BITS, true, 2>, attr[0]) : go(qmm_tcgen05_kernel<BITS, false, 2>, attr[1]);
    return p.ksplit > 1 ? go(qmm_tcgen05_kernel<BITS, true, 1>, attr[2]) : go(qmm_tcgen05_kernel<BITS, false, 1>, attr[3]);
}

// X as a 2-D tensor [rows, K] of 16-bit elements, box 64 x TN
cudaError_t make_x_map(CUtensorMap *tmap, const void *x, int rows, int K, int TN, int op_f16, std::string *why) {
    return make_map_2d(tmap, op_f16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, x, rows, K, TN, BK, why);
}

cudaError_t launch_any(int bits, cudaStream_t st, const CUtensorMap &tmap, const QmmParams &p, int grid, long long w_rows, std::string *why) {
    QmmMaps maps{tmap, tmap, tmap, tmap};                // what does not travel by TMA is not read
    cudaError_t e = cudaSuccess;
    // packed words [rows, words], boxes of 128 bytes x 128 rows; scales and biases [rows, groups], of sp_bytes x 128 rows
    if (p.raw && (bits == 4 || bits == 8)) e = make_map_2d(&maps.w, CU_TENSOR_MAP_DATA_TYPE_UINT32, 4, p.w, w_rows, p.wpr, BMW, 32, why);
    if (p.raw && p.sp_copy == 2) {
        if (e == cudaSuccess) e = make_map_2d(&maps.scales, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, p.scales, w_rows, p.gpr, BMW, p.sp_bytes / 2, why);
        if (e == cudaSuccess) e = make_map_2d(&maps.biases, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, p.biases, w_rows, p.gpr, BMW, p.sp_bytes / 2, why);
    }
    if (e != cudaSuccess) return e;
    switch (bits) {
        case 2: return launch_bits<2>(st, maps, p, grid);
        case 3: return launch_bits<3>(st, maps, p, grid);
        case 4: return launch_bits<4>(st, maps, p, grid);
        case 5: return launch_bits<5>(st, maps, p, grid);
        case 6: return launch_bits<6>(st, maps, p, grid);
        default: return launch_bits<8>(st, maps, p, grid);
    }
}

// Accumulators, ring depth, raw buffers and spans of scales for p.TN / p.wide.  The raw path needs groups of 32, 64 or 128 and 4-byte aligned scale / bias
// arrays.  Two accumulators where they leave A four k blocks.  Two k blocks per hand-off up to 128 token rows: waits and arrivals are paid half as
// often.  A third raw buffer and longer spans are taken where the ring keeps four stages beside them, or all that the columns of A hold.
void plan_smem(QmmParams &p, Ctx *ctx, int bits) {
    const auto al = [](const void *ptr, size_t n) { return reinterpret_cast<uintptr_t>(ptr) % n == 0; };
    p.nacc = !p.wide && 2 * p.TN <= TMEM_COLS - 4 * A_COLS ? 2 : 1;
    p.a_col0 = static_cast<uint32_t>((p.wide ? 2 : p.nacc) * p.TN);
    p.raw = ctx->qmm_raw != 0 && p.gs_shift >= 5 && p.gs_shift <= 7 && al(p.scales, 4) && al(p.biases, 4);
    p.raw8 = (p.wpr * 4) % 16 != 0;
    p.raw_blk = bits == 8 && p.wide ? 2 : SB_PER_RAW;
    p.raw_tile = static_cast<uint32_t>(raw_bytes(bits, p.raw_blk));
    p.kps = p.raw && !p.wide && p.TN <= 128 ? 2 : 1;
    const int slot = (p.wide || p.kps == 2 ? 2 : 1) * p.TN * BK * 2;
    int most = (TMEM_COLS - static_cast<int>(p.a_col0)) / (A_COLS * p.kps);
    if (most > MAX_STAGES) most = MAX_STAGES;
    p.nraw = 0;
    p.sp_bytes = 64;
    p.nst = RING_BYTES / slot;
    if (p.raw) {
        // the first form whose ring is deep enough, else the last
        const int fewest = p.raw_blk == 2 ? 3 : 2, want = most < 4 ? most : 4;
        for (p.sp_bytes = 64; ; p.sp_bytes = 32) {
            for (p.nraw = fewest + 1; ; --p.nraw) {
                p.nst = (RING_BYTES - p.nraw * static_cast<int>(p.raw_tile) - 2 * sp_buffer(p.sp_bytes)) / slot;
                if (p.nst >= want || p.nraw == fewest) break;
            }
            if (p.nst >= want || p.sp_bytes == 32) break;
        }
    }
    if (p.nst > most) p.nst = most;
    if (ctx->qmm_max_stages > 0 && p.nst > ctx->qmm_max_stages) p.nst = ctx->qmm_max_stages;
    p.raw_off = static_cast<uint32_t>(p.nst * slot);
    p.sp_off = p.raw_off + p.nraw * p.raw_tile;
    p.sp_kb = ((p.sp_bytes / 2) << p.gs_shift) / BK;
    p.sp_copy = !al(p.scales, 16) || !al(p.biases, 16) ? 0 : p.gpr % 8 == 0 ? 2 : 1;
}

void fill_common(QmmParams &p, Ctx *ctx, const void *w, const void *scales, const void *biases, void *out, int N, int K,
                 int bits, int group_size, int dt, int TN) {
    p.w = static_cast<const uint32_t *>(w);
    p.scales = scales;
    p.biases = biases;
    p.out = out;
    p.outs[0] = out;
    p.n_outs = 1;
    p.out_ld = N;
    p.status = ctx->d_status;
    p.N = N; p.K = K;
    p.sb_dt = dt;
    p.out_dt = dt;
    p.op_f16 = 1;   // bf16 activations are converted to scaled f16 first (see rows_to_f16_kernel)
    p.gs_shift = 0;
    while ((1 << p.gs_shift) < group_size) ++p.gs_shift;
    p.wpr = K * bits / 32;
    p.gpr = K / group_size;
    p.TN = TN;
    p.wide = 0;
    p.ksplit = 1;
    p.sb_total = static_cast<long long>(N) * p.gpr;          // a gather launch multiplies by its experts
    p.partial = nullptr;
    p.pdl_roles = 0;               // the dense launcher turns it on: a gather launch reads a work list the previous kernel built
    plan_smem(p, ctx, bits);
    p.hint_ns = static_cast<uint32_t>(ctx->qmm_wait_hint_ns);
    const uint32_t fmt = p.op_f16 ? 0u : 1u;           // both operands carry the same 16-bit format
    p.idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | (static_cast<uint32_t>(TN >> 3) << 17) |
              (static_cast<uint32_t>(BMW >> 4) << 24);
}

void set_out_vec(QmmParams &p) {
    p.out_vec = p.N % 8 == 0 && p.out_ld % 8 == 0;
    for (int d = 0; d < p.n_outs; ++d) p.out_vec = p.out_vec && reinterpret_cast<uintptr_t>(p.outs[d]) % 16 == 0;
}

// bf16 activations: stage a scaled f16 copy of x in the context's conversion buffer.
cudaError_t stage_x(Ctx *ctx, cudaStream_t st, const void *x, int rows, int K, int dt, const void **x_op,
                    const float **tok_scale, std::string *why) {
    *x_op = x;
    *tok_scale = nullptr;
    if (dt == MTC_F16) return cudaSuccess;
    const size_t need = ((static_cast<size_t>(rows) * K * 2 + 255) & ~static_cast<size_t>(255)) + static_cast<size_t>(rows) * sizeof(float);
    cudaError_t ge = grow_block(ctx, st, &ctx->d_xconv, &ctx->xconv_bytes, need, why);
    if (ge != cudaSuccess) return ge;
    __half *y = static_cast<__half *>(ctx->d_xconv);
    float *scale = reinterpret_cast<float *>(static_cast<char *>(ctx->d_xconv) + ((static_cast<size_t>(rows) * K * 2 + 255) & ~static_cast<size_t>(255)));
    cudaError_t e = launch_rows_to_f16(st, x, y, scale, rows, K);
    if (e != cudaSuccess) return e;
    *x_op = y;
    *tok_scale = scale;
    return cudaSuccess;
}

// Prices of a dense launch's forms, us, fitted together to 62000 launches in the forms that 2900 products of 17 to 2048 rows can take, every width (the one
// taken is 1.025 times as long as the fastest in the mean; with prices fitted to a dozen products it was 1.07, since slices went through memory where clusters
// are faster: 66 x 4224 x 1664 12.0 us, 8.1 in clusters of two; 453 x 384 x 3840 12.8, 9.4 in clusters of three.  One product in fifty became more than 5 %
// slower by the new ones, up to 24 %: 1332 x 320 x 1408 at 5 bits 10.1 us as 14 items, 12.5 in 14 pairs.)
// A k block of an item on one SM by its token rows: up to 128 the hand-offs of two k blocks at a time, then of one, above 192 and with two chunks the tensor
// cores, behind which other widths than 4 and 8 bits hide what more they take a code.  Rows of scales that are no whole 16-byte pieces are copied
// by hand; rows of words that start on 8-byte boundaries only set a pace of their own.
double kb_cost(int TN, bool wide, int K, int bits, bool pieces) {
    const double more = wide || TN > 192 ? 0.0 : bits == 2 ? 0.034 : bits == 3 ? 0.049 : bits == 5 ? 0.095 : bits == 6 ? 0.046 : 0.0;
    const double by_hand = pieces ? 0.0 : wide ? 0.021 : TN <= 128 ? 0.033 : 0.038;
    const double us = wide ? 0.24 + 0.00201 * TN : TN <= 128 ? 0.226 + 0.0007 * TN : TN <= 192 ? 0.349 : 0.349 + 0.00195 * (TN - 192);
    return std::max(us + more + by_hand, K * bits / 8 % 16 != 0 ? 0.116 * bits : 0.0);
}
// a further item on the same SM: its accumulators drain before the next pair starts, or beside it where there are two sets
double item_cost(int TN, bool wide) { return wide ? 0.4 + 0.012 * 2 * TN : TN > 192 ? 0.13 + 0.0106 * TN : 0.13; }
constexpr double kMoreItems = 1.06;     // whole items narrower than cover the rows have to be that much cheaper (1.0: forms 1.0265 times the fastest in the mean, 1.06: 1.0245, 1.1: 1.0258)
// K slices that add up in memory, beside the k blocks of one: the second kernel, for each slice, for each f32 partial sum that is written and read.
constexpr double kSlicedUs = 7.2, kEachSliceUs = 0.054, kSliceUs = 1.52e-6;
// Clusters of one to eight CTAs, one CTA an SM, that are resident at once (cudaOccupancyMaxActiveClusters: the GPCs do not divide evenly)
// (45 of three are, but with all of them at once products of x in bf16 took 1.1 to 1.2 times as long as with 44)
constexpr int kClusters[9] = {0, 148, 74, 44, 33, 26, 22, 15, 15};
// Slices that are the CTAs of a cluster: launch, barriers and sum; for each token row; for the share of such clusters that run, which wait for each other's SMs
// (f16 products follow one another without a conversion of x between them), and steeply for the last tenth of the pairs (414 x 1536 x 1536 in 72 of them 16.1
// us, 13.1 in 48).
double cluster_cost(int S, int rows, long long units, bool f16) {
    const double share = static_cast<double>(units) / kClusters[S];
    return (S <= 4 ? 2.03 : 4.22) + 0.0106 * rows + ((S == 2 ? 0.77 : 2.95) + (f16 ? 1.21 : 0.0)) * share + (S == 2 ? 11.9 * std::max(0.0, share - 0.9) : 0.0);
}

// How a dense launch covers its M token rows: items of one chunk (TN rows, one accumulator) or of two (the dequantised W stage
// is built once for both), chunks of equal width (333 rows are 2 x 176, not 256 + 77), and K slices where the items alone
// would leave SMs idle.  Every form is priced by the rounds of the grid it takes.
struct DensePlan {
    int TN, items_m, ksplit, halves, cluster;      // halves: wide items of an incomplete last round that run as two single-chunk items each
    bool wide;
};
//
// Slices cost a block of the context: at most kSliceBytes of partial sums, so that a rising prompt length cannot pile up outgrown
// blocks without bound (they are kept until the context goes), and so that the sum kernel's 32-bit index holds every output.
// slices = false: the best plan without them, for a caller whose block cannot grow.
constexpr size_t kSliceBytes = size_t{512} << 20;
// options "qmm_ksplit" and "qmm_wide"; form 1: items of two chunks
bool slices_allowed(const Ctx *ctx, int M, int form) {
    return ctx->qmm_ksplit && (ctx->qmm_wide == 1 || M <= TN_MAX) && (form == 0 || (ctx->qmm_wide && M > TN_MAX));
}
DensePlan plan_dense(const Ctx *ctx, int M, int N, int K, int bits, int group_size, bool f16, bool slices = true) {
    const bool pieces = K / group_size % 8 == 0;
    const int n_tiles = (N + BMW - 1) / BMW, nkb = K / BK, nsb = (nkb + SB_PER_RAW - 1) / SB_PER_RAW, sms = ctx->sm_count;
    const auto up16 = [](int v) { return (v + 15) / 16 * 16; };
    if (ctx->qmm_force_tn > 0) return DensePlan{ctx->qmm_force_tn, (M + ctx->qmm_force_tn - 1) / ctx->qmm_force_tn, 1, 0, 0, false};
    constexpr int tn_wide = (TMEM_COLS - 3 * A_COLS) / 2;      // two accumulators and three k blocks of A (5-, 6- and 8-bit rings have two stages there)
    DensePlan best{};
    double best_us = 1e30;
    auto offer = [&](double us, const DensePlan &p) {
        if (us < best_us - 1e-9) {
            best_us = us;
            best = p;
        }
    };
    for (int form = 0; form < 2; ++form) {                     // 0: one chunk per item, 1: two
        if (form == 1 && (!ctx->qmm_wide || M <= TN_MAX)) continue;
        if (form == 0 && ctx->qmm_wide == 2 && M > TN_MAX) continue;                 // 2: whenever the shape allows (tests)
        const bool wide = form == 1;
        const int most = wide ? 2 * tn_wide : TN_MAX, fewest = (M + most - 1) / most;
        // as few items as cover the rows, and up to twice as many, narrower ones (not below 48 rows: 26 x 1536 x 1536 6.8 us as one, 8.6 as two)
        for (int items_m = fewest, last_tn = 0; items_m <= 2 * fewest + 2; ++items_m) {
            const int TN = wide ? up16((M + 2 * items_m - 1) / (2 * items_m)) : up16((M + items_m - 1) / items_m);
            if (TN == last_tn || (items_m > fewest && TN < 48)) continue;
            last_tn = TN;
            if ((items_m - 1) * (wide ? 2 : 1) * TN >= M) continue;                  // the last one would be empty
            const double one = kb_cost(TN, false, K, bits, pieces), kb_us = kb_cost(TN, wide, K, bits, pieces), item_us = item_cost(TN, wide);
            const long long units = static_cast<long long>(n_tiles) * items_m;
            // the last round of wide items on twice as many SMs, a chunk each, where that still is one round and every unit has two
            const int left = static_cast<int>(units % sms), last_rows = M - (items_m - 1) * 2 * TN;
            const bool tail = wide && units > sms && left > 0 && 2 * left <= sms && last_rows > TN;
            for (int S = 1; S <= 16; ++S) {
                if (S > 1 && (!slices || !ctx->qmm_ksplit || S > nsb || (ctx->qmm_wide != 1 && M > TN_MAX))) break;
                if (S > 1 && static_cast<size_t>(S) * M * N * sizeof(float) > kSliceBytes) break;
                const double kb = S == 1 ? nkb : (nsb + S - 1) / S * SB_PER_RAW;
                const long long full = units * S / sms, rest = units * S % sms;
                const double each_us = S == 1 ? item_us : item_cost(0, false);
                double us = full * (kb * kb_us + each_us);
                if (rest > 0) us += (S == 1 && tail ? kb * one : kb * kb_us) + each_us;
                if (S == 1 && items_m > fewest) us *= kMoreItems;
                if (S > 1) us += kSlicedUs + kEachSliceUs * S + static_cast<double>(S) * M * N * kSliceUs;
                offer(us, DensePlan{TN, items_m, S, S == 1 && tail ? left : 0, 0, wide});
            }
            // slices that are the CTAs of a cluster each and add up in shared memory: no block, no second kernel, but one round that the GPCs' odd sizes
            // leave room for; the sums take the ring's place
            if (!slices_allowed(ctx, M, form) || (wide ? 2 : 1) * TN * BMW * 4 > RING_BYTES) continue;
            for (int S = 2; S <= (wide ? 2 : 8) && S <= nsb; ++S) {
                if (units > kClusters[S] * sms / kNumSMsB200) continue;
                offer((nsb + S - 1) / S * SB_PER_RAW * kb_us + cluster_cost(S, (wide ? 2 : 1) * TN, units, f16), DensePlan{TN, items_m, S, 0, 1, wide});
            }
        }
    }
    return best;
}

// out[m, n] = sum over the K slices of partial[s][m, n], in slice order, times the factor of token row m; V outputs of a row per
// thread (16-byte loads of every slice in flight for V = 4)
struct SumOuts {
    void *outs[8];
    int n_outs;
    long long ld;
};
template <int V>
__global__ void __launch_bounds__(256) ksplit_sum_kernel(const float *partial, const float *tok_scale, const SumOuts o, int M, int N, int S, int dt) {
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");       // launched while the product kernel runs
    const size_t mn = static_cast<size_t>(M) * N;
    const uint32_t per_row = N / V;
    for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < mn / V; i += static_cast<size_t>(gridDim.x) * blockDim.x) {
        // 32-bit division: the partial sums of a launch are at most kSliceBytes
        const uint32_t m = static_cast<uint32_t>(i) / per_row, n = (static_cast<uint32_t>(i) - m * per_row) * V;
        float v[V];
        if constexpr (V == 4) {
            float4 pv[16];
#pragma unroll
            for (int q = 0; q < 16; ++q)
                if (q < S) pv[q] = *reinterpret_cast<const float4 *>(partial + static_cast<size_t>(q) * mn + i * 4);
            v[0] = pv[0].x; v[1] = pv[0].y; v[2] = pv[0].z; v[3] = pv[0].w;
#pragma unroll
            for (int q = 1; q < 16; ++q)
                if (q < S) { v[0] += pv[q].x; v[1] += pv[q].y; v[2] += pv[q].z; v[3] += pv[q].w; }
        } else {
            float pv[16];
#pragma unroll
            for (int q = 0; q < 16; ++q)
                if (q < S) pv[q] = partial[static_cast<size_t>(q) * mn + i];
            v[0] = pv[0];
#pragma unroll
            for (int q = 1; q < 16; ++q)
                if (q < S) v[0] += pv[q];
        }
        if (tok_scale) {
            const float f = tok_scale[m];
#pragma unroll
            for (int e = 0; e < V; ++e) v[e] *= f;
        }
        for (int d = 0; d < o.n_outs; ++d) {
            const size_t at = static_cast<size_t>(m) * o.ld + n;
            if (V == 4 && o.ld % 4 == 0 && reinterpret_cast<uintptr_t>(o.outs[d]) % 8 == 0) {
                *reinterpret_cast<uint2 *>(static_cast<unsigned short *>(o.outs[d]) + at) =
                    make_uint2(pack_out(v[0], v[V > 1 ? 1 : 0], dt == MTC_F16), pack_out(v[V > 2 ? 2 : 0], v[V > 3 ? 3 : 0], dt == MTC_F16));
            } else {
#pragma unroll
                for (int e = 0; e < V; ++e) st_from_f32(o.outs[d], at + e, v[e], dt);
            }
        }
    }
}

}  // namespace

namespace {
cudaError_t encode_map(CUtensorMap *map, CUtensorMapDataType type, int rank, const void *base, const cuuint64_t *dims, const cuuint64_t *strides,
                       const cuuint32_t *box, CUtensorMapSwizzle swizzle, std::string *why) {
    EncodeTiledFn encode = get_encode_fn();
    if (!encode) {
        if (why) *why = "cuTensorMapEncodeTiled is not available from the driver";
        return cudaErrorNotSupported;
    }
    const cuuint32_t estr[3] = {1, 1, 1};
    const CUresult r = encode(map, type, rank, const_cast<void *>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                              swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        if (why) *why = "cuTensorMapEncodeTiled failed with code " + std::to_string(static_cast<int>(r));
        return cudaErrorInvalidValue;
    }
    return cudaSuccess;
}
}  // namespace

cudaError_t make_map_2d(CUtensorMap *map, CUtensorMapDataType type, int elem_bytes, const void *base, long long rows, long long cols,
                        int box_rows, int box_cols, std::string *why) {
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows)};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(cols) * elem_bytes};
    const cuuint32_t box[2] = {static_cast<cuuint32_t>(box_cols), static_cast<cuuint32_t>(box_rows)};
    const int width = box_cols * elem_bytes;
    return encode_map(map, type, 2, base, dims, strides, box, width == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : width == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B, why);
}

cudaError_t make_map_blocks(CUtensorMap *map, const void *base, long long rows, long long cols, int box_rows, int box_blocks, std::string *why) {
    const cuuint64_t dims[3] = {64, static_cast<cuuint64_t>(rows), static_cast<cuuint64_t>(cols / 64)};
    const cuuint64_t strides[2] = {static_cast<cuuint64_t>(cols) * 2, 128};
    const cuuint32_t box[3] = {64, static_cast<cuuint32_t>(box_rows), static_cast<cuuint32_t>(box_blocks)};
    return encode_map(map, CU_TENSOR_MAP_DATA_TYPE_UINT16, 3, base, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B, why);
}

bool qmm_tcgen05_supported(int M, int N, int K, int bits, int group_size, int dt, const void *w, const void *x,
                           const void *out) {
    const bool bits_ok = bits == 2 || bits == 3 || bits == 4 || bits == 5 || bits == 6 || bits == 8;
    const bool gs_ok = group_size >= 32 && (group_size & (group_size - 1)) == 0 && K % group_size == 0;
    const auto al = [](const void *ptr, size_t a) { return reinterpret_cast<uintptr_t>(ptr) % a == 0; };
    return bits_ok && gs_ok && (dt == MTC_F16 || dt == MTC_BF16) && M > 0 && N > 0 && K % BK == 0 && al(w, 16) &&
           al(x, 16) && al(out, 2);
}

// A CTA an item, or one an SM: then no more of them than the rounds need, so that all take as many items (256 items as 128 CTAs with two each;
// where the last round is items of one chunk each, all of them)
static int dense_grid(const DensePlan &plan, int items, int sms) {
    if (plan.cluster || items <= sms) return items;
    const int rounds = (items + sms - 1) / sms;
    return plan.halves ? sms : (items + rounds - 1) / rounds;
}

// The form of a dense launch, for mtc_launch_of
void qmm_tcgen05_form(const Ctx *ctx, int M, int N, int K, int bits, int group_size, int dt, mtc_launch_info *info) {
    const DensePlan plan = plan_dense(ctx, M, N, K, bits, group_size, dt == MTC_F16);
    const int items = (N + BMW - 1) / BMW * plan.items_m * plan.ksplit + plan.halves;
    info->ctas = dense_grid(plan, items, ctx->sm_count);
    info->cluster = plan.cluster ? plan.ksplit : 1;
    info->k_slices = plan.ksplit;
}

cudaError_t launch_qmm_tcgen05(Ctx *ctx, cudaStream_t st, const void *w, const void *scales, const void *biases,
                               const void *x, void *out, int M, int N, int K, int bits, int group_size, int dt,
                               std::string *why, void *const *outs, int n_outs, long long out_ld) {
    const int sms = ctx->sm_count;
    DensePlan plan = plan_dense(ctx, M, N, K, bits, group_size, dt == MTC_F16);
    if (plan.ksplit > 1 && !plan.cluster) {
        cudaError_t ge = grow_block(ctx, st, &ctx->d_ksplit, &ctx->ksplit_bytes, static_cast<size_t>(plan.ksplit) * M * N * sizeof(float), why);
        if (ge != cudaSuccess) {
            if (M <= 16) return ge;         // the caller has a kernel without scratch for these
            // during capture, or out of memory: the same product without slices needs no block
            if (ge != cudaErrorStreamCaptureUnsupported) cudaGetLastError();
            if (why) why->clear();
            plan = plan_dense(ctx, M, N, K, bits, group_size, dt == MTC_F16, false);
        }
    }
    const int TN = plan.TN;
    const void *x_op = nullptr;
    const float *tok_scale = nullptr;
    cudaError_t e = stage_x(ctx, st, x, M, K, dt, &x_op, &tok_scale, why);
    if (e != cudaSuccess) return e;
    CUtensorMap tmap;
    e = make_x_map(&tmap, x_op, M, K, TN, 1, why);
    if (e != cudaSuccess) return e;
    QmmParams p{};
    fill_common(p, ctx, w, scales, biases, out, N, K, bits, group_size, dt, TN);
    p.tok_scale = tok_scale;
    if (outs) {                         // the result is a column block of wider row-major matrices, possibly on other GPUs
        for (int i = 0; i < n_outs && i < 8; ++i) p.outs[i] = outs[i];
        p.out = outs[0];
        p.n_outs = n_outs;
        p.out_ld = out_ld;
    }
    p.M = M;
    p.m_chunks = (M + TN - 1) / TN;
    p.n_tiles = (N + BMW - 1) / BMW;
    p.pdl_roles = early_weights(ctx, st);
    p.wide = plan.wide ? 1 : 0;
    plan_smem(p, ctx, bits);
    p.m_chunks = plan.items_m;
    p.wide_items = p.n_tiles * p.m_chunks - plan.halves;      // the last units run as two single-chunk items each
    p.dense_items = p.wide_items + 2 * plan.halves;
    // Few weight-row tiles: they alone would leave most SMs idle, so K is cut into slices that run as items of their own (f32
    // partial sums, added in slice order by a second small kernel).
    if (plan.ksplit > 1) {
        p.ksplit = plan.ksplit;
        plan_smem(p, ctx, bits);                // slices start at super-blocks
        p.partial = static_cast<float *>(ctx->d_ksplit);
        p.cluster = plan.cluster;
        p.dense_items = p.n_tiles * p.m_chunks * plan.ksplit;
    }
    set_out_vec(p);
    const int grid = dense_grid(plan, p.dense_items, sms);
    e = launch_any(bits, st, tmap, p, grid, N, why);
    if (e != cudaSuccess || p.ksplit == 1 || p.cluster) return e;
    const bool vec = N % 4 == 0;
    size_t sgrid = (static_cast<size_t>(M) * N / (vec ? 4 : 1) + 255) / 256;
    if (sgrid > static_cast<size_t>(sms) * 8) sgrid = static_cast<size_t>(sms) * 8;
    SumOuts so{};
    for (int i = 0; i < p.n_outs; ++i) so.outs[i] = p.outs[i];
    so.n_outs = p.n_outs;
    so.ld = p.out_ld;
    return launch_pdl(vec ? ksplit_sum_kernel<4> : ksplit_sum_kernel<1>, static_cast<int>(sgrid), 256, 0, st, static_cast<const float *>(p.partial),
                      p.tok_scale, so, M, N, p.ksplit, dt);
}

// scratch bytes the gather work list needs for these sizes
size_t gather_items_bytes(int total_rows, int n_experts, int N, int TN) {
    const size_t n_tiles = (N + BMW - 1) / BMW;
    const size_t max_items = n_tiles * (static_cast<size_t>(total_rows) / TN + n_experts + 1);
    return 16 + max_items * sizeof(int4);
}

cudaError_t launch_gather_qmm_tcgen05(Ctx *ctx, cudaStream_t st, const void *x, const void *w, const void *scales,
                                      const void *biases, const uint32_t *expert_offsets, const uint32_t *indices,
                                      void *out, int total_rows, int N, int K, int n_experts, int bits, int group_size,
                                      int dt, void *scratch, size_t scratch_bytes, std::string *why) {
    // token rows per item: about twice the mean rows per expert, so most experts are one chunk
    int TN = ctx->qmm_force_tn;
    if (TN <= 0) {
        const int mean = (total_rows + n_experts - 1) / n_experts;
        TN = ((2 * mean + 15) / 16) * 16;
        if (TN < 32) TN = 32;
        if (TN > TN_MAX) TN = TN_MAX;
    }
    const size_t need = gather_items_bytes(total_rows, n_experts, N, TN);
    if (!scratch || scratch_bytes < need) {
        if (why) *why = "gather_qmm: work-list scratch too small";
        return cudaErrorInvalidValue;
    }
    const int n_tiles = (N + BMW - 1) / BMW;
    const int max_items = static_cast<int>((scratch_bytes - 16) / sizeof(int4));
    int *count = static_cast<int *>(scratch);
    int4 *items = reinterpret_cast<int4 *>(static_cast<char *>(scratch) + 16);
    build_items_kernel<<<1, 256, 2 * (n_experts + 1) * sizeof(int), st>>>(expert_offsets, indices, total_rows, n_experts,
                                                                         n_tiles, TN, count, items, max_items, ctx->d_status);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    const void *x_op = nullptr;
    const float *tok_scale = nullptr;
    e = stage_x(ctx, st, x, total_rows, K, dt, &x_op, &tok_scale, why);
    if (e != cudaSuccess) return e;
    CUtensorMap tmap;
    e = make_x_map(&tmap, x_op, total_rows, K, TN, 1, why);
    if (e != cudaSuccess) return e;
    QmmParams p{};
    fill_common(p, ctx, w, scales, biases, out, N, K, bits, group_size, dt, TN);
    p.tok_scale = tok_scale;
    p.sb_total *= n_experts;
    p.M = total_rows;
    p.items = items;
    p.item_count = count;
    set_out_vec(p);
    return launch_any(bits, st, tmap, p, ctx->sm_count, static_cast<long long>(n_experts) * N, why);
}

// ---- gather_qmm for callers that cannot allocate ---------------------------------------------------
// Some hosts of this library may not call cudaMalloc at the point where they run a MoE layer:
// allocator-managed processes where every device byte is accounted for at start-up, and latency-critical
// loops that must not take the allocator's lock or meet an out-of-memory error in the middle of a step.  mtc_gather_qmm_static does the same
// work as mtc_gather_qmm on the tensor-core path but takes its scratch (the work list and the scaled-f16
// copy of bf16 activations) from one fixed array that lives in the library image: every GPU that loads
// the library holds these bytes until the process exits.  Limits below; sizes beyond them are refused.
constexpr size_t kStaticItems = 16384;                        // work items (16 bytes each)
constexpr size_t kStaticXElems = 8u << 20;                    // bf16 activations staged as f16: m_total * k_in elements
constexpr size_t kStaticRows = 65536;                         // rows of x (one f32 factor each)
constexpr size_t kStaticListBytes = 16 + kStaticItems * sizeof(int4);
constexpr size_t kStaticXOff = (kStaticListBytes + 255) & ~static_cast<size_t>(255);
constexpr size_t kStaticScaleOff = kStaticXOff + kStaticXElems * 2;
constexpr size_t kStaticBytes = kStaticScaleOff + kStaticRows * sizeof(float);

static __device__ __align__(256) unsigned char g_gather_static[kStaticBytes];

// The array's name is a host-side handle, not a device address: the address each device gave it is
// looked up once per device (with that device current) and cached.
cudaError_t gather_static_base(unsigned char **base) {
    static unsigned char *cache[64] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    if (!cache[dev]) {
        void *ptr = nullptr;
        e = cudaGetSymbolAddress(&ptr, g_gather_static);
        if (e != cudaSuccess) return e;
        cache[dev] = static_cast<unsigned char *>(ptr);
    }
    *base = cache[dev];
    return cudaSuccess;
}

cudaError_t launch_gather_qmm_static(Ctx *ctx, cudaStream_t st, const void *x, const void *w, const void *scales,
                                     const void *biases, const uint32_t *expert_offsets, const uint32_t *indices,
                                     void *out, int total_rows, int N, int K, int n_experts, int bits, int group_size,
                                     int dt, std::string *why) {
    int TN = ctx->qmm_force_tn;
    if (TN <= 0) {
        const int mean = (total_rows + n_experts - 1) / n_experts;
        TN = ((2 * mean + 15) / 16) * 16;
        if (TN < 32) TN = 32;
        if (TN > TN_MAX) TN = TN_MAX;
    }
    if (gather_items_bytes(total_rows, n_experts, N, TN) > kStaticListBytes) {
        if (why) *why = "gather_qmm_static: more than " + std::to_string(kStaticItems) + " work items (n_out/128 * (m_total/chunk + n_experts))";
        return cudaErrorInvalidValue;
    }
    if (dt == MTC_BF16 && (static_cast<size_t>(total_rows) * K > kStaticXElems || static_cast<size_t>(total_rows) > kStaticRows)) {
        if (why) *why = "gather_qmm_static: bf16 activations are limited to m_total * k_in <= " + std::to_string(kStaticXElems) +
                        " elements and m_total <= " + std::to_string(kStaticRows);
        return cudaErrorInvalidValue;
    }
    unsigned char *base = nullptr;
    cudaError_t e = gather_static_base(&base);
    if (e != cudaSuccess) return e;
    const int n_tiles = (N + BMW - 1) / BMW;
    int *count = reinterpret_cast<int *>(base);
    int4 *items = reinterpret_cast<int4 *>(base + 16);
    // the list and its count are rewritten by every call; nothing in the array has to start at zero
    build_items_kernel<<<1, 256, 2 * (n_experts + 1) * sizeof(int), st>>>(expert_offsets, indices, total_rows, n_experts,
                                                                         n_tiles, TN, count, items, static_cast<int>(kStaticItems), ctx->d_status);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    const void *x_op = x;
    const float *tok_scale = nullptr;
    if (dt == MTC_BF16) {
        __half *y = reinterpret_cast<__half *>(base + kStaticXOff);
        float *scale = reinterpret_cast<float *>(base + kStaticScaleOff);
        if ((e = launch_rows_to_f16(st, x, y, scale, total_rows, K)) != cudaSuccess) return e;
        x_op = y;
        tok_scale = scale;
    }
    CUtensorMap tmap;
    e = make_x_map(&tmap, x_op, total_rows, K, TN, 1, why);
    if (e != cudaSuccess) return e;
    QmmParams p{};
    fill_common(p, ctx, w, scales, biases, out, N, K, bits, group_size, dt, TN);
    p.tok_scale = tok_scale;
    p.sb_total *= n_experts;
    p.M = total_rows;
    p.items = items;
    p.item_count = count;
    set_out_vec(p);
    return launch_any(bits, st, tmap, p, ctx->sm_count, static_cast<long long>(n_experts) * N, why);
}

}  // namespace mtc
