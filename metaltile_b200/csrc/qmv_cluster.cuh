// qmv_cluster — quantized products of 5 to 16 token rows: 4- and 8-bit codes, the activations staged once an SM; K split over a cluster of CTAs
// where their rows are too long for that (one CTA by itself is the usual launch).
//
//   out[m, n] = sum_k (q(n,k) * scale[n, k/G] + bias[n, k/G]) * x[m, k]      1 <= M <= 16, f32 accumulation
//
// The codes are the A operand of mma.sync as they sit in the words, the activations the B operand, staged in fragment order,
// exactly as in qmv_frag.cuh (whose field and fragment rules are used here).  What differs is where things wait:
//   * a lane takes SEG / 4 neighbouring codes of each SEG-code segment (SEG = 64, or 32 for groups of 32), so the four lanes of a quad
//     share a group and all eight columns of an MMA belong to tokens;
//   * one CTA of 16 warps an SM stages the activations once for all of its warps; where a row of them does not fit beside the rings, or
//     costs more to stage than it serves (8 tokens of K = 14336 are 229 KB for 28 weight rows an SM), two, four or eight CTAs of a cluster take
//     a part of K each and add their partial tiles through distributed shared memory.  A cluster costs 0.8 us a doubling and four CTAs only
//     fill 132 of 148 SMs, so it is the last resort, not the default;
//   * words arrive as TMA boxes of 16 rows x 256 (128) bytes in a private ring of two units a warp, scales and biases beside them by
//     cp.async, 16 bytes a lane (one unit ahead in registers they were the longest wait: gate and up, 8 tokens 20.3 -> 19.0 us; as 8-byte
//     copies through L1 the LSU queue stood still: 33 us);
//   * the (tile, unit) pairs of a CTA are one flat sequence cut into 16 contiguous shares: every warp has the same number of units to within
//     one, and no barrier stands between tiles.  A warp leaves one partial tile for every tile that its share touches; they are added at the
//     end in the order of K (deterministic).
//
// What bounds it (28672 x 4096, 8 tokens: 16.6 us, 66 MB; 17.6 where every fourth launch drains, as in the profile of its counters): the ring alone streams at 5.6 TB/s (11.8 us with its launch); the products take 4 us
// that the stream does not hide (43 instructions a 64-code segment of 16 rows where the stream leaves 100 issue slots, at 16 warps'
// latency), staging the activations 1.5, the last sum and the stores 1.  Taken back: rings of 3 and 4 units (the partial tiles lose their room
// and a launch takes two passes: 25 -> 30 us at 16 tokens), every 16th unit to a warp instead of a run of them (partial tiles: five passes,
// 22 us), the bias term as m16n8k8 MMAs (fewer instructions, same time), 8 warps and two CTAs an SM.
#pragma once

#include <cuda.h>

#include "common.cuh"
#include "far_tokens.cuh"
#include "qmv_frag.cuh"

namespace mtc {

struct alignas(64) CluArgs {
    CUtensorMap map[4];          // words of each projection: {128 bytes, lines of a row, rows}
    FragProj p[4];
    int n_proj, tiles;           // projections that share x; 16-row tiles of all of them
    const void *x;
    uint32_t *status;
    int M, K, gs_shift;
    uint32_t s_pitch;            // bytes of a row of scales
    int units;                   // units of a row
    int cs_shift;                // log2 of the CTAs of a cluster
    int per, per_more, passes;   // tiles of a cluster (one more in the first per_more); passes over them (partial tiles of one pass fit shared memory)
    int touch;                   // partial tiles a warp may leave in a pass
    uint32_t plane;              // bytes of one piece of the staged activations
    uint32_t off_sum, off_scale, off_bar, off_red;
    int early;                   // weights may be read before the previous kernel of the stream is complete
};

namespace clu {

constexpr int kWarps = 16;                                  // one CTA an SM
constexpr int kDepth = 2;                                   // units in a warp's ring
constexpr uint32_t kSpin = 1u << 22;

__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t rank_addr(uint32_t addr, uint32_t rank) {     // the same place in another CTA's shared memory
    uint32_t a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(addr), "r"(rank));
    return a;
}
__device__ __forceinline__ float4 ld_rank(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
    return v;
}
template <int N>
__device__ __forceinline__ void lds(const char *p, uint32_t (&v)[N]) {
    if constexpr (N == 1) {
        v[0] = *reinterpret_cast<const uint32_t *>(p);
    } else if constexpr (N == 2) {
        const uint2 q = *reinterpret_cast<const uint2 *>(p);
        v[0] = q.x; v[1] = q.y;
    } else {
#pragma unroll
        for (int i = 0; i < N; i += 4) {
            const uint4 q = *reinterpret_cast<const uint4 *>(p + 4 * i);
            v[i] = q.x; v[i + 1] = q.y; v[i + 2] = q.z; v[i + 3] = q.w;
        }
    }
}
__device__ __forceinline__ void sts16(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ bool full_try(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
__device__ __forceinline__ void request_words(uint32_t dst, const CUtensorMap *map, int line, int row, uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
                 ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(0), "r"(line), "r"(row), "r"(bar) : "memory");
}
__device__ __forceinline__ void cp16(uint32_t dst, const void *src, uint32_t bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}

// Scales and biases of a unit: B bytes of each of 16 rows, in windows of 16 bytes.
template <int B>
constexpr uint32_t kScaleSlot = 32 * (B < 16 ? 16 : B);
template <int B>
__device__ __forceinline__ void lds_scales(const char *p, uint32_t (&v)[B < 4 ? 1 : B / 4]) {
    if constexpr (B == 2) v[0] = *reinterpret_cast<const uint16_t *>(p);
    else lds(p, v);
}
template <int XT>
__device__ __forceinline__ float scale_of(const uint32_t *v, int group) {          // group: a constant where this is inlined
    if (XT == MTC_F32) return __uint_as_float(v[group]);
    const uint32_t w = v[group >> 1];
    if (XT == MTC_BF16) return __uint_as_float((group & 1) ? (w & 0xFFFF0000u) : (w << 16));
    return __half2float(__ushort_as_half(static_cast<unsigned short>((group & 1) ? w >> 16 : w & 0xFFFFu)));
}

// Register r of a lane's codes of a segment: the pair code_lo(r), code_hi(r) in place.
template <int BITS, bool BF>
__device__ __forceinline__ uint32_t field(const uint32_t *w, int r) {
    constexpr uint32_t one = (1u << BITS) - 1u;
    const int b = frag::field_bit<BITS>(r), s = frag::field_shift<BITS, BF>(r);
    return (w[BITS == 4 ? r >> 2 : r >> 1] >> s) & ((one << (b - s)) * 0x10001u);
}

// The activations of (segment, token, quad lane): LC values, loaded ...
template <int XT, int LC>
struct XUnit {
    static constexpr int R = XT == MTC_F32 ? LC : LC / 2;
    uint32_t r[R];
    __device__ __forceinline__ void load(const void *x, size_t at, bool real) {
        const uint4 *p = reinterpret_cast<const uint4 *>(static_cast<const char *>(x) + at * (XT == MTC_F32 ? 4 : 2));
#pragma unroll
        for (int q = 0; q < R / 4; ++q) {
            const uint4 f = real ? p[q] : make_uint4(0u, 0u, 0u, 0u);
            r[4 * q] = f.x; r[4 * q + 1] = f.y; r[4 * q + 2] = f.z; r[4 * q + 3] = f.w;
        }
    }
};
// ... and stored in the order of the fields, per piece LC / 8 16-byte blocks.  f32: returns their sum.
template <int BITS, int XT, int LC>
__device__ __forceinline__ float stage_unit(const XUnit<XT, LC> &v, uint32_t dst, uint32_t flip, uint32_t plane) {
    if constexpr (XT == MTC_F32) {
        float s4[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
        for (int q = 0; q < LC; ++q) s4[q & 3] += __uint_as_float(v.r[q]);
        uint32_t o[3][4];
#pragma unroll
        for (int r = 0; r < LC / 2; ++r) {
            const float sc = __uint_as_float(static_cast<uint32_t>(127 + far_tokens::kUp - frag::field_pos<BITS, true>(r)) << 23);
            float lo = __uint_as_float(v.r[frag::code_lo<BITS>(r)]) * sc, hi = __uint_as_float(v.r[frag::code_hi<BITS>(r)]) * sc;
#pragma unroll
            for (int p = 0; p < 3; ++p) {
                const uint32_t b = frag::pack_bf16(lo, hi);
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
                for (int p = 0; p < 3; ++p) sts16((dst + p * plane + ((r >> 2) << 4)) ^ flip, o[p][0], o[p][1], o[p][2], o[p][3]);
            }
        }
        return (s4[0] + s4[1]) + (s4[2] + s4[3]);
    } else {
        uint32_t o[4];
#pragma unroll
        for (int r = 0; r < LC / 2; ++r) {
            const int lo = frag::code_lo<BITS>(r), hi = frag::code_hi<BITS>(r);
            uint32_t b = __byte_perm(v.r[lo >> 1], v.r[hi >> 1], ((lo & 1) ? 0x32 : 0x10) | ((hi & 1) ? 0x7600 : 0x5400));
            if (XT == MTC_BF16) {         // times 2^(kUp - pos): exact, subnormals included
                const uint32_t e = static_cast<uint32_t>(127 + far_tokens::kUp - frag::field_pos<BITS, true>(r)) << 7;
                asm("mul.rn.bf16x2 %0, %0, %1;" : "+r"(b) : "r"(e * 0x10001u));
            }
            o[r & 3] = b;
            if ((r & 3) == 3) sts16((dst + ((r >> 2) << 4)) ^ flip, o[0], o[1], o[2], o[3]);
        }
        return 0.0f;
    }
}

// The outputs of tokens that are out of range, once more: by the warps that have stored them (the tiles of every pass as in the kernel).
// far: shared memory that nothing uses any more.
template <int BITS, int XT>
__device__ __noinline__ void far_outputs(const CluArgs &a, uint32_t *far) {
    constexpr int ESZ = XT == MTC_F32 ? 4 : 2;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, cs = 1 << a.cs_shift, cr = blockIdx.x & (cs - 1), cid = static_cast<int>(blockIdx.x) >> a.cs_shift;
    const int t_lo = cid * a.per + min(cid, a.per_more), t_n = a.per + (cid < a.per_more);
    const auto token = [&](int t) { return static_cast<const char *>(a.x) + static_cast<size_t>(t) * a.K * ESZ; };
    if (warp < a.M) {                                                              // as many warps as tokens
        const uint32_t is = far_tokens::out_of_range<XT>(token(warp), a.K);
        if (lane == 0) far[warp] = is;
    }
    __syncthreads();
    for (int t = 0; t < a.M; ++t) {
        if (far[t] == 0) continue;
        for (int pass = 0; pass < a.passes; ++pass) {
            const int ta = t_lo + t_n * pass / a.passes, tb = t_lo + t_n * (pass + 1) / a.passes;
            for (int tile = ta + cr * kWarps + warp; tile < tb; tile += cs * kWarps) {
                int pi = 0;
                for (int j = 1; j < a.n_proj; ++j)
                    if (tile >= a.p[j].tile0) pi = j;
                const FragProj &pr = a.p[pi];
                const int n0 = (tile - pr.tile0) * 16;
                for (int n = n0; n < min(n0 + 16, pr.N); ++n) {
                    const size_t row = static_cast<size_t>(n), groups = row * a.s_pitch;
                    const float o = far_tokens::sum<BITS, XT>(pr.w + row * (a.K / 32 * BITS), static_cast<const char *>(pr.scales) + groups,
                                                              static_cast<const char *>(pr.biases) + groups, token(t), a.K, a.gs_shift);
                    if (lane == 0) st_from_f32(pr.out, static_cast<size_t>(t) * pr.N + n, o, XT);
                }
            }
        }
    }
}

// UB: 128-byte lines of a row in a unit; NG: groups of a unit (1: the group is a unit or longer)
template <int BITS, int XT, int NT, int SEG, int NG, int UB>
__global__ void __launch_bounds__(32 * kWarps, 1) qmv_cluster_kernel(const __grid_constant__ CluArgs a) {
    constexpr bool BF = XT != MTC_F16;
    constexpr int W = kWarps, P = frag::kPieces<XT>, ESZ = XT == MTC_F32 ? 4 : 2;
    constexpr int UC = UB * 1024 / BITS, US = UC / SEG, LC = SEG / 4, MP = 8 * NT;
    constexpr int SEG_BYTES = SEG * BITS / 8, LW = SEG_BYTES / 16;                 // a lane's words of a segment and row
    constexpr int SB = NG * ESZ, SR = SB < 4 ? 1 : SB / 4;                         // bytes and registers of a unit's scales of a row
    constexpr uint32_t SLOT = 16 * UB * 128, SSLOT = kScaleSlot<SB>;               // words and scales of a unit
    constexpr uint32_t XSEG = MP * 4 * LC * 2;                                     // bytes of a staged segment (one piece)
    constexpr uint32_t TILE = 16 * MP * 4;                                         // bytes of a partial tile: [row][token]
    static_assert(US >= 1 && (US % NG == 0 || NG == 1) && LC % 8 == 0, "shape of a unit");
    extern __shared__ __align__(1024) char smem[];
    const uint32_t sm0 = static_cast<uint32_t>(__cvta_generic_to_shared(smem));    // the rings come first: TMA's swizzle goes by address
    const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0), lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    // Integer divisions stand in the way of the first request (a launch of 4096 x 4096 took 0.5 us longer with them): shifts, products with
    // what the host divided, and quotients by a float reciprocal (exact: the values are far below 2^23 / 2).
    const int cs = 1 << a.cs_shift, cr = a.cs_shift ? static_cast<int>(cluster_rank()) : 0, cid = static_cast<int>(blockIdx.x) >> a.cs_shift;
    const auto rank_unit = [&](int r) { return r * a.units >> a.cs_shift; };
    const auto quotient = [](int n, int d) { return static_cast<int>((static_cast<float>(n) + 0.5f) * (1.0f / static_cast<float>(d))); };
    const int u0 = rank_unit(cr), nu = rank_unit(cr + 1) - u0;                     // this CTA's units of a row: u0 .. u0 + nu - 1
    const int t_lo = cid * a.per + min(cid, a.per_more), t_n = a.per + (cid < a.per_more);         // this cluster's tiles
    const auto pass_tile = [&](int i) { return t_lo + (i == 0 ? 0 : i == a.passes ? t_n : t_n * i / a.passes); };
    // Shares of `total` units: warp w has those from share(w) up to share(w + 1)
    const auto share = [](int w, int total) { return total >= kWarps ? total * w / kWarps : min(w, total); };
    if (!a.early) asm volatile("griddepcontrol.wait;" ::: "memory");

    const uint32_t ring = sm0 + warp * (kDepth * SLOT), bar = sm0 + a.off_bar + warp * (kDepth * 8);
    if (lane == 0) {
#pragma unroll
        for (int i = 0; i < kDepth; ++i) asm volatile("mbarrier.init.shared::cta.b64 [%0], 33;" ::"r"(bar + 8 * i) : "memory");   // TMA, and a lane's scales each
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();

    // ---- copies: this warp's units in order, a contiguous share of each pass's (tile, unit) pairs ----
    int c_pass = 0, c_left = 0, c_tile = 0, c_u = 0, c_row = 0;
    const CUtensorMap *c_map = nullptr;
    const char *c_src = nullptr;              // the row's scales (lane even) or biases (odd) of row lane / 2 of the tile
    uint32_t c_size = 0;                      // bytes from there to the end of the matrix
    auto open_tile = [&]() {
        int pi = 0;
#pragma unroll
        for (int i = 1; i < 4; ++i)
            if (i < a.n_proj && c_tile >= a.p[i].tile0) pi = i;
        const FragProj &pr = a.p[pi];
        c_map = &a.map[pi];
        c_row = (c_tile - pr.tile0) * 16;
        const int row = min(c_row + (lane >> 1), pr.N - 1);
        c_src = static_cast<const char *>((lane & 1) ? pr.biases : pr.scales) + static_cast<size_t>(row) * a.s_pitch;
        c_size = min(static_cast<uint32_t>(pr.N - row), 2u) * a.s_pitch;           // a window reaches into the next row at most
    };
    auto open_pass = [&]() {                  // the first pass from c_pass on in which this warp has units
        for (; c_pass < a.passes; ++c_pass) {
            const int ta = pass_tile(c_pass), total = (pass_tile(c_pass + 1) - ta) * nu, f0 = share(warp, total);
            c_left = share(warp + 1, total) - f0;
            if (c_left > 0) {
                c_tile = quotient(f0, nu);
                c_u = f0 - c_tile * nu;
                c_tile += ta;
                open_tile();
                return;
            }
        }
    };
    // Lane l copies the scales (l even) or biases (l odd) of row l / 2: the 16-byte windows that hold the unit's.
    const uint32_t s_dst = sm0 + a.off_scale + warp * (kDepth * SSLOT) + (lane & 1) * (SSLOT / 2) + (lane >> 1) * (SSLOT / 32);
    auto copy_next = [&](int slot) {
        if (c_left <= 0) return;
        const int u = u0 + c_u;
        if (lane == 0) request_words(ring + slot * SLOT, c_map, u * UB, c_row, bar + 8 * slot, SLOT);
        if constexpr (SB < 16) {                                                   // the last window may be cut short by the end of the matrix
            const uint32_t off = (static_cast<uint32_t>(u * UC) >> a.gs_shift) * ESZ;
            const char *const src = c_src + off;
            const uint32_t low = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(src)) & 15u, left = c_size - off + low;
            cp16(s_dst + slot * SSLOT, src - low, min(left, 16u));
        } else {
#pragma unroll
            for (int i = 0; i < SB; i += 16) cp16(s_dst + slot * SSLOT + i, c_src + u * SB + i, 16u);
        }
        asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar + 8 * slot) : "memory");
        if (--c_left == 0) {
            ++c_pass;
            open_pass();
        } else if (++c_u == nu) {
            c_u = 0;
            ++c_tile;
            open_tile();
        }
    };
    open_pass();
    // One unit a warp before the activations, the others behind them: what is requested first delays what is waited for first (gate and
    // up, 8 tokens: 18.3 -> 17.6 us).
    copy_next(0);
    asm volatile("griddepcontrol.launch_dependents;");

    // ---- activations of this CTA's part of K: a warp takes eight tokens of a segment at a time ----
    const uint32_t xs = sm0 + W * kDepth * SLOT;
    const char *const xs_p = smem + W * kDepth * SLOT;
    char *const sums_p = smem + a.off_sum;
    if (a.early) asm volatile("griddepcontrol.wait;" ::: "memory");
    constexpr int kBatch = XT == MTC_F32 ? 2 : 4;             // loads in flight together
    const int n_stage = nu * US * NT;
    for (int i0 = warp; i0 < n_stage; i0 += kBatch * W) {
      XUnit<XT, LC> v[kBatch];
#pragma unroll
      for (int j = 0; j < kBatch; ++j) {
        const int i = i0 + j * W, s = NT == 1 ? i : i >> 1, tok = (NT == 1 ? 0 : (i & 1) * 8) + g;
        v[j].load(a.x, static_cast<size_t>(tok) * a.K + static_cast<size_t>(u0) * UC + s * SEG + t * LC, i < n_stage && tok < a.M);
      }
      if (i0 == warp)                                         // the other units of the ring, once
#pragma unroll
        for (int j = 1; j < kDepth; ++j) copy_next(j);
#pragma unroll
      for (int j = 0; j < kBatch; ++j) {
        const int i = i0 + j * W, s = NT == 1 ? i : i >> 1, tok = (NT == 1 ? 0 : (i & 1) * 8) + g;
        if (i >= n_stage) break;
        const uint32_t at = static_cast<uint32_t>(s * MP + tok) * (4 * LC * 2) + t * (LC * 2), flip = LC == 16 ? (g & 1) << 4 : 0;
        float sum = stage_unit<BITS, XT, LC>(v[j], xs + at, flip, a.plane);
        if constexpr (XT == MTC_F32) {
            sum += __shfl_xor_sync(0xffffffffu, sum, 1);
            sum += __shfl_xor_sync(0xffffffffu, sum, 2);
            if (t == 0) *reinterpret_cast<float *>(sums_p + (s * MP + tok) * 4) = sum * __uint_as_float((127u - far_tokens::kUnit) << 23);      // in the units of the products
        } else {                              // the sums in the units of the products: against codes that are all one
            __syncwarp();
            float d[4];
#pragma unroll
            for (int q = 0; q < LC / 8; ++q) {
                const uint4 b = *reinterpret_cast<const uint4 *>(xs_p + ((at + q * 16) ^ flip));
                const uint32_t o[4] = {0x10001u << frag::field_pos<BITS, BF>(4 * q), 0x10001u << frag::field_pos<BITS, BF>(4 * q + 1),
                                       0x10001u << frag::field_pos<BITS, BF>(4 * q + 2), 0x10001u << frag::field_pos<BITS, BF>(4 * q + 3)};
                frag::mma<BF>(d, o[0], o[0], o[1], o[1], b.x, b.y, q == 0);
                frag::mma<BF>(d, o[2], o[2], o[3], o[3], b.z, b.w, false);
            }
            if (g == 0) *reinterpret_cast<float2 *>(sums_p + (s * MP + tok + 2 * t) * 4) = make_float2(d[0], d[1]);
        }
      }
    }
    if (warp >= n_stage)                                      // a short row has fewer pieces than warps: these did not come by
#pragma unroll
        for (int j = 1; j < kDepth; ++j) copy_next(j);
    __syncthreads();

    // ---- products ----
    uint32_t *const odd = reinterpret_cast<uint32_t *>(smem + a.off_bar + W * kDepth * 8);         // a result may be of a token out of range (far_tokens.cuh);
    if (XT != MTC_F16 && threadIdx.x == 0) *odd = 0;                               // set behind the barrier of a pass
    const float post = XT == MTC_F16 ? __uint_as_float((127u + 24u) << 23) : __uint_as_float((127u + far_tokens::kUnit) << 23);
    // Row r of a unit is UB lines of 128 bytes; TMA stores 16-byte chunk c of line l at c ^ (l & 7): the rows a load phase reads (two
    // of 64 bytes, four of 32, eight of 16) fall on different banks.
    uint32_t w_lane[UB];
#pragma unroll
    for (int h = 0; h < UB; ++h)
        w_lane[h] = static_cast<uint32_t>(warp * (kDepth * SLOT) + (g * UB + h) * 128) + (((((t * LW) >> 2) ^ (g * UB + h)) & 7) << 4) + ((t * LW) & 3) * 4;
    const uint32_t x_lane = static_cast<uint32_t>(g * 4 + t) * (LC * 2) ^ (LC == 16 ? (g & 1) << 4 : 0);
    const char *const s_lane = smem + a.off_scale + warp * (kDepth * SSLOT) + g * (SSLOT / 32);
    const uint32_t red0 = sm0 + a.off_red, s_low[2] = {g * a.s_pitch, (g + 8) * a.s_pitch};       // tiles start on 16 rows: only the row in the tile counts
    int slot = 0;
    uint32_t parity = 0, spin = kSpin;
#pragma unroll 1
    for (int pass = 0; pass < a.passes; ++pass) {
        const int ta = pass_tile(pass), n_tiles = pass_tile(pass + 1) - ta, total = n_tiles * nu;
        const int f0 = share(warp, total), f1 = share(warp + 1, total);
        char *mine = smem + a.off_red + static_cast<uint32_t>(warp * a.touch) * TILE + (g * MP + 2 * t) * 4;
        int u = f0 - quotient(f0, nu) * nu;
        float acc[NT][4];
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[nt][j] = 0.0f;
#pragma unroll 1
        for (int f = f0; f < f1; ++f) {
            for (uint32_t i = 0; !full_try(bar + 8 * slot, parity); ++i)
                if (i >= spin) {                                                   // the copies did not arrive: tell the host, wait no more
                    if (lane == 0) atomicCAS(a.status, 0u, 0xA01u);
                    spin = 0;
                    break;
                }
            uint32_t sc[4][SR];                                                    // scales of rows g, g + 8, biases of the two
            const char *const su = sums_p + static_cast<uint32_t>(u) * (US * MP * 4) + t * 8;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const char *q = s_lane + slot * SSLOT + (j >> 1) * (SSLOT / 2) + (j & 1) * (SSLOT / 4);
                if (SB < 16) q += (s_low[j & 1] + ((static_cast<uint32_t>((u0 + u) * UC) >> a.gs_shift) * ESZ)) & 15u;
                lds_scales<SB>(q, sc[j]);
            }
            const uint32_t xo = x_lane + static_cast<uint32_t>(u) * (US * XSEG);
            const char *const xa = xs_p + xo, *const xb = xs_p + (xo ^ 16u);
#pragma unroll
            for (int p = 0; p < US; ++p) {
                uint32_t wl[LW], wh[LW];
                const char *const wa = smem + ((w_lane[p * SEG_BYTES / 128] + slot * SLOT) ^ (p * SEG_BYTES & 127));
                lds(wa, wl);
                lds(wa + 8 * UB * 128, wh);
                float d[NT][4], e[P == 3 ? NT : 1][4], f3[P == 3 ? NT : 1][4];
#pragma unroll
                for (int q = 0; q < LC / 8; ++q) {                                 // 16 bytes of B: two MMAs
                    uint32_t al[4], ah[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        al[i] = field<BITS, BF>(wl, 4 * q + i);
                        ah[i] = field<BITS, BF>(wh, 4 * q + i);
                    }
#pragma unroll
                    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                        for (int pc = 0; pc < P; ++pc) {
                            uint32_t b[4];
                            lds((q ? xb : xa) + p * XSEG + nt * (8 * 4 * LC * 2) + pc * a.plane, b);
                            if (P == 3 && pc > 0) {
                                frag::mma<BF>(f3[nt], al[0], ah[0], al[1], ah[1], b[0], b[1], q == 0 && pc == 1);
                                frag::mma<BF>(f3[nt], al[2], ah[2], al[3], ah[3], b[2], b[3], false);
                            } else {
                                frag::mma<BF>(d[nt], al[0], ah[0], al[1], ah[1], b[0], b[1], q == 0);
                                frag::mma<BF>(P == 3 ? e[nt] : d[nt], al[2], ah[2], al[3], ah[3], b[2], b[3], P == 3 && q == 0);
                            }
                        }
                }
                const float s_l = scale_of<XT>(sc[0], p * NG / US), s_h = scale_of<XT>(sc[1], p * NG / US);
#pragma unroll
                for (int nt = 0; nt < NT; ++nt) {
                    if (P == 3) {
#pragma unroll
                        for (int j = 0; j < 4; ++j) d[nt][j] = (d[nt][j] + e[nt][j]) + f3[nt][j];
                    }
                    const float b_l = scale_of<XT>(sc[2], p * NG / US), b_h = scale_of<XT>(sc[3], p * NG / US);
                    const float2 x = *reinterpret_cast<const float2 *>(su + p * (MP * 4) + nt * 32);
                    acc[nt][0] = fmaf(s_l, d[nt][0], fmaf(b_l, x.x, acc[nt][0]));
                    acc[nt][1] = fmaf(s_l, d[nt][1], fmaf(b_l, x.y, acc[nt][1]));
                    acc[nt][2] = fmaf(s_h, d[nt][2], fmaf(b_h, x.x, acc[nt][2]));
                    acc[nt][3] = fmaf(s_h, d[nt][3], fmaf(b_h, x.y, acc[nt][3]));
                }
            }
            __syncwarp();                                                          // every lane is done with the slot
            copy_next(slot);
            if (++slot == kDepth) {
                slot = 0;
                parity ^= 1u;
            }
            if (++u == nu || f + 1 == f1) {                                        // this warp's part of a tile
                u = 0;
#pragma unroll
                for (int nt = 0; nt < NT; ++nt) {
                    *reinterpret_cast<float2 *>(mine + nt * 32) = make_float2(acc[nt][0], acc[nt][1]);
                    *reinterpret_cast<float2 *>(mine + nt * 32 + 8 * MP * 4) = make_float2(acc[nt][2], acc[nt][3]);
#pragma unroll
                    for (int j = 0; j < 4; ++j) acc[nt][j] = 0.0f;
                }
                mine += TILE;
            }
        }
        if (cs > 1) cluster_sync();
        else __syncthreads();
        // The sum over the ranks and warps of every tile, in that order (of K).  A warp takes a tile, a lane four tokens of a row (NT rows).
        for (int tl = cr * W + warp; tl < n_tiles; tl += cs * W) {
            float4 v[NT];
#pragma unroll
            for (int i = 0; i < NT; ++i) v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            for (int r = 0; r < cs; ++r) {
                const int nr = rank_unit(r + 1) - rank_unit(r), all = n_tiles * nr;
                const int start = lane < W ? share(lane, all) : all;               // lane w: first unit of warp w
                const int wa = 31 - __clz(__ballot_sync(0xffffffffu, start <= tl * nr));       // has the tile's first unit; later ones start in the tile
                const int wb = 31 - __clz(__ballot_sync(0xffffffffu, start < (tl + 1) * nr));
                const int nth = tl - quotient(__shfl_sync(0xffffffffu, start, wa), nr);
                const uint32_t at = red0 + lane * 16 + static_cast<uint32_t>(wa * a.touch) * TILE, next = static_cast<uint32_t>(a.touch) * TILE;
                auto add = [&](const float4 &q, int i) { v[i].x += q.x; v[i].y += q.y; v[i].z += q.z; v[i].w += q.w; };
                if (cs == 1) {
                    const char *q = smem + (at - sm0);
#pragma unroll
                    for (int i = 0; i < NT; ++i) add(*reinterpret_cast<const float4 *>(q + nth * TILE + i * 512), i);
#pragma unroll 4
                    for (int w = wa + 1; w <= wb; ++w) {
                        q += next;
#pragma unroll
                        for (int i = 0; i < NT; ++i) add(*reinterpret_cast<const float4 *>(q + i * 512), i);
                    }
                } else {
                    uint32_t q = rank_addr(at, r);
#pragma unroll
                    for (int i = 0; i < NT; ++i) add(ld_rank(q + nth * TILE + i * 512), i);
#pragma unroll 4
                    for (int w = wa + 1; w <= wb; ++w) {
                        q += next;
#pragma unroll
                        for (int i = 0; i < NT; ++i) add(ld_rank(q + i * 512), i);
                    }
                }
            }
            const int tile = ta + tl;
            int pi = 0;
#pragma unroll
            for (int j = 1; j < 4; ++j)
                if (j < a.n_proj && tile >= a.p[j].tile0) pi = j;
            const FragProj &pr = a.p[pi];
#pragma unroll
            for (int i = 0; i < NT; ++i) {
                const int idx = i * 32 + lane, row = idx / (MP / 4), tok = idx % (MP / 4) * 4, nn = (tile - pr.tile0) * 16 + row;
                const float o[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (nn < pr.N && tok + j < a.M) {
                        st_from_f32(pr.out, static_cast<size_t>(tok + j) * pr.N + nn, o[j] * post, XT);
                        if (XT != MTC_F16 && far_tokens::odd<XT>(o[j])) *odd = 1;
                    }
            }
        }
        // no partial tile is rewritten, and no CTA leaves, while another reads it
        if (cs > 1) cluster_sync();
        else if (pass + 1 < a.passes || XT != MTC_F16) __syncthreads();
    }
    if (XT != MTC_F16 && *odd != 0) far_outputs<BITS, XT>(a, reinterpret_cast<uint32_t *>(smem));
}

// ---- host side -----------------------------------------------------------------------------------------------------
struct Shape {
    int nt, group, xt;
};

cudaError_t word_maps(CluArgs &a, int row_bytes, int ub);

struct Plan {
    int shift = -1, clusters = 0, passes = 0, touch = 0;
    uint32_t plane = 0, off_sum = 0, off_scale = 0, off_bar = 0, off_red = 0, smem = 0;
    double cost = 1e30;
};
constexpr uint32_t kSmemMax = 227 * 1024;

// pieces: of an activation; us: segments of a unit; xseg: bytes of a staged segment and piece; slot, sslot: bytes of the words and scales of a unit
inline Plan make_plan(int tiles, int units, int pieces, int us, uint32_t xseg, int mp, uint32_t slot, uint32_t sslot, int sms) {
    constexpr int W = kWarps;
    const uint32_t tile = 16 * mp * 4;
    Plan best;
    for (int shift = 0; shift <= 3; ++shift) {
        const int cs = 1 << shift;
        if (cs > units) break;
        Plan p;
        p.shift = shift;
        const int nu = (units + cs - 1) / cs, nu_min = units / cs;
        p.plane = static_cast<uint32_t>(nu) * us * xseg;
        p.off_sum = W * kDepth * slot + p.plane * pieces;
        p.off_scale = (p.off_sum + static_cast<uint32_t>(nu) * us * mp * 4 + 15) / 16 * 16;
        p.off_bar = p.off_scale + W * kDepth * sslot;
        p.off_red = (p.off_bar + W * kDepth * 8 + 4 + 127) / 128 * 128;           // barriers, a word on the results
        if (p.off_red > kSmemMax) continue;
        p.clusters = cs <= 2 ? sms / cs : cs == 4 ? sms * 33 / 148 : sms * 15 / 148;       // what fits the GPCs at once
        if (p.clusters > tiles) p.clusters = tiles;
        const int per = (tiles + p.clusters - 1) / p.clusters;                     // tiles of the largest cluster
        int len = 0;
        for (p.passes = 1; p.passes <= per; ++p.passes) {
            len = ((per + p.passes - 1) / p.passes * nu + W - 1) / W;
            p.touch = (len + nu_min - 2) / nu_min + 1;
            if (p.off_red + W * p.touch * tile <= kSmemMax) break;
        }
        if (p.passes > per) continue;
        p.smem = p.off_red + W * p.touch * tile;
        // clocks: a unit of 4 KB on a full SM ~3600 (two token tiles 5600), the sum of a pass and what it drains, a round of staged segments, the
        // cluster's launch and barriers (4096 x 4096, 8 tokens, one to four CTAs: 5.9, 6.7, 7.5 us)
        const double staging = static_cast<double>((nu * us * (mp / 8) + W - 1) / W) * pieces;
        p.cost = p.passes * (len * (mp == 8 ? 3600.0 : 5600.0) * pieces * (slot / 4096.0) + 2500.0) + staging * 350.0 + shift * 1500.0;
        if (p.cost < best.cost) best = p;
    }
    return best;
}

// 128-byte lines of a row in a unit: two; one for two token tiles and for three pieces (their activations leave less room for rings and
// partial tiles) and for groups of 32 (registers of scales)
constexpr int lines(int dt, int M, int group) { return dt == MTC_F32 || M > 8 || group == 32 ? 1 : 2; }

inline Plan shape_plan(const mtc_qmv_desc &d, int tiles, int sms) {
    const int esz = static_cast<int>(dtype_size(d.dtype)), ub = lines(d.dtype, d.M, d.group_size), unit = ub * 1024 / d.bits;
    const int seg = d.group_size == 32 ? 32 : 64, mp = d.M <= 8 ? 8 : 16, bytes = (d.group_size < unit ? unit / d.group_size : 1) * esz;
    return make_plan(tiles, d.K / unit, d.dtype == MTC_F32 ? 3 : 1, unit / seg, mp * seg * 2, mp, 16 * ub * 128, 32 * (bytes < 16 ? 16 : bytes), sms);
}

template <int BITS, int XT, int NT, int SEG, int NG, int UB>
cudaError_t launch_one(cudaStream_t st, CluArgs &a, const Plan &p) {
    a.units = a.K / (UB * 1024 / BITS);
    cudaError_t e = word_maps(a, a.K / 8 * BITS, UB);
    if (e != cudaSuccess) return e;
    auto kern = qmv_cluster_kernel<BITS, XT, NT, SEG, NG, UB>;
    static PerDeviceAttr attr;
    e = attr.set(kern, kSmemMax);
    if (e != cudaSuccess) return e;
    a.cs_shift = p.shift;
    a.per = a.tiles / p.clusters;
    a.per_more = a.tiles % p.clusters;
    a.passes = p.passes;
    a.touch = p.touch;
    a.plane = p.plane;
    a.off_sum = p.off_sum;
    a.off_scale = p.off_scale;
    a.off_bar = p.off_bar;
    a.off_red = p.off_red;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(p.clusters << p.shift);
    cfg.blockDim = dim3(32 * kWarps);
    cfg.dynamicSmemBytes = p.smem;
    cfg.stream = st;
    cudaLaunchAttribute la[2];
    la[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    la[0].val.programmaticStreamSerializationAllowed = 1;
    la[1].id = cudaLaunchAttributeClusterDimension;
    la[1].val.clusterDim.x = 1u << p.shift;
    la[1].val.clusterDim.y = 1;
    la[1].val.clusterDim.z = 1;
    cfg.attrs = la;
    cfg.numAttrs = p.shift > 0 ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, kern, a);
}

template <int BITS, int XT, int NT>
cudaError_t launch_groups(cudaStream_t st, CluArgs &a, const Shape &s, const Plan &p) {
    constexpr int UB = lines(XT, NT * 8, 64), kSegs = UB * 1024 / BITS / 64;                // 8, 4 or 2
    if (s.group == 32) return launch_one<BITS, XT, NT, 32, 32 / BITS, 1>(st, a, p);
    if (s.group == 64) return launch_one<BITS, XT, NT, 64, kSegs, UB>(st, a, p);
    if (s.group == 128) return launch_one<BITS, XT, NT, 64, kSegs / 2, UB>(st, a, p);
    if constexpr (kSegs == 8)
        if (s.group == 256) return launch_one<BITS, XT, NT, 64, 2, UB>(st, a, p);
    return launch_one<BITS, XT, NT, 64, 1, UB>(st, a, p);
}

template <int BITS>
cudaError_t launch_bits(cudaStream_t st, CluArgs &a, const Shape &s, const Plan &p) {
    if (s.xt == MTC_F32) return s.nt == 1 ? launch_groups<BITS, MTC_F32, 1>(st, a, s, p) : launch_groups<BITS, MTC_F32, 2>(st, a, s, p);
    if (s.xt == MTC_F16) return s.nt == 1 ? launch_groups<BITS, MTC_F16, 1>(st, a, s, p) : launch_groups<BITS, MTC_F16, 2>(st, a, s, p);
    return s.nt == 1 ? launch_groups<BITS, MTC_BF16, 1>(st, a, s, p) : launch_groups<BITS, MTC_BF16, 2>(st, a, s, p);
}

}  // namespace clu

// one translation unit per width (qmv_cluster_b*.cu)
cudaError_t launch_cluster_b4(cudaStream_t, CluArgs &, const clu::Shape &, const clu::Plan &);
cudaError_t launch_cluster_b8(cudaStream_t, CluArgs &, const clu::Shape &, const clu::Plan &);

}  // namespace mtc
