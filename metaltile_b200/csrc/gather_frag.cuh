// gather_frag — the grouped (mixture-of-experts) quantized product where an expert sees a handful of rows, every width:
//
//   out[r, n] = sum_k (q(e, n, k) * scale[e, n, k/G] + bias[e, n, k/G]) * x[r, k],   e = the expert that owns row r
//
// x rows are sorted by expert (expert_offsets, CSR).  Stands in for mt_moe_gather_qmm_{int4*,b3,b5,b6,b8}
// (crates/metaltile-std/src/ffai/moe.rs:358-1363) while a layer decodes: the tcgen05 kernel dequantises 128 x 64 blocks whatever the rows
// (0.42 us a block) behind a work list, a permutation and a conversion of their own; here the packed words of 16 weight rows go from
// global memory into MMA fragments as in qmv_frag.cuh, whose modes, fields and steps are used as they are, and one launch covers gate and up.
//
// Work.  A PASS is (expert, up to CAP * NT of its rows); every CTA derives the passes from expert_offsets by itself (a scan over the experts
// in shared memory: a launch less than a table).  The 16-row tiles of all passes are dealt to SLOTS - KS warps of a CTA that split K - as
// contiguous ranges, so that a warp stages the activations of its part of K once for the tiles of a pass that it owns.  The KS partial tiles are
// added in warp order behind a barrier of the slot: deterministic, and independent of how many tiles there are.
//
// What bounds it: as the fragment kernel, issue and latency; all of it waits for the kernel before (the offsets).  Measured where its rule stands
// (runtime.cu): 64 experts of 1088 x 448, 26 rows, 6-bit 86 -> 28 us a layer; 32 of 1024 x 768, 48 rows, 2-bit 69 -> 34.
#pragma once

#include "common.cuh"
#include "far_tokens.cuh"
#include "qmv_frag.cuh"

namespace mtc {

struct GfArgs {
    const uint32_t *w[2];            // one or two matrix sets that read the same rows (gate and up)
    const void *scales[2], *biases[2];
    void *out[2];
    const void *x;
    const uint32_t *offsets;         // [n_experts + 1]
    const uint32_t *row_src;         // row m of the product is row row_src[m] of x (null: row m)
    uint32_t *status;
    int n_src_rows, n_experts, m_total;
    int n_out, K, gs_shift, wpr, gpr, steps;
    int tpm, tpe;                    // 16-row tiles of a matrix; of all matrices of an expert
    int ks;                          // warps of a slot
    uint32_t off_sum, off_part, warp_bytes, off_red;
};

namespace gfrag {

using namespace frag;

constexpr int kGfWarps = 8;          // two CTAs an SM

struct RowX {                        // one row of activations, as stage_chunk reads it
    const void *x;
    int K, M;
};

struct Tile {
    int pass, expert, tok0, ntok, second, row0;
};
// The rows of expert e: how many, from `lo` on
__device__ __forceinline__ int rows_of(const GfArgs &a, int e, int &lo) {
    const uint32_t p = a.offsets[e], q = a.offsets[e + 1], m = static_cast<uint32_t>(a.m_total);
    lo = static_cast<int>(min(p, m));
    if (p > m || q > m || q < p) atomicCAS(a.status, 0u, 0x901u);                      // clamped and reported
    return max(static_cast<int>(min(q, m)) - lo, 0);
}
// start[e]: passes of MP rows before expert e
template <int MP>
__device__ __forceinline__ void locate(const GfArgs &a, const int *start, int tile, Tile &q) {
    q.pass = tile / a.tpe;
    const int r = tile - q.pass * a.tpe;
    int lo = 0, hi = a.n_experts;                                      // the last expert with start[e] <= pass: it has rows
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (start[mid] <= q.pass) lo = mid; else hi = mid;
    }
    q.expert = lo;
    int first;
    const int rows = rows_of(a, lo, first), done = (q.pass - start[lo]) * MP;
    q.tok0 = first + done;
    q.ntok = min(MP, rows - done);
    q.second = r >= a.tpm ? 1 : 0;
    q.row0 = (r - (q.second ? a.tpm : 0)) * 16;
}
// The row of x that row r of the product is
__device__ __forceinline__ const char *row_of(const GfArgs &a, int r) {
    size_t row = static_cast<size_t>(r);
    if (a.row_src) {
        const uint32_t s = a.row_src[row];
        if (s >= static_cast<uint32_t>(a.n_src_rows)) atomicCAS(a.status, 0u, 0x903u);     // not a row of x: row 0 is read instead
        row = s < static_cast<uint32_t>(a.n_src_rows) ? s : 0;
    }
    return static_cast<const char *>(a.x) + row * (static_cast<size_t>(a.K) * 2);
}

// The outputs of rows that are out of range (far_tokens.cuh), once more, by the warp that has stored them: of tiles t_lo to t_hi, two rows of x a
// turn.
template <int BITS, int XT, int MP>
__device__ __noinline__ void far_rows(const GfArgs &a, const int *start, int t_lo, int t_hi) {
    const int lane = threadIdx.x & 31, slice = (threadIdx.x >> 5) % a.ks;
    uint32_t far = 0;
    __syncwarp();
    for (int tile = t_lo, pass = -1; tile < t_hi; ++tile) {
        Tile q;
        locate<MP>(a, start, tile, q);
        if (q.pass != pass) far = 0;
        for (int e = slice * 32; e < q.ntok * 16; e += 32 * a.ks)
            for (int tok = e >> 4; tok < min((e >> 4) + 2, q.ntok); ++tok) {
                const char *const x = row_of(a, q.tok0 + tok);
                if (q.pass != pass && far_tokens::out_of_range<XT>(x, a.K)) far |= 1u << tok;
                if (!(far >> tok & 1u)) continue;
                for (int n = q.row0; n < min(q.row0 + 16, a.n_out); ++n) {
                    const size_t row = static_cast<size_t>(q.expert) * a.n_out + n, groups = row * a.gpr * 2;
                    const float v = far_tokens::sum<BITS, XT>(a.w[q.second] + row * a.wpr, static_cast<const char *>(a.scales[q.second]) + groups,
                                                              static_cast<const char *>(a.biases[q.second]) + groups, x, a.K, a.gs_shift);
                    if (lane == 0) st_from_f32(a.out[q.second], static_cast<size_t>(q.tok0 + tok) * a.n_out + n, v, XT);
                }
            }
        pass = q.pass;
    }
}

template <int BITS, int XT, int MODE, int NT>
__global__ void __launch_bounds__(32 * kGfWarps, 2) gather_frag_kernel(const __grid_constant__ GfArgs a) {
    constexpr int RUN = MODE == G8 ? 2 : kRun<BITS>, H = MODE == G8 ? 2 : 1, CAP = kCap<MODE>, MP = CAP * NT, ESZ = 2;
    constexpr uint32_t STEP = MP * 4 * kPitch<XT>, SUM = NT * H * 4 * 8;
    static_assert(MODE != S1 && XT != MTC_F32, "forms of this kernel");
    extern __shared__ __align__(128) char smem[];
    const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0), lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int slots = kGfWarps / a.ks, slot = warp / a.ks, slice = warp - slot * a.ks;
    pdl_enter();                     // the offsets, the rows
    // ---- passes: start[e] = passes before expert e ----
    int *start = reinterpret_cast<int *>(smem);
    for (int e = threadIdx.x; e < a.n_experts; e += 32 * kGfWarps) {
        int lo;
        start[e + 1] = (rows_of(a, e, lo) + MP - 1) / MP;
    }
    if (threadIdx.x == 0) start[0] = 0;
    __syncthreads();
    if (warp == 0) {
        int carry = 0;
        for (int e0 = 1; e0 <= a.n_experts; e0 += 32) {
            int v = e0 + lane <= a.n_experts ? start[e0 + lane] : 0;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int up = __shfl_up_sync(0xffffffffu, v, d);
                if (lane >= d) v += up;
            }
            if (e0 + lane <= a.n_experts) start[e0 + lane] = carry + v;
            carry += __shfl_sync(0xffffffffu, v, 31);
        }
    }
    __syncthreads();
    const long long total = min(static_cast<long long>(start[a.n_experts]) * a.tpe, 0x7FFFFFFFll);        // offsets that overlap could name more
    const long long id = static_cast<long long>(blockIdx.x) * slots + slot, n_slots = static_cast<long long>(gridDim.x) * slots;
    const int t_lo = static_cast<int>(total * id / n_slots), t_hi = static_cast<int>(total * (id + 1) / n_slots);
    if (t_lo >= t_hi) return;        // whole slots leave: the barriers below are their own

    // ---- requests: one run of steps in registers, one run ahead of the products (see qmv_frag_kernel) ----
    const int total_runs = (a.steps + RUN - 1) / RUN, r0 = slice * total_runs / a.ks, r1 = (slice + 1) * total_runs / a.ks;
    const int n_units = MODE == G8 ? a.K >> 6 : a.K >> 5;                          // halves (G8) or chunks of a row
    uint32_t wl[RUN][BITS], wh[RUN][BITS];
    Affine<XT, MODE, RUN, 0> sc, bi;
#pragma unroll
    for (int i = 0; i < RUN; ++i)
#pragma unroll
        for (int j = 0; j < BITS; ++j) wl[i][j] = wh[i][j] = 0u;
#pragma unroll
    for (int j = 0; j < sc.W; ++j) sc.r[0][j] = sc.r[1][j] = bi.r[0][j] = bi.r[1][j] = 0u;
    const char *wrow[2] = {nullptr, nullptr}, *srow[2] = {nullptr, nullptr}, *brow[2] = {nullptr, nullptr};     // rows g, g + 8 of the tile being requested
    int l_tile = t_lo, l_run = r0;
    bool whole = true;
    Tile lt;
    auto open_tile = [&]() {
        locate<MP>(a, start, l_tile, lt);
        const size_t row0 = static_cast<size_t>(lt.expert) * a.n_out;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const size_t row = row0 + min(lt.row0 + g + 8 * j, a.n_out - 1);
            wrow[j] = reinterpret_cast<const char *>(a.w[lt.second]) + row * (static_cast<size_t>(a.wpr) * 4) + (MODE == G8 ? t * (BITS * 2) : t * (BITS * 4));
            srow[j] = static_cast<const char *>(a.scales[lt.second]) + row * (static_cast<size_t>(a.gpr) * ESZ);
            brow[j] = static_cast<const char *>(a.biases[lt.second]) + row * (static_cast<size_t>(a.gpr) * ESZ);
        }
    };
    auto request_words = [&](int i, bool on) {
        if (!on) return;
        const uint32_t off = static_cast<uint32_t>(l_run * RUN + i) * (16 * BITS);
        if (whole) {
            load_words<BITS, MODE>(wrow[0] + off, wl[i]);
            load_words<BITS, MODE>(wrow[1] + off, wh[i]);
        } else {
            const int s = l_run * RUN + i;
            const bool on0 = (MODE == G8 ? 2 * s : 4 * s + t) < n_units, on1 = 2 * s + 1 < n_units;
            load_words<BITS, MODE>(wrow[0] + off, wl[i], on0, on1);
            load_words<BITS, MODE>(wrow[1] + off, wh[i], on0, on1);
        }
    };
    auto request_affine = [&](const char *const (&p)[2], Affine<XT, MODE, RUN, 0> &f, int i, bool on) {
        if (!on) return;
#pragma unroll
        for (int h = 0; h < H; ++h) {
            const int s = l_run * RUN + i;
            const int k = MODE == G8 ? 128 * s + 64 * h : MODE == S4 ? 128 * s + 64 * (t >> 1) : 128 * s + 32 * t;
            const uint32_t off = static_cast<uint32_t>(k >> a.gs_shift) * ESZ;
            const bool in = whole || (MODE == G8 ? 2 * s + h : MODE == S4 ? 4 * s + 2 * (t >> 1) : 4 * s + t) < n_units;
#pragma unroll
            for (int j = 0; j < 2; ++j) ld_scale<XT>(p[j] + off, &f.r[j][i * H + h], in);
        }
    };
    auto advance = [&]() -> bool {   // to the next run of this warp; false: there is none
        if (++l_run == r1) {
            l_run = r0;
            if (++l_tile >= t_hi) return false;
            open_tile();
        }
        whole = (l_run + 1) * (RUN * 128) <= a.K;
        return true;
    };
    bool more = r0 < r1;
    if (more) {
        open_tile();
        whole = (l_run + 1) * (RUN * 128) <= a.K;
#pragma unroll
        for (int i = 0; i < RUN; ++i) {
            request_words(i, true);
            request_affine(srow, sc, i, true);
            request_affine(brow, bi, i, true);
        }
    }

    // ---- activations of this warp's part of K for the rows of a pass ----
    BRegs br;
    const bool on = MODE == S2 ? (g >> 1) == t : MODE == S4 ? (g >> 2) == (t >> 1) : true;
    const int tok_l = MODE == S2 ? g & 1 : MODE == S4 ? g & 3 : g;                 // this lane's token in a tile of columns
    char *const part = smem + a.off_part + warp * a.warp_bytes, *const sums = part + a.off_sum;
    const uint32_t frag0 = static_cast<uint32_t>(__cvta_generic_to_shared(part)) + static_cast<uint32_t>((tok_l * 4 + t) * kPitch<XT>);
    auto stage = [&](const Tile &q) {
        __syncwarp();
        static_assert(32 % (4 * MP) == 0, "a lane stages one token");
        const int em = (lane >> 2) % MP, et = lane & 3, n = (r1 - r0) * RUN * 4 * MP;
        RowX rx{a.x, a.K, em < q.ntok ? 1 : 0};
        if (rx.M) rx.x = row_of(a, q.tok0 + em);
        for (int e0 = 0; e0 < n; e0 += 32) {
            const int e = e0 + lane, es = (e >> 2) / MP, k = (r0 * RUN + es) * 128;
            float sum = 0.0f;
            if (e < n)
                sum = stage_chunk<BITS, XT, MODE, far_tokens::kUp>(rx, 0, MODE == G8 ? k + 16 * et : k + 32 * et, MODE == G8 ? k + 64 + 16 * et : k + 32 * et + 16,
                                                  part + static_cast<size_t>(e) * kPitch<XT>);
            if (MODE != G8) {
                // in the units of the products: x times 2^kUp against codes times 2^-133, f16: codes times 2^-24
                constexpr uint32_t unit = (XT == MTC_F16 ? 127u - 24u : 127u - far_tokens::kUnit) << 23;
                if (MODE == S4) sum += __shfl_xor_sync(0xffffffffu, sum, 1);                       // chunks 0 and 1, 2 and 3
                const uint32_t at = (em / CAP) * 32 + (MODE == S2 ? et * 8 : (et >> 1) * 16) + (em % CAP) * 4;
                if (e < n && (MODE != S4 || !(et & 1))) *reinterpret_cast<float *>(sums + es * SUM + at) = sum * __uint_as_float(unit);
            }
        }
        __syncwarp();
        for (int s = 0; s < (MODE == G8 ? (r1 - r0) * RUN : 0); ++s) {             // G8 adds over the quad: against codes that are all one
            const uint32_t none[BITS] = {};
            float d[NT][H][4];
            step_mma<BITS, XT, MODE, NT, true>(none, none, frag0 + s * STEP, on, br, d);
            if (lane < 4) {
#pragma unroll
                for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                    for (int h = 0; h < H; ++h) reinterpret_cast<float2 *>(sums + s * SUM + (nt * H + h) * 32)[t] = make_float2(d[nt][h][0], d[nt][h][1]);
            }
        }
        __syncwarp();
    };

    // ---- tiles ----
    const float post = XT == MTC_F16 ? __uint_as_float((127u + 24u) << 23) : __uint_as_float((127u + far_tokens::kUnit) << 23);
    float *const red = reinterpret_cast<float *>(smem + a.off_red) + slot * a.ks * (2 * MP * 16);     // [buffer][warp of the slot][token][row]
    int staged = -1, buf = 0;
    bool odd = false;                // a sum that this lane has stored may be of a row out of range (far_tokens.cuh)
    for (int tile = t_lo; tile < t_hi; ++tile) {
        Tile q;
        locate<MP>(a, start, tile, q);
        if (q.pass != staged) {
            stage(q);
            staged = q.pass;
        }
        float acc[NT][4];
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[nt][j] = 0.0f;
        for (int run = r0; run < r1; ++run) {
            more = more && advance();
            const uint32_t at = frag0 + (run - r0) * (RUN * STEP);
            const char *sat = sums + (run - r0) * (RUN * SUM) + t * 8;
#pragma unroll
            for (int i = 0; i < RUN; ++i)
#pragma unroll
                for (int h = 0; h < H; ++h) {
                    const float b_l = bi.get(i, h, 0, t), b_h = bi.get(i, h, 1, t);
#pragma unroll
                    for (int nt = 0; nt < NT; ++nt) {
                        const float2 xs = *reinterpret_cast<const float2 *>(sat + i * SUM + (nt * H + h) * 32);
                        acc[nt][0] = fmaf(b_l, xs.x, acc[nt][0]);
                        acc[nt][1] = fmaf(b_l, xs.y, acc[nt][1]);
                        acc[nt][2] = fmaf(b_h, xs.x, acc[nt][2]);
                        acc[nt][3] = fmaf(b_h, xs.y, acc[nt][3]);
                    }
                }
#pragma unroll
            for (int i = 0; i < RUN; ++i) request_affine(brow, bi, i, more);
#pragma unroll
            for (int i = 0; i < RUN; ++i) {
                float d[NT][H][4];
                step_mma<BITS, XT, MODE, NT, false>(wl[i], wh[i], at + i * STEP, on, br, d);
                request_words(i, more);
#pragma unroll
                for (int h = 0; h < H; ++h) {
                    const float s_l = sc.get(i, h, 0, t), s_h = sc.get(i, h, 1, t);
#pragma unroll
                    for (int nt = 0; nt < NT; ++nt) {
                        acc[nt][0] = fmaf(s_l, d[nt][h][0], acc[nt][0]);
                        acc[nt][1] = fmaf(s_l, d[nt][h][1], acc[nt][1]);
                        acc[nt][2] = fmaf(s_h, d[nt][h][2], acc[nt][2]);
                        acc[nt][3] = fmaf(s_h, d[nt][h][3], acc[nt][3]);
                    }
                }
                request_affine(srow, sc, i, more);
            }
        }
        // this warp's partial tile, then the sum over the slot's warps: [token][16 rows].  Two buffers: one barrier a tile.
        float *mine = red + (buf * a.ks + slice) * (MP * 16);
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                float v = acc[nt][j];
                if (MODE == S2) v += __shfl_xor_sync(0xffffffffu, v, 1);
                if (MODE != G8) v += __shfl_xor_sync(0xffffffffu, v, 2);
                const bool holds = MODE == G8 ? true : MODE == S4 ? t < 2 : t == 0;
                const int tok = nt * CAP + (MODE == G8 || MODE == S4 ? 2 * t : 0) + (j & 1);
                if (holds) mine[tok * 16 + g + (j >> 1) * 8] = v;
            }
        if (a.ks == 1) __syncwarp();
        else asm volatile("bar.sync %0, %1;" ::"r"(slot + 1), "r"(32 * a.ks) : "memory");
        for (int e = slice * 32 + lane; e < q.ntok * 16; e += 32 * a.ks) {
            const int row = e & 15, tok = e >> 4;
            const float *base = red + buf * a.ks * (MP * 16) + e;
            float v = base[0];
            for (int s = 1; s < a.ks; ++s) v += base[s * (MP * 16)];
            if (q.row0 + row < a.n_out) {
                st_from_f32(a.out[q.second], static_cast<size_t>(q.tok0 + tok) * a.n_out + q.row0 + row, v * post, XT);
                odd = odd || far_tokens::odd<XT>(v);
            }
        }
        buf ^= 1;
    }
    if (__any_sync(0xffffffffu, odd)) far_rows<BITS, XT, MP>(a, start, t_lo, t_hi);
}

// ---- host side -----------------------------------------------------------------------------------------------------
struct Plan {
    int ks = 0;
    uint32_t off_sum = 0, off_part = 0, warp_bytes = 0, off_red = 0, smem = 0;
};
constexpr uint32_t kGfSmem = 113 * 1024;

// The split of K depends on nothing but the shape of one product, so that fused and separate calls agree.
inline Plan make_plan(int K, int n_experts, int bits, int mode, int nt) {
    const int cap = mode == S2 ? 2 : mode == S4 ? 4 : 8, mp = cap * nt, run = mode == G8 ? 2 : bits <= 4 ? 4 : 2, runs = ((K + 127) / 128 + run - 1) / run;
    const uint32_t frags = mp * 4 * kPitch<MTC_F16>, sum = nt * (mode == G8 ? 2 : 1) * 32;
    Plan best;
    for (int ks = 1; ks <= kGfWarps; ks <<= 1) {
        if (ks >= 2 * runs && ks > 1) break;               // more than half of the warps would have no run
        Plan p;
        p.ks = ks;
        const int mine = (runs + ks - 1) / ks * run;
        p.off_sum = mine * frags;
        p.warp_bytes = (mine * (frags + sum) + 127) / 128 * 128;
        p.off_part = (static_cast<uint32_t>(n_experts + 1) * 4 + 127) / 128 * 128;
        p.off_red = p.off_part + kGfWarps * p.warp_bytes;
        p.smem = p.off_red + kGfWarps * 2 * mp * 64;
        if (p.smem > kGfSmem) continue;
        best = p;
        if (mine <= 8) break;        // enough warps on a tile: a longer chain of warps only adds sums
    }
    return best;
}

template <int BITS, int XT, int MODE, int NT>
cudaError_t launch_one(cudaStream_t st, const GfArgs &a, const Plan &p, int sms) {
    auto kern = gather_frag_kernel<BITS, XT, MODE, NT>;
    static PerDeviceAttr attr;
    const cudaError_t e = attr.set(kern, kGfSmem);
    return e != cudaSuccess ? e : launch_pdl(kern, 2 * sms, 32 * kGfWarps, p.smem, st, a);
}

struct Shape {
    int mode, nt, xt;
};

template <int BITS, int XT>
cudaError_t launch_type(cudaStream_t st, const GfArgs &a, const Shape &s, const Plan &p, int sms) {
    if (s.mode == S2) {
        if (s.nt == 1) return launch_one<BITS, XT, S2, 1>(st, a, p, sms);
        if (s.nt == 2) return launch_one<BITS, XT, S2, 2>(st, a, p, sms);
        return launch_one<BITS, XT, S2, 4>(st, a, p, sms);
    }
    if (s.mode == S4 && s.nt == 1) return launch_one<BITS, XT, S4, 1>(st, a, p, sms);
    if constexpr (BITS == 4 || BITS == 8) return launch_one<BITS, XT, G8, 1>(st, a, p, sms);
    else return launch_one<BITS, XT, S4, 2>(st, a, p, sms);
}

template <int BITS>
cudaError_t launch_bits(cudaStream_t st, const GfArgs &a, const Shape &s, const Plan &p, int sms) {
    return s.xt == MTC_F16 ? launch_type<BITS, MTC_F16>(st, a, s, p, sms) : launch_type<BITS, MTC_BF16>(st, a, s, p, sms);
}

}  // namespace gfrag

// one translation unit per width (gather_frag_b*.cu)
#define MTC_GF(B) cudaError_t launch_gather_frag_b##B(cudaStream_t, const GfArgs &, const gfrag::Shape &, const gfrag::Plan &, int);
MTC_GF(2) MTC_GF(3) MTC_GF(4) MTC_GF(5) MTC_GF(6) MTC_GF(8)
#undef MTC_GF

}  // namespace mtc
