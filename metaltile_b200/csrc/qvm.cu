// qvm — the quantized vector-matrix product, the dual of qmv: the weight matrix is stored transposed, [K, N], codes packed
// along N, and the groups run along K:
//
//   out[m, c] = sum_d (q(d, c) * scale[d / G, c] + bias[d / G, c]) * x[m, d]
//
// w u32[K, N*bits/32] (row d = LSB-first bit-stream of N codes), scales / biases T[K/G, N], x T[M, K], out T[M, N].
// Stands in for mt_qvm_b{3,4,5,6,8} and mt_qvm_int4_fast (crates/metaltile-std/src/mlx/quantized.rs:4397-4530,4582-4700).
//
// Three kernels: the one described here, one that streams 4- and 8-bit codes through shared memory for one token, and one on the warp-level tensor
// cores for several tokens (below).  All are launched
// while the previous kernel of the stream drains and request their first weights before it is complete (4096 x 14336 4-bit, one
// token, back to back: 16.4 -> 14.5 us).  Every packed word is read once per row of x.  A lane owns the columns of one packed word (2 / 4 / 8-bit:
// 16 / 8 / 4 columns) or of one 32-column period of the bit-stream (3 / 5 / 6-bit: b words), so a warp reads whole
// lines of a weight row; a warp walks whole groups of K rows and uses the algebraic split per group,
//   acc[c] += scale[g, c] * sum_d q(d, c) x[d]  +  bias[g, c] * sum_d x[d],
// the 8 warps of a CTA take different groups of the same column tile and add up in shared memory in a fixed order, and
// K is split over CTAs (partial sums in a context scratch block, added in a fixed order by a second small kernel), so
// results are deterministic.
#include "common.cuh"

namespace mtc {
namespace {

constexpr int kQvWarps = 8;

template <int BITS>
struct QvShape {
    static constexpr bool kStream = BITS == 3 || BITS == 5 || BITS == 6;
    static constexpr int WPT = kStream ? BITS : 1;              // words per lane and weight row
    static constexpr int CPT = kStream ? 32 : 32 / BITS;        // columns per lane
};

// Code j of a lane's words as an unshifted bit field below bit 24, and the position p of its lowest bit there.
template <int BITS>
struct QvCode {
    static constexpr uint32_t MASK = (1u << BITS) - 1u;
    __device__ static constexpr int pos(int j) {
        const int sh = (j * BITS) & 31;
        if (sh + BITS > 32) return 0;                      // straddles two words: assembled at bit 0
        return sh + BITS <= 24 ? sh : sh - 16;             // high fields are taken from the word shifted down by 16
    }
    template <int W>
    __device__ __forceinline__ static uint32_t field(const uint32_t (&w)[W], int j) {      // j: compile-time after unrolling
        const int bit = j * BITS, wi = bit >> 5, sh = bit & 31;
        if (sh + BITS > 32) return ((w[wi] >> sh) | (w[wi + 1] << (32 - sh))) & MASK;
        if (sh + BITS <= 24) return w[wi] & (MASK << sh);
        return (w[wi] >> 16) & (MASK << (sh - 16));
    }
};

constexpr int kQvTickets = 4096;               // arrival counters at the head of the partial-sum block (one per column tile and x row)

// NW consecutive 32-bit words from a 16-byte (NW % 4 == 0) or 8-byte (NW == 2) aligned address: RO = the read-only path (scales and
// biases), else plain loads (activations, which the previous kernel may be writing: pdl_enter)
template <bool RO, int NW>
__device__ __forceinline__ void qv_ld(const void *p, uint32_t (&o)[NW]) {
    static_assert(NW == 2 || NW % 4 == 0, "vector loads of 8 or 16 bytes");
    if (NW == 2) {
        const uint2 *src = static_cast<const uint2 *>(p);
        const uint2 v = RO ? __ldg(src) : *src;
        o[0] = v.x;
        o[1] = v.y;
    } else {
#pragma unroll
        for (int i = 0; i < NW / 4; ++i) {
            const uint4 *src = static_cast<const uint4 *>(p) + i;
            const uint4 v = RO ? __ldg(src) : *src;
            o[4 * i] = v.x; o[4 * i + 1] = v.y; o[4 * i + 2] = v.z; o[4 * i + 3] = v.w;
        }
    }
}
// element i (compile-time after unrolling) of a vector of DT values held as words
template <int DT, int NW>
__device__ __forceinline__ float qv_elem(const uint32_t (&v)[NW], int i) {
    if (DT == MTC_F32) return __uint_as_float(v[i]);
    const uint32_t wd = v[i >> 1];
    if (DT == MTC_BF16) return __uint_as_float((i & 1) ? (wd & 0xFFFF0000u) : (wd << 16));
    const __half2 h = *reinterpret_cast<const __half2 *>(&wd);
    return (i & 1) ? __high2float(h) : __low2float(h);
}

// What a lane needs for one slab of R rows: its packed words of every row, the R activations, and the scales and biases
// of its columns in the slab's group - all fetched with 8- or 16-byte loads before any of it is used.
template <int BITS, int DT>
struct QvSlab {
    using S = QvShape<BITS>;
    static constexpr int R = S::kStream ? 8 : 16;
    static constexpr int ESZ = DT == MTC_F32 ? 4 : 2;
    static constexpr int XW = R * ESZ / 4, SW = S::CPT * ESZ / 4;
    uint32_t w[R][S::WPT];
    uint32_t x[XW], sc[SW], bi[SW];
};

template <int BITS, int DT>
__global__ void __launch_bounds__(kQvWarps * 32, 2) qvm_kernel(const uint32_t *w, const void *scales, const void *biases, const void *x,
                                                               float *partial, uint32_t *tickets, void *out, int M, int N, int K, int gs, int KC, int early) {
    using S = QvShape<BITS>;
    using Slab = QvSlab<BITS, DT>;
    constexpr int R = Slab::R, ESZ = Slab::ESZ;
    __shared__ float red[kQvWarps][32 * S::CPT + 1];
    __shared__ uint32_t s_last;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int tile = blockIdx.x, kc = blockIdx.y, m = blockIdx.z;
    const int col0 = (tile * 32 + lane) * S::CPT;                  // first column of this lane
    const bool on = col0 < N;                                      // N % CPT == 0: a lane is in or out as a whole
    const int wpr = N * BITS / 32, n_groups = K / gs;
    const uint32_t *wl = w + (static_cast<size_t>(tile) * 32 + lane) * S::WPT;
    const char *xrow = static_cast<const char *>(x) + static_cast<size_t>(m) * K * ESZ;
    const char *sc0 = static_cast<const char *>(scales) + static_cast<size_t>(col0) * ESZ;
    const char *bi0 = static_cast<const char *>(biases) + static_cast<size_t>(col0) * ESZ;
    float acc[S::CPT];
#pragma unroll
    for (int j = 0; j < S::CPT; ++j) acc[j] = 0.0f;
    // a warp's unit of work is a slab of R consecutive rows of one group; a matrix has K / R units per column tile to
    // spread over warps and CTAs.  The loads of a warp's next slab are issued before its current slab is multiplied.
    const int upg = gs / R, n_units = n_groups * upg;              // gs % R == 0 (host)
    const int ustep = KC * kQvWarps;
    auto fetch_w = [&](int u, Slab &sl) {
        const int g = u / upg, d0 = g * gs + (u - g * upg) * R;
        const uint32_t *wp = wl + static_cast<size_t>(d0) * wpr;
#pragma unroll
        for (int r = 0; r < R; ++r) {
#pragma unroll
            for (int i = 0; i < S::WPT; ++i) sl.w[r][i] = __ldg(wp + i);
            wp += wpr;
        }
        qv_ld<true, Slab::SW>(sc0 + static_cast<size_t>(g) * N * ESZ, sl.sc);
        qv_ld<true, Slab::SW>(bi0 + static_cast<size_t>(g) * N * ESZ, sl.bi);
    };
    auto fetch_x = [&](int u, Slab &sl) {
        const int g = u / upg, d0 = g * gs + (u - g * upg) * R;
        qv_ld<false, Slab::XW>(xrow + static_cast<size_t>(d0) * ESZ, sl.x);
    };
    auto fetch = [&](int u, Slab &sl) {
        fetch_w(u, sl);
        fetch_x(u, sl);
    };
    if (!early) asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;");
    // weights are constants of the model: the first slab may be requested while the previous kernel of the stream still runs
    const int u0 = kc * kQvWarps + warp;
    Slab sa;
    if (early && on && u0 < n_units) fetch_w(u0, sa);
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (on && u0 < n_units) {
        if (early) fetch_x(u0, sa);
        else fetch(u0, sa);
    }
    // No integer-to-float conversion: the bits of a code, left where they sit in the word (below bit 24), read as an
    // f32 are q * 2^(p - 149) exactly - the subnormals and the first binade are one linear ramp, multiplied at full
    // rate - and x is pre-multiplied by 2^64 (exact; |x| < 2^63) so that products are normal numbers; the factor
    // 2^(85 - p) of column j leaves with the group's scale.  One LOP3 and one FFMA per code.
    auto multiply = [&](const Slab &sl) {
        float raw[S::CPT];
#pragma unroll
        for (int j = 0; j < S::CPT; ++j) raw[j] = 0.0f;
        float xs = 0.0f;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const float xv = qv_elem<DT>(sl.x, r);
            xs += xv;
            const float xp = xv * 18446744073709551616.0f;                   // 2^64
#pragma unroll
            for (int j = 0; j < S::CPT; ++j) raw[j] = fmaf(xp, __uint_as_float(QvCode<BITS>::field(sl.w[r], j)), raw[j]);
        }
#pragma unroll
        for (int j = 0; j < S::CPT; ++j) {
            const float post = __uint_as_float(static_cast<uint32_t>(127 + 85 - QvCode<BITS>::pos(j)) << 23);     // 2^(85 - p)
            acc[j] = fmaf(qv_elem<DT>(sl.sc, j) * post, raw[j], fmaf(qv_elem<DT>(sl.bi, j), xs, acc[j]));
        }
    };
    if (on) {
        int u = u0;
        if (S::kStream || BITS == 2) {                             // 3 / 5 / 6-bit (b words per row) and 2-bit (16 columns): one slab in registers
            while (u < n_units) {
                multiply(sa);
                u += ustep;
                if (u < n_units) fetch(u, sa);
            }
        } else if (u < n_units) {
            Slab sb;
            for (;;) {
                u += ustep;
                if (u < n_units) fetch(u, sb);
                multiply(sa);
                if (u >= n_units) break;
                u += ustep;
                if (u < n_units) fetch(u, sa);
                multiply(sb);
                if (u >= n_units) break;
            }
        }
    }
#pragma unroll
    for (int j = 0; j < S::CPT; ++j) red[warp][j * 32 + lane] = acc[j];
    __syncthreads();
    // column (tile * 32 + l) * CPT + j of the tile: summed over the warps in warp order
    for (int idx = threadIdx.x; idx < 32 * S::CPT; idx += kQvWarps * 32) {
        const int j = idx >> 5, l = idx & 31;
        const int c = (tile * 32 + l) * S::CPT + j;
        if (c >= N) continue;
        float v = 0.0f;
#pragma unroll
        for (int q = 0; q < kQvWarps; ++q) v += red[q][idx];
        if (KC == 1) st_from_f32(out, static_cast<size_t>(m) * N + c, v, DT);
        else partial[(static_cast<size_t>(kc) * M + m) * N + c] = v;
    }
    if (KC == 1 || tickets == nullptr) return;
    // K chunks: the CTA that arrives last for (column tile, x row) adds the chunks in chunk order (deterministic) and
    // leaves the counter at zero for the next launch.  Nothing waits for anything.
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        const uint32_t old = atomicAdd(tickets + static_cast<size_t>(m) * gridDim.x + tile, 1u);
        s_last = old == static_cast<uint32_t>(KC - 1) ? 1u : 0u;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    for (int idx = threadIdx.x; idx < 32 * S::CPT; idx += kQvWarps * 32) {
        const int j = idx >> 5, l = idx & 31;
        const int c = (tile * 32 + l) * S::CPT + j;
        if (c >= N) continue;
        float v = 0.0f;
        const float *src = partial + static_cast<size_t>(m) * N + c;
        const size_t stride = static_cast<size_t>(M) * N;
        float pv[32];                                              // KC <= 32: every load in flight, added in chunk order
#pragma unroll
        for (int i = 0; i < 32; ++i) pv[i] = i < KC ? __ldcg(src + i * stride) : 0.0f;
#pragma unroll
        for (int i = 0; i < 32; ++i) v += pv[i];
        st_from_f32(out, static_cast<size_t>(m) * N + c, v, DT);
    }
    if (threadIdx.x == 0) tickets[static_cast<size_t>(m) * gridDim.x + tile] = 0u;
}

// ---- one token, 4- and 8-bit codes ----------------------------------------------------------------------------------------------
// The same arithmetic with the packed words on their way through shared memory.  Above, a warp has one or two slabs in flight and waits between
// them, with 3 instructions a code beside.  Here a warp owns a contiguous range of units (16 rows of 128 bytes) of its CTA's chunk of K and keeps four of
// them in flight with 16-byte asynchronous copies; x waits as f32 times 2^64 beside the sum of every unit, so a code costs one LOP3, one FFMA and a
// quarter of an instruction more, and scales are applied once a group (f32: once a unit) to the sum of its units' sums, from registers that were loaded when the group began.  One CTA of 16 warps
// an SM, which has the SM's shared memory to itself: with room for two, CTAs land in pairs and leave SMs idle (17.9 us for the first shape below), and
// two or three CTAs of 8 warps in twice or three times as many chunks of K pay more for start and sum (13.5, 14.4).  Six units in flight: 14.0; 24 warps:
// 13.8.  bf16, 4-bit groups of 64, K x N 14336 x 4096 14.8 -> 13.2 us, 4096 x 4096 7.5 -> 7.0, 4096 x 14336 14.7 -> 13.0, 16384 x 16384 52.4 -> 36.3 (4.2
// TB/s), 8-bit 8192 x 8192 22.8 -> 15.4 (4.6 TB/s), 2048 x 16384 13.8 -> 9.0.  Bound by the ALU pipe and the start and end of the launch.
constexpr int kQrDepth = 4, kQrRows = 16, kQrWarps = 16;      // units in flight a warp, rows of a unit
constexpr int kQrRing = kQrWarps * kQrDepth * kQrRows * 128;
constexpr int kQrMaxUnits = (226 * 1024 - kQrRing) / ((kQrRows + 1) * 4);                            // of a CTA: their x fit beside the ring
constexpr int qr_smem(int units) { return kQrRing + units * (kQrRows + 1) * 4; }

// The end of a CTA as in the kernel above (which keeps its own: with a shared one its 2-bit f32 form took 1.14 times as long): its warps' sums red[warp][column j of lane l at j * 32 + l] added in warp order, then the chunks of K.
template <int CPT, int DT, int WARPS>
__device__ __forceinline__ void qv_finish(const float *red, int pitch, uint32_t *s_last, float *partial, uint32_t *tickets, void *out, int M, int N, int KC) {
    const int tile = blockIdx.x, kc = blockIdx.y, m = blockIdx.z;
    // column (tile * 32 + l) * CPT + j of the tile: summed over the warps in warp order
    for (int idx = threadIdx.x; idx < 32 * CPT; idx += WARPS * 32) {
        const int j = idx >> 5, l = idx & 31;
        const int c = (tile * 32 + l) * CPT + j;
        if (c >= N) continue;
        float v = 0.0f;
#pragma unroll
        for (int q = 0; q < WARPS; ++q) v += red[q * pitch + idx];
        if (KC == 1) st_from_f32(out, static_cast<size_t>(m) * N + c, v, DT);
        else partial[(static_cast<size_t>(kc) * M + m) * N + c] = v;
    }
    if (KC == 1 || tickets == nullptr) return;
    // K chunks: the CTA that arrives last for (column tile, x row) adds the chunks in chunk order (deterministic) and
    // leaves the counter at zero for the next launch.  Nothing waits for anything.
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        const uint32_t old = atomicAdd(tickets + static_cast<size_t>(m) * gridDim.x + tile, 1u);
        *s_last = old == static_cast<uint32_t>(KC - 1) ? 1u : 0u;
    }
    __syncthreads();
    if (!*s_last) return;
    __threadfence();
    for (int idx = threadIdx.x; idx < 32 * CPT; idx += WARPS * 32) {
        const int j = idx >> 5, l = idx & 31;
        const int c = (tile * 32 + l) * CPT + j;
        if (c >= N) continue;
        float v = 0.0f;
        const float *src = partial + static_cast<size_t>(m) * N + c;
        const size_t stride = static_cast<size_t>(M) * N;
        float pv[32];                                              // KC <= 32: every load in flight, added in chunk order
#pragma unroll
        for (int i = 0; i < 32; ++i) pv[i] = i < KC ? __ldcg(src + i * stride) : 0.0f;
#pragma unroll
        for (int i = 0; i < 32; ++i) v += pv[i];
        st_from_f32(out, static_cast<size_t>(m) * N + c, v, DT);
    }
    if (threadIdx.x == 0) tickets[static_cast<size_t>(m) * gridDim.x + tile] = 0u;
}

template <int BITS, int DT>
__global__ void __launch_bounds__(kQrWarps * 32, 1) qvm_ring_kernel(const uint32_t *w, const void *scales, const void *biases, const void *x,
                                                                     float *partial, uint32_t *tickets, void *out, int M, int N, int K, int gs, int KC, int early) {
    constexpr int CPT = 32 / BITS, ESZ = DT == MTC_F32 ? 4 : 2, SW = CPT * ESZ / 4, D = kQrDepth, R = kQrRows;
    extern __shared__ __align__(16) unsigned char qr_raw[];
    __shared__ uint32_t s_last;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int tile = blockIdx.x, kc = blockIdx.y, m = blockIdx.z;
    const int col0 = (tile * 32 + lane) * CPT;
    const bool on = col0 < N;                                      // N % CPT == 0: a lane is in or out as a whole
    const int wpr = N * BITS / 32, units = K / R, upg = gs / R;    // gs % 16 == 0, wpr % 4 == 0 (host)
    const int c0 = static_cast<int>(static_cast<long long>(units) * kc / KC), nu = static_cast<int>(static_cast<long long>(units) * (kc + 1) / KC) - c0;
    const int u0 = c0 + nu * warp / kQrWarps, u1 = c0 + nu * (warp + 1) / kQrWarps;
    float *sx = reinterpret_cast<float *>(qr_raw + kQrRing), *ssum = sx + nu * R;
    const uint32_t *ring = reinterpret_cast<const uint32_t *>(qr_raw) + warp * (D * R * 32) + lane;
    const uint32_t dst0 = static_cast<uint32_t>(__cvta_generic_to_shared(qr_raw)) + warp * (D * R * 128) + lane * 16;
    const int piece = tile * 32 + (lane & 7) * 4;
    const uint32_t bytes = piece < wpr ? 16u : 0u;
    const char *src = reinterpret_cast<const char *>(w + static_cast<size_t>(u0 * R + (lane >> 3)) * wpr + (bytes ? piece : 0));
    const size_t step = static_cast<size_t>(wpr) * 16;             // bytes of four rows
    int slot_in = 0, next = u0;
    auto fetch = [&]() {                                           // a group per call, so that waits count units
        if (next < u1) {
            const uint32_t dst = dst0 + slot_in * (R * 128);
#pragma unroll
            for (int i = 0; i < R / 4; ++i)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + i * 512), "l"(src + i * step), "r"(bytes) : "memory");
            src += (R / 4) * step;
            ++next;
            if (++slot_in == D) slot_in = 0;
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    if (!early) asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;");
    // weights are constants of the model: requested while the previous kernel of the stream still runs
#pragma unroll
    for (int i = 0; i < D; ++i) fetch();
    const char *sc = static_cast<const char *>(scales) + static_cast<size_t>(on ? col0 : 0) * ESZ, *bi = static_cast<const char *>(biases) + static_cast<size_t>(on ? col0 : 0) * ESZ;
    const size_t srow = static_cast<size_t>(N) * ESZ;
    int g = u0 / upg, left = upg - (u0 - g * upg);                 // group, units to its end
    uint32_t sv[SW], bv[SW];
    if (u0 < u1) {
        qv_ld<true, SW>(sc + g * srow, sv);
        qv_ld<true, SW>(bi + g * srow, bv);
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
    for (int i = threadIdx.x; i < nu * (R / 4); i += kQrWarps * 32) {      // four values a thread, whole units by four lanes
        const unsigned who = __activemask();
        constexpr int XW = ESZ;
        uint32_t xw[XW];
        qv_ld<false, XW>(static_cast<const char *>(x) + (static_cast<size_t>(m) * K + static_cast<size_t>(c0) * R + 4 * i) * ESZ, xw);
        const float v0 = qv_elem<DT>(xw, 0), v1 = qv_elem<DT>(xw, 1), v2 = qv_elem<DT>(xw, 2), v3 = qv_elem<DT>(xw, 3), up = 18446744073709551616.0f;       // 2^64: see multiply above
        *reinterpret_cast<float4 *>(sx + 4 * i) = make_float4(v0 * up, v1 * up, v2 * up, v3 * up);
        float t = (v0 + v1) + (v2 + v3);
        t += __shfl_xor_sync(who, t, 1);
        t += __shfl_xor_sync(who, t, 2);
        if ((i & 3) == 0) ssum[i / 4] = t;
    }
    __syncthreads();
    float acc[CPT], of_group[CPT], xs = 0.0f;
#pragma unroll
    for (int j = 0; j < CPT; ++j) acc[j] = of_group[j] = 0.0f;
    int slot = 0;
    for (int u = u0; u < u1; ++u) {
        asm volatile("cp.async.wait_group %0;" ::"n"(D - 1) : "memory");
        __syncwarp();
        const uint32_t *wp = ring + slot * (R * 32);
        const float *xp = sx + (u - c0) * R;
        uint32_t wd[R][1];
#pragma unroll
        for (int r = 0; r < R; ++r) wd[r][0] = wp[r * 32];
        __syncwarp();
        fetch();                                                   // the slot is in registers
        float raw[CPT];
#pragma unroll
        for (int j = 0; j < CPT; ++j) raw[j] = 0.0f;
#pragma unroll
        for (int r4 = 0; r4 < R; r4 += 4) {
            const float4 xv = *reinterpret_cast<const float4 *>(xp + r4);
            const float xr[4] = {xv.x, xv.y, xv.z, xv.w};
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int j = 0; j < CPT; ++j) raw[j] = fmaf(xr[r], __uint_as_float(QvCode<BITS>::field(wd[r4 + r], j)), raw[j]);
        }
        xs += ssum[u - c0];
        if (++slot == D) slot = 0;
        const bool end = --left == 0 || u + 1 == u1;
        // sums of codes are those of a unit, as above (f32 with a whole group of them: the error against 64 bits was 1.1 to 2 times as large)
#pragma unroll
        for (int j = 0; j < CPT; ++j) of_group[j] = DT == MTC_F32 ? raw[j] : of_group[j] + raw[j];
        if (DT == MTC_F32 || end) {
#pragma unroll
            for (int j = 0; j < CPT; ++j) {
                const float post = __uint_as_float(static_cast<uint32_t>(127 + 85 - QvCode<BITS>::pos(j)) << 23);     // 2^(85 - p)
                acc[j] = fmaf(qv_elem<DT>(sv, j) * post, of_group[j], fmaf(qv_elem<DT>(bv, j), xs, acc[j]));
                of_group[j] = 0.0f;
            }
            xs = 0.0f;
        }
        if (end) {
            left = upg;
            if (u + 1 < u1) {
                ++g;
                qv_ld<true, SW>(sc + g * srow, sv);
                qv_ld<true, SW>(bi + g * srow, bv);
            }
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();                                               // the ring's place holds the warps' sums
    float *red = reinterpret_cast<float *>(qr_raw);
    constexpr int PITCH = 32 * CPT;
#pragma unroll
    for (int j = 0; j < CPT; ++j) red[warp * PITCH + j * 32 + lane] = acc[j];
    __syncthreads();
    qv_finish<CPT, DT, kQrWarps>(red, PITCH, &s_last, partial, tickets, out, M, N, KC);
}

__global__ void __launch_bounds__(256) qvm_sum_kernel(const float *partial, void *out, size_t mn, int KC, int dt) {
    for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < mn; i += static_cast<size_t>(gridDim.x) * blockDim.x) {
        float v = 0.0f;
        for (int q0 = 0; q0 < KC; q0 += 8) {                       // eight loads in flight, added in chunk order
            float pv[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) pv[j] = q0 + j < KC ? partial[static_cast<size_t>(q0 + j) * mn + i] : 0.0f;
#pragma unroll
            for (int j = 0; j < 8; ++j) v += pv[j];
        }
        st_from_f32(out, i, v, dt);
    }
}

// any N, any group size: one thread per output element, rows of w walked one by one
__global__ void __launch_bounds__(256) qvm_generic_kernel(const uint32_t *w, const void *scales, const void *biases, const void *x,
                                                          void *out, int M, int N, int K, int gs, int bits, int dt) {
    const size_t mn = static_cast<size_t>(M) * N, wpr = static_cast<size_t>(N) * bits / 32;
    for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < mn; i += static_cast<size_t>(gridDim.x) * blockDim.x) {
        const int m = static_cast<int>(i / N), c = static_cast<int>(i - static_cast<size_t>(m) * N);
        float acc = 0.0f;
        for (int d = 0; d < K; ++d) {
            const float q = static_cast<float>(code_at(w + d * wpr, static_cast<uint32_t>(c), bits));
            const size_t si = static_cast<size_t>(d / gs) * N + c;
            acc = fmaf(fmaf(q, ld_as_f32(scales, si, dt), ld_as_f32(biases, si, dt)), ld_as_f32(x, static_cast<size_t>(m) * K + d, dt), acc);
        }
        st_from_f32(out, i, acc, dt);
    }
}

// ---- 2 / 4 / 8-bit codes under 16-bit activations: the tensor cores --------------------------------------------------
// One LOP3 and one FFMA per code (the kernel above) are 2.7 issue slots a code with everything around them, about the time of
// the bytes, and a row of x more is all of it again.  Here a word masked in place is an MMA operand: a 16-bit float whose
// exponent field is 0 or 1 is linear in its low bits, so `word & 0x000F000F` (then << 4, and both after >> 8) holds the codes
// of columns c and c + 4 as two exact values.  They belong to different columns but the same row of K, so:
//   * an MMA (m16n8k16) has as its rows 8 words x 2 column classes of the word, as its k positions 8 rows of K x the two halves;
//   * its 8 result columns are 4 slots x (low half, high half): x[d] stands in the low half of even columns and in the
//     high half of odd ones, zero elsewhere, so a lane's two results of a row are the sums of its low and high columns;
//   * the 4 slots are MP tokens x 4 / MP ranges of K (MP = 1, 2, 4): for one token lane t of a quad ends with the sums
//     of the t-th range, and applies only that range's scales to them - no work is repeated over the quad.
// A slab is 32 rows of K x the columns of a warp (WPL words a lane): lane (g, t) copies rows 8t .. 8t+7 of its own
// columns with cp.async and is the only one to read them, so no barrier stands between the loads and the products.
// What bounds it: latency.  A warp has four slabs or fewer to do and 16 of them an SM at 128 registers issue 0.3 instructions a
// clock; a slab costs 1.2 issue slots a code whatever the number of tokens.  14336 x 4096 4-bit groups of 64, bf16, 2 / 4 tokens:
// 25.3 / 45.4 us in the kernel above, 17.5 / 22.4 us here.
constexpr int kQmWarps = 16;

template <int BITS>
struct QmShape {
    static constexpr int WPL = BITS == 2 ? 2 : 4;                  // words per lane and row
    static constexpr int CPW = 32 / BITS;                          // columns per word
    static constexpr int CPL = WPL * CPW;                          // columns per lane
    static constexpr int NP = BITS == 8 ? 1 : BITS == 4 ? 2 : 4;   // MMAs (pairs of column classes) per word
    static constexpr int COLS = 8 * CPL;                           // columns of a CTA
    static constexpr int SCH = CPL / 8;                            // 16-byte chunks of a lane's scales
    static constexpr int W_BYTES = 8 * 32 * WPL * 4, X_BYTES = 32 * 16, SC_BYTES = 2 * SCH * 32 * 16;
    static constexpr int STAGE = W_BYTES + X_BYTES;
    static constexpr int WARP_BYTES = 2 * STAGE + SC_BYTES;
    static constexpr int SMEM = kQmWarps * WARP_BYTES;
    static_assert(SMEM >= kQmWarps * COLS * 4 * 4, "the partial sums of four tokens take the place of the slabs");
    // class cl of a word: columns cl and cl + CPW / 2, at bit pos of each half after the shift
    __host__ __device__ static constexpr int pos(int cl) { return BITS == 8 ? 0 : BITS == 4 ? 4 * (cl & 1) : 2 * (cl & 3); }
    __device__ __forceinline__ static uint32_t field(uint32_t w, int cl) {
        const uint32_t m = ((1u << BITS) - 1u) * 0x10001u;
        return (cl >= NP ? w >> 8 : w) & (m << pos(cl));
    }
};

__device__ __forceinline__ void qm_cp16(uint32_t dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void qm_cp8(uint32_t dst, const void *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}

template <int DT>
__device__ __forceinline__ void qm_mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    if (DT == MTC_BF16)
        asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
            : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
    else
        asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
            : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

struct QmArgs {
    const uint32_t *w;
    const void *scales, *biases, *x;
    float *partial;
    uint32_t *tickets;
    void *out;
    int M, N, K, gs, KC;
    int ch_log2, bs;             // slabs of a range (within one group) as a power of two, slabs of a batch (at most 4 / MP ranges)
    int slabs, batches;
    int early;                   // weights may be read before the previous kernel of the stream is complete
};

template <int BITS, int DT, int MP>
__global__ void __launch_bounds__(kQmWarps * 32, 1) qvm_mma_kernel(const QmArgs a) {
    using S = QmShape<BITS>;
    constexpr bool BF = DT == MTC_BF16;
    extern __shared__ __align__(16) char smem[];
    __shared__ uint32_t s_last;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    const int tile = blockIdx.x, kc = blockIdx.y, m0 = blockIdx.z * MP;
    const int col0 = tile * S::COLS + g * S::CPL;                  // N is a multiple of CPL: a lane's columns exist or not as a whole
    const bool on = col0 < a.N;
    const size_t wpr = static_cast<size_t>(a.N) * BITS / 32;
    char *const mine = smem + warp * S::WARP_BYTES;
    const uint32_t mine_s = static_cast<uint32_t>(__cvta_generic_to_shared(mine));
    constexpr uint32_t SC_OFF = 2 * S::STAGE;
    // as a source of x this lane stands for column g of the MMA: slot g >> 1 (token, range), half g & 1
    const int x_tok = m0 + (g >> 1) % MP, x_rng = (g >> 1) / MP;
    const char *xrow = static_cast<const char *>(a.x) + (static_cast<size_t>(x_tok) * a.K + 8 * t) * 2;
    const bool x_on = x_tok < a.M;
    // as a holder of results it stands for slot t
    const int r_rng = t / MP;
    const uint32_t *wl = a.w + static_cast<size_t>(8 * t) * wpr + static_cast<size_t>(col0) / S::CPW;

    const int stride = a.KC * kQmWarps;
    struct At { int b, j, cnt; };
    auto batch_at = [&](int b) { return At{b, 0, b < a.batches ? min(a.bs, a.slabs - b * a.bs) : 0}; };
    auto next = [&](const At &c) { return c.j + 1 < c.cnt ? At{c.b, c.j + 1, c.cnt} : batch_at(c.b + stride); };
    auto issue_w = [&](const At &c, int stage) {
        if (c.cnt > 0) {
            const int slab = c.b * a.bs + c.j;
            const uint32_t dst = mine_s + stage * S::STAGE;
            if (on) {
                const uint32_t *src = wl + static_cast<size_t>(slab) * 32 * wpr;
#pragma unroll
                for (int r = 0; r < 8; ++r) {
                    if (S::WPL == 4) qm_cp16(dst + (r * 32 + lane) * 16, src);
                    else qm_cp8(dst + (r * 32 + lane) * 8, src);
                    src += wpr;
                }
            }
        }
    };
    auto issue_x = [&](const At &c, int stage) {
        if (c.cnt > 0 && x_on && x_rng == c.j >> a.ch_log2)
            qm_cp16(mine_s + stage * S::STAGE + S::W_BYTES + lane * 16, xrow + static_cast<size_t>(c.b * a.bs + c.j) * 64);
    };
    auto issue_scales = [&](const At &c) {                         // those of range r_rng of the batch
        const int slab = c.b * a.bs + (r_rng << a.ch_log2);
        if (on && c.cnt > (r_rng << a.ch_log2)) {
            const size_t at = (static_cast<size_t>(slab * 32 / a.gs) * a.N + col0) * 2;
#pragma unroll
            for (int i = 0; i < S::SCH; ++i) {
                qm_cp16(mine_s + SC_OFF + (i * 32 + lane) * 16, static_cast<const char *>(a.scales) + at + 16 * i);
                qm_cp16(mine_s + SC_OFF + ((S::SCH + i) * 32 + lane) * 16, static_cast<const char *>(a.biases) + at + 16 * i);
            }
        }
    };

    float acc[S::CPL];
#pragma unroll
    for (int c = 0; c < S::CPL; ++c) acc[c] = 0.0f;
    At cur = batch_at(kc + a.KC * warp), ahead = next(cur);
    if (!a.early) asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;");
    // weights are constants of the model: the first slabs may be requested while the previous kernel of the stream still runs
    issue_w(cur, 0);
    issue_w(ahead, 1);
    issue_scales(cur);                                             // later batches: with the slab after their first one
    if (a.early) asm volatile("griddepcontrol.wait;" ::: "memory");
    if (cur.cnt > 0) {
        float raw[S::WPL][S::NP][4], xs[4];
        auto clear = [&]() {
#pragma unroll
            for (int i = 0; i < S::WPL; ++i)
#pragma unroll
                for (int q = 0; q < S::NP; ++q)
#pragma unroll
                    for (int v = 0; v < 4; ++v) raw[i][q][v] = 0.0f;
#pragma unroll
            for (int v = 0; v < 4; ++v) xs[v] = 0.0f;
        };
        clear();
        issue_x(cur, 0);
        asm volatile("cp.async.commit_group;" ::: "memory");
        issue_x(ahead, 1);
        asm volatile("cp.async.commit_group;" ::: "memory");
        for (int n = 0; cur.cnt > 0; ++n) {
            const int stage = n & 1;
            const bool last = cur.j + 1 == cur.cnt;
            if (last && cur.j == 0) asm volatile("cp.async.wait_group 0;" ::: "memory");       // its scales came with the next slab
            else asm volatile("cp.async.wait_group 1;" ::: "memory");
            const char *st = mine + stage * S::STAGE;
            uint32_t bx[8];
            if (x_on && x_rng == cur.j >> a.ch_log2) {
                const uint4 xv = *reinterpret_cast<const uint4 *>(st + S::W_BYTES + lane * 16);
                const uint32_t x2[4] = {xv.x, xv.y, xv.z, xv.w};
#pragma unroll
                for (int r = 0; r < 8; ++r) {
                    if (BF) {                                      // times 2^64, exact: products with q * 2^(p - 133) are normal numbers
                        const float f = __uint_as_float((r & 1) ? (x2[r >> 1] & 0xFFFF0000u) : (x2[r >> 1] << 16)) * 18446744073709551616.0f;
                        bx[r] = __float_as_uint(f) >> ((g & 1) ? 0 : 16);
                    } else {
                        bx[r] = ((r & 1) ? x2[r >> 1] >> 16 : x2[r >> 1] & 0xFFFFu) << ((g & 1) ? 16 : 0);
                    }
                }
            } else {
#pragma unroll
                for (int r = 0; r < 8; ++r) bx[r] = 0u;
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                uint32_t wa[S::WPL], wb[S::WPL];
                if (S::WPL == 4) {
                    const uint4 va = *reinterpret_cast<const uint4 *>(st + ((2 * j) * 32 + lane) * 16);
                    const uint4 vb = *reinterpret_cast<const uint4 *>(st + ((2 * j + 1) * 32 + lane) * 16);
                    wa[0] = va.x; wa[1] = va.y; wa[S::WPL - 2] = va.z; wa[S::WPL - 1] = va.w;
                    wb[0] = vb.x; wb[1] = vb.y; wb[S::WPL - 2] = vb.z; wb[S::WPL - 1] = vb.w;
                } else {
                    const uint2 va = *reinterpret_cast<const uint2 *>(st + ((2 * j) * 32 + lane) * 8);
                    const uint2 vb = *reinterpret_cast<const uint2 *>(st + ((2 * j + 1) * 32 + lane) * 8);
                    wa[0] = va.x; wa[1] = va.y;
                    wb[0] = vb.x; wb[1] = vb.y;
                }
                qm_mma<DT>(xs, 0x00010001u, 0x00010001u, 0x00010001u, 0x00010001u, bx[2 * j], bx[2 * j + 1]);      // the sums of x: codes that are all one
#pragma unroll
                for (int i = 0; i < S::WPL; ++i)
#pragma unroll
                    for (int q = 0; q < S::NP; ++q)
                        qm_mma<DT>(raw[i][q], S::field(wa[i], 2 * q), S::field(wa[i], 2 * q + 1), S::field(wb[i], 2 * q), S::field(wb[i], 2 * q + 1),
                                   bx[2 * j], bx[2 * j + 1]);
            }
            if (last) {
                if (cur.cnt > (r_rng << a.ch_log2) && on) {                // else this slot's range does not exist: its sums are zero, its scales unset
                    constexpr int E = BF ? 69 : 24;                // 2^(133 - 64), 2^24
                    const float xsum = xs[0] * __uint_as_float((127u + E) << 23);
#pragma unroll
                    for (int cc = 0; cc < S::SCH; ++cc) {
                        const uint4 sv = *reinterpret_cast<const uint4 *>(mine + SC_OFF + (cc * 32 + lane) * 16);
                        const uint4 bv = *reinterpret_cast<const uint4 *>(mine + SC_OFF + ((S::SCH + cc) * 32 + lane) * 16);
                        const uint32_t s4[4] = {sv.x, sv.y, sv.z, sv.w}, b4[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
                        for (int e = 0; e < 8; ++e) {
                            const int c = cc * 8 + e, i = c / S::CPW, k = c % S::CPW;
                            const int half = k / (S::CPW / 2), cl = k % (S::CPW / 2);
                            const float post = __uint_as_float(static_cast<uint32_t>(127 + E - S::pos(cl)) << 23);
                            acc[c] = fmaf(qv_elem<DT>(s4, e) * post, raw[i][cl >> 1][(cl & 1) * 2 + half], fmaf(qv_elem<DT>(b4, e), xsum, acc[c]));
                        }
                    }
                }
                clear();
            }
            cur = ahead;
            ahead = next(ahead);
            issue_w(ahead, stage);
            issue_x(ahead, stage);
            if (cur.cnt > 0 && cur.j == 0) issue_scales(cur);
            asm volatile("cp.async.commit_group;" ::: "memory");
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    // one token: the four ranges of a quad are added, lane t keeping CPL / 4 of the columns; two: two ranges, CPL / 2
    constexpr int KEEP = S::CPL / (4 / MP);
    if (MP <= 2) {
        constexpr int H = S::CPL / 2;
        const bool up = t & 2;
#pragma unroll
        for (int c = 0; c < H; ++c) {
            const float give = up ? acc[c] : acc[c + H], keep = up ? acc[c + H] : acc[c];
            acc[c] = keep + __shfl_xor_sync(0xffffffffu, give, 2);
        }
    }
    if (MP == 1) {
        constexpr int H = S::CPL / 4;
        const bool up = t & 1;
#pragma unroll
        for (int c = 0; c < H; ++c) {
            const float give = up ? acc[c] : acc[c + H], keep = up ? acc[c + H] : acc[c];
            acc[c] = keep + __shfl_xor_sync(0xffffffffu, give, 1);
        }
    }
    const int tok = t % MP;
    const int keep0 = g * S::CPL + (MP == 1 ? (t >> 1) * (S::CPL / 2) + (t & 1) * (S::CPL / 4) : MP == 2 ? (t >> 1) * (S::CPL / 2) : 0);
    __syncthreads();                                               // the slabs are consumed: their place takes the partial sums
    float *red = reinterpret_cast<float *>(smem);
    // [warp][token][position]: positions of a lane are KEEP apart, which would be a bank conflict of KEEP: they stand permuted, element e of all lanes together
    constexpr int PER = S::COLS / KEEP;                            // lanes that hold a token's columns
    const int slot = keep0 / KEEP;
#pragma unroll
    for (int e = 0; e < KEEP; ++e) red[((warp * MP + tok) * KEEP + e) * PER + slot] = acc[e];
    __syncthreads();
    const int active = min(kQmWarps, (a.batches - kc + a.KC - 1) / a.KC);        // warps that had a batch
    for (int idx = threadIdx.x; idx < MP * S::COLS; idx += kQmWarps * 32) {
        const int tk = idx / S::COLS, c = idx - tk * S::COLS, n = tile * S::COLS + c;
        if (n >= a.N || m0 + tk >= a.M) continue;
        float v = 0.0f;
        const float *src = red + (tk * KEEP + c % KEEP) * PER + c / KEEP;
        for (int q = 0; q < active; ++q) v += src[q * MP * S::COLS];
        const size_t at = static_cast<size_t>(m0 + tk) * a.N + n;
        if (a.KC == 1) st_from_f32(a.out, at, v, DT);
        else a.partial[static_cast<size_t>(kc) * a.M * a.N + at] = v;
    }
    if (a.KC == 1 || a.tickets == nullptr) return;
    // the CTA that arrives last for (column tile, tokens) adds the chunks in chunk order and leaves the counter at zero
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        const uint32_t old = atomicAdd(a.tickets + static_cast<size_t>(blockIdx.z) * gridDim.x + tile, 1u);
        s_last = old == static_cast<uint32_t>(a.KC - 1) ? 1u : 0u;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    for (int idx = threadIdx.x; idx < MP * S::COLS; idx += kQmWarps * 32) {
        const int tk = idx / S::COLS, n = tile * S::COLS + idx - tk * S::COLS;
        if (n >= a.N || m0 + tk >= a.M) continue;
        const size_t at = static_cast<size_t>(m0 + tk) * a.N + n, step = static_cast<size_t>(a.M) * a.N;
        float v = 0.0f;
        float pv[32];                                              // KC <= 32: every load in flight
#pragma unroll
        for (int i = 0; i < 32; ++i) pv[i] = i < a.KC ? __ldcg(a.partial + at + i * step) : 0.0f;
#pragma unroll
        for (int i = 0; i < 32; ++i) v += pv[i];
        st_from_f32(a.out, at, v, DT);
    }
    if (threadIdx.x == 0) a.tickets[static_cast<size_t>(blockIdx.z) * gridDim.x + tile] = 0u;
}

int qm_cols(int bits) { return bits == 8 ? QmShape<8>::COLS : bits == 4 ? QmShape<4>::COLS : QmShape<2>::COLS; }

template <int BITS, int DT, int MP>
cudaError_t qm_go(cudaStream_t st, const QmArgs &a) {
    using S = QmShape<BITS>;
    static PerDeviceAttr attr;
    cudaError_t e = attr.set(qvm_mma_kernel<BITS, DT, MP>, S::SMEM);
    if (e != cudaSuccess) return e;
    const dim3 grid((a.N + S::COLS - 1) / S::COLS, a.KC, (a.M + MP - 1) / MP);
    return launch_pdl(qvm_mma_kernel<BITS, DT, MP>, grid, kQmWarps * 32, S::SMEM, st, a);
}
template <int BITS>
cudaError_t qm_launch(cudaStream_t st, const QmArgs &a, int dt) {
    if (dt == MTC_F16) return a.M == 1 ? qm_go<BITS, MTC_F16, 1>(st, a) : a.M == 2 ? qm_go<BITS, MTC_F16, 2>(st, a) : qm_go<BITS, MTC_F16, 4>(st, a);
    return a.M == 1 ? qm_go<BITS, MTC_BF16, 1>(st, a) : a.M == 2 ? qm_go<BITS, MTC_BF16, 2>(st, a) : qm_go<BITS, MTC_BF16, 4>(st, a);
}

template <int BITS, int DT>
cudaError_t qr_go(cudaStream_t st, dim3 grid, const uint32_t *w, const void *scales, const void *biases, const void *x, float *partial, uint32_t *tickets,
                  void *out, int M, int N, int K, int gs, int KC, int early) {
    static PerDeviceAttr attr;
    cudaError_t e = attr.set(qvm_ring_kernel<BITS, DT>, qr_smem(kQrMaxUnits));
    if (e != cudaSuccess) return e;
    const int units = (K / kQrRows + KC - 1) / KC;
    return launch_pdl(qvm_ring_kernel<BITS, DT>, grid, kQrWarps * 32, qr_smem(units), st, w, scales, biases, x, partial, tickets, out, M, N, K, gs, KC, early);
}
template <int BITS>
cudaError_t qr_launch(cudaStream_t st, const void *w, const void *scales, const void *biases, const void *x, float *partial,
                      uint32_t *tickets, void *out, int M, int N, int K, int gs, int KC, int dt, int early) {
    constexpr int COLS = 32 * (32 / BITS);
    const dim3 grid((N + COLS - 1) / COLS, KC, M);
    const uint32_t *wp = static_cast<const uint32_t *>(w);
    if (dt == MTC_F32) return qr_go<BITS, MTC_F32>(st, grid, wp, scales, biases, x, partial, tickets, out, M, N, K, gs, KC, early);
    if (dt == MTC_F16) return qr_go<BITS, MTC_F16>(st, grid, wp, scales, biases, x, partial, tickets, out, M, N, K, gs, KC, early);
    return qr_go<BITS, MTC_BF16>(st, grid, wp, scales, biases, x, partial, tickets, out, M, N, K, gs, KC, early);
}

template <int BITS>
cudaError_t qvm_launch(cudaStream_t st, const void *w, const void *scales, const void *biases, const void *x, float *partial,
                       uint32_t *tickets, void *out, int M, int N, int K, int gs, int KC, int dt, int early) {
    using S = QvShape<BITS>;
    const int tiles = (N + 32 * S::CPT - 1) / (32 * S::CPT);
    const dim3 grid(tiles, KC, M);
    const uint32_t *wp = static_cast<const uint32_t *>(w);
    const auto kern = dt == MTC_F32 ? qvm_kernel<BITS, MTC_F32> : dt == MTC_F16 ? qvm_kernel<BITS, MTC_F16> : qvm_kernel<BITS, MTC_BF16>;
    return launch_pdl(kern, grid, kQvWarps * 32, 0, st, wp, scales, biases, x, partial, tickets, out, M, N, K, gs, KC, early);
}

}  // namespace

// Which kernel: 2 / 4 / 8-bit codes under 16-bit activations, whole lanes of columns and whole slabs of 32 rows within a group can
// go to the tensor cores.  For one token of 4- or 8-bit codes the two kernels are within 15 % of one another, the one above
// being ahead; every further token costs it another pass (4096 x 4096 4-bit, 1 / 2 / 4 tokens: 7.2 / 11.6 / 19.4 us above,
// 7.9 / 9.2 / 13.0 us here; 14336 x 4096 8-bit, 4 tokens: 64.7 against 25.3).  2-bit codes are bound by issue slots from the first
// token on (4096 x 4096: 11.3 against 7.3 us).  Below the sizes of the rule the time is the start and the end of a launch, which
// are longer here (more shared memory, 16 warps to add up): 1024 x 1024 4-bit, 4 tokens: 5.1 above, 8.5 here.
static bool qvm_takes_mma(int M, int N, int K, int bits, int group_size, int dt) {
    if (dt == MTC_F32 || (bits != 2 && bits != 4 && bits != 8) || N % (bits == 8 ? 16 : 32) != 0 || group_size % 32 != 0 || K % group_size != 0)
        return false;
    const long long codes = static_cast<long long>(N) * K;
    if (bits == 2) return codes >= 1 << 20;
    return M >= 2 && N >= 1024 && codes >= (bits == 4 ? 8 << 20 : 4 << 20);
}

static int qvm_ring_chunks(int sms, int N, int K, int bits) {
    const int tiles = (N + 1024 / bits - 1) / (1024 / bits), units = K / kQrRows;
    int kc = sms / tiles;                     // one CTA an SM
    if (kc > units / kQrWarps) kc = units / kQrWarps;
    if (kc > 32) kc = 32;
    return kc < 1 ? 1 : kc;
}
// One token through the ring: rows of whole 16-byte pieces, x of a CTA's chunk beside the ring, and enough codes to pay for a CTA of 16 warps (4-bit
// 2048 x 1024 4.9 against 5.7 us here, 4096 x 1024 6.9 against 5.9; 8-bit 4096 x 2048 5.5
// against 5.7, 4096 x 4096 7.5 against 7.2, 2048 x 16384 13.8 against 9.0).
// Further tokens would read the words again for each: f32, 2 tokens of 4096 x 4096 11.8 above, 13.3 here.
static bool qvm_takes_ring(int sms, int M, int N, int K, int bits) {
    if (M != 1 || (bits != 4 && bits != 8) || N * bits / 32 % 4 != 0 || static_cast<long long>(N) * K < (bits == 4 ? 4 << 20 : 12 << 20)) return false;
    const int kc = qvm_ring_chunks(sms, N, K, bits);
    return (K / kQrRows + kc - 1) / kc <= kQrMaxUnits;
}

// slabs of 32 rows that share a range: as many as a group and a batch of 128 rows allow (fewer scales to read and apply where
// several tokens leave fewer ranges); ranges of a batch: no more than give every warp of the device a batch
static void qm_batches(int sms, int M, int N, int K, int bits, int group_size, int *ch_log2, int *bs) {
    const int ranges = M == 1 ? 4 : M == 2 ? 2 : 1;
    const long long tiles = (N + qm_cols(bits) - 1) / qm_cols(bits), all = K / 32 * tiles, warps = static_cast<long long>(sms) * kQmWarps;
    int lg = 0;
    while ((ranges << (lg + 1)) <= 4 && (group_size / 32) % (2 << lg) == 0 && all >= (warps << (lg + 1))) ++lg;
    long long r = (all + (warps << lg) - 1) / (warps << lg);
    if (r > ranges) r = ranges;
    *ch_log2 = lg;
    *bs = static_cast<int>(r < 1 ? 1 : r) << lg;
}

// Split of K over CTAs for these sizes (1 = a CTA owns all of K for its column tile): as many CTAs as are resident at once.
int qvm_k_chunks(int sms, int M, int N, int K, int bits, int group_size, int dt) {
    if (qvm_takes_mma(M, N, K, bits, group_size, dt)) {
        int ch, bs;
        qm_batches(sms, M, N, K, bits, group_size, &ch, &bs);
        const int tiles = (N + qm_cols(bits) - 1) / qm_cols(bits), batches = (K / 32 + bs - 1) / bs;
        int kc = sms / tiles;
        // two batches a CTA at least: a CTA more adds to the sum over CTAs what it takes from the products
        if (kc > (batches + 1) / 2) kc = (batches + 1) / 2;
        if (kc > 32) kc = 32;
        return kc < 1 ? 1 : kc;
    }
    if (qvm_takes_ring(sms, M, N, K, bits)) return qvm_ring_chunks(sms, N, K, bits);
    const int cpt = (bits == 3 || bits == 5 || bits == 6) ? 32 : 32 / bits;
    const int tiles = (N + 32 * cpt - 1) / (32 * cpt);
    const int units = K / ((bits == 3 || bits == 5 || bits == 6) ? 8 : 16);      // slabs of R rows
    int kc = 2 * sms / tiles;                 // never more CTAs than are resident at once (two per SM): a few CTAs in a second round would double the time
    const int most = (units + kQvWarps - 1) / kQvWarps;
    if (kc > most) kc = most;
    if (kc > 32) kc = 32;                     // the chunks of a column tile are added by one CTA
    return kc < 1 ? 1 : kc;
}

bool qvm_fast_supported(int N, int K, int bits, int group_size) {
    const int cpt = (bits == 3 || bits == 5 || bits == 6) ? 32 : 32 / bits;
    return N % cpt == 0 && K % group_size == 0 && group_size % 16 == 0 && (bits == 2 || bits == 3 || bits == 4 || bits == 5 || bits == 6 || bits == 8);
}

size_t qvm_scratch_bytes(int M, int N, int KC) {
    return KC > 1 ? kQvTickets * sizeof(uint32_t) + static_cast<size_t>(KC) * M * N * sizeof(float) : 0;
}

// scratch: qvm_scratch_bytes when KC > 1 (qvm_k_chunks), else unused; its first kQvTickets words are arrival counters
// that are zero between launches (the caller zeroes them when the block is allocated)
cudaError_t launch_qvm(Ctx *ctx, cudaStream_t st, const void *w, const void *scales, const void *biases, const void *x, void *out,
                       int M, int N, int K, int bits, int group_size, int dt, void *scratch, int KC) {
    if (M <= 0 || N <= 0) return cudaSuccess;
    const auto al16 = [](const void *p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; };
    const bool vec_ok = al16(w) && al16(scales) && al16(biases) && al16(x) && (static_cast<size_t>(K) * dtype_size(dt)) % 16 == 0;
    if (!qvm_fast_supported(N, K, bits, group_size) || M > 65535 || !vec_ok) {
        const size_t mn = static_cast<size_t>(M) * N;
        size_t grid = (mn + 255) / 256;
        if (grid > static_cast<size_t>(ctx->sm_count) * 16) grid = static_cast<size_t>(ctx->sm_count) * 16;
        qvm_generic_kernel<<<static_cast<int>(grid), 256, 0, st>>>(static_cast<const uint32_t *>(w), scales, biases, x, out, M, N, K,
                                                                    group_size, bits, dt);
        return cudaGetLastError();
    }
    if (KC > 1 && !scratch) return cudaErrorInvalidValue;
    const int cpt = (bits == 3 || bits == 5 || bits == 6) ? 32 : 32 / bits;
    const int tile_cols = qvm_takes_mma(M, N, K, bits, group_size, dt) ? qm_cols(bits) : 32 * cpt;
    const long long n_tickets = static_cast<long long>((N + tile_cols - 1) / tile_cols) * M;
    uint32_t *tickets = KC > 1 && n_tickets <= kQvTickets ? static_cast<uint32_t *>(scratch) : nullptr;   // else a second kernel adds the chunks
    float *partial = KC > 1 ? reinterpret_cast<float *>(static_cast<uint32_t *>(scratch) + kQvTickets) : nullptr;
    cudaError_t e;
    const int early = early_weights(ctx, st);
    if (qvm_takes_mma(M, N, K, bits, group_size, dt)) {
        QmArgs a{static_cast<const uint32_t *>(w), scales, biases, x, partial, tickets, out, M, N, K, group_size, KC, 0, 1, K / 32, 0, early};
        qm_batches(ctx->sm_count, M, N, K, bits, group_size, &a.ch_log2, &a.bs);
        a.batches = (a.slabs + a.bs - 1) / a.bs;
        e = bits == 2 ? qm_launch<2>(st, a, dt) : bits == 4 ? qm_launch<4>(st, a, dt) : qm_launch<8>(st, a, dt);
    } else if (qvm_takes_ring(ctx->sm_count, M, N, K, bits)) {
        e = bits == 4 ? qr_launch<4>(st, w, scales, biases, x, partial, tickets, out, M, N, K, group_size, KC, dt, early)
                      : qr_launch<8>(st, w, scales, biases, x, partial, tickets, out, M, N, K, group_size, KC, dt, early);
    } else switch (bits) {
        case 2: e = qvm_launch<2>(st, w, scales, biases, x, partial, tickets, out, M, N, K, group_size, KC, dt, early); break;
        case 3: e = qvm_launch<3>(st, w, scales, biases, x, partial, tickets, out, M, N, K, group_size, KC, dt, early); break;
        case 4: e = qvm_launch<4>(st, w, scales, biases, x, partial, tickets, out, M, N, K, group_size, KC, dt, early); break;
        case 5: e = qvm_launch<5>(st, w, scales, biases, x, partial, tickets, out, M, N, K, group_size, KC, dt, early); break;
        case 6: e = qvm_launch<6>(st, w, scales, biases, x, partial, tickets, out, M, N, K, group_size, KC, dt, early); break;
        default: e = qvm_launch<8>(st, w, scales, biases, x, partial, tickets, out, M, N, K, group_size, KC, dt, early); break;
    }
    if (e != cudaSuccess || KC == 1 || tickets) return e;
    const size_t mn = static_cast<size_t>(M) * N;
    size_t grid = (mn + 255) / 256;
    if (grid > static_cast<size_t>(ctx->sm_count) * 8) grid = static_cast<size_t>(ctx->sm_count) * 8;
    qvm_sum_kernel<<<static_cast<int>(grid), 256, 0, st>>>(partial, out, mn, KC, dt);
    return cudaGetLastError();
}

}  // namespace mtc
