// Host side of the fragment kernel (qmv_frag.cuh): which shapes it takes and which of its forms runs.
#include "qmv_frag.cuh"

namespace mtc {

namespace {

// How the token rows are laid over the MMA's columns, for one launch of M rows (see the modes in qmv_frag.cuh).
frag::Shape pick_shape(int M, int K, int bits, int group, int dt, bool aligned16) {
    using namespace frag;
    Shape s{S1, 1, 0, dt};
    const bool halves = group % 64 == 0;                   // two chunks, or the two halves of a step, share a group
    if (M == 1) s.mode = S1;
    else if (M == 2) s.mode = S2;
    else if (!halves) { s.mode = S2; s.nt = M <= 4 ? 2 : 4; }
    else if (M <= 4) s.mode = S4;
    else if (bits == 4 || bits == 8) { s.mode = G8; s.nt = M <= 8 ? 1 : 2; }
    else { s.mode = S4; s.nt = M <= 8 ? 2 : 4; }
    if (bits == 4 && dt != MTC_F32 && K % 512 == 0 && aligned16 && (group == 64 || group == 128) && (s.nt == 1 || s.mode == G8))
        s.vec = group == 64 ? 6 : 7;
    return s;
}

// token rows of one launch: f32 activations take three times the shared memory, groups of 32 half of the columns
int rows_per_launch(int group, int dt) { return dt == MTC_F32 || group % 64 != 0 ? 8 : 16; }

}  // namespace

bool qmv_frag_supported(int M, int N, int K, int bits, int group_size, int dt, const void *w, const void *scales, const void *biases, const void *x) {
    const auto al = [](const void *p, size_t n) { return reinterpret_cast<uintptr_t>(p) % n == 0; };
    if (!(bits == 2 || bits == 3 || bits == 4 || bits == 5 || bits == 6 || bits == 8)) return false;
    if (M < 1 || M > 16 || N < 1 || K < 32 || K % 32 != 0) return false;
    if (group_size < 32 || (group_size & (group_size - 1)) != 0 || K % group_size != 0) return false;
    if (static_cast<long long>(N) * K / 8 * bits >= (1ll << 32) - 65536) return false;                    // 32-bit byte offsets
    return al(w, 16) && al(x, 16) && al(scales, dtype_size(dt)) && al(biases, dtype_size(dt));
}

// 1 to 4 projections that read the same activations, each writing its own output
cudaError_t launch_qmv_frag(Ctx *ctx, cudaStream_t st, const mtc_qmv_desc *d, int n) {
    if (n < 1 || n > 4) return cudaErrorInvalidValue;
    const int M = d[0].M, K = d[0].K, bits = d[0].bits, dt = d[0].dtype, esz = static_cast<int>(dtype_size(dt));
    int gs_shift = 0;
    while ((1 << gs_shift) < d[0].group_size) ++gs_shift;
    const int per = rows_per_launch(d[0].group_size, dt);
    for (int m0 = 0; m0 < M; m0 += per) {
        FragArgs a{};
        a.M = M - m0 < per ? M - m0 : per;
        a.K = K;
        a.gs_shift = gs_shift;
        a.wpr = static_cast<int>(static_cast<long long>(K) * bits / 32);
        a.gpr = K / d[0].group_size;
        a.steps = (K + 127) / 128;
        a.x = static_cast<const char *>(d[0].x) + static_cast<size_t>(m0) * K * esz;
        a.early = early_weights(ctx, st);
        a.n_proj = n;
        bool aligned16 = true;
        for (int i = 0; i < n; ++i) {
            FragProj &p = a.p[i];
            p.w = static_cast<const uint32_t *>(d[i].w);
            p.scales = d[i].scales;
            p.biases = d[i].biases;
            p.out = static_cast<char *>(d[i].outs[0]) + static_cast<size_t>(m0) * d[i].N * esz;
            p.N = d[i].N;
            p.tile0 = a.tiles;
            a.tiles += (d[i].N + 15) / 16;
            aligned16 = aligned16 && reinterpret_cast<uintptr_t>(p.scales) % 16 == 0 && reinterpret_cast<uintptr_t>(p.biases) % 16 == 0;
        }
        const frag::Shape s = pick_shape(a.M, K, bits, d[0].group_size, dt, aligned16);
        cudaError_t e;
        switch (bits) {
            case 2: e = launch_frag_b2(st, a, s, ctx->sm_count); break;
            case 3: e = launch_frag_b3(st, a, s, ctx->sm_count); break;
            case 4: e = launch_frag_b4(st, a, s, ctx->sm_count); break;
            case 5: e = launch_frag_b5(st, a, s, ctx->sm_count); break;
            case 6: e = launch_frag_b6(st, a, s, ctx->sm_count); break;
            default: e = launch_frag_b8(st, a, s, ctx->sm_count); break;
        }
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace mtc
