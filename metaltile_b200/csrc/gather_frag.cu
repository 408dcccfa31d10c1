// Host side of the grouped fragment kernel (gather_frag.cuh): which shapes it takes and which of its forms runs.
#include "gather_frag.cuh"

namespace mtc {

namespace {

// How the rows of a pass are laid over the MMA's columns: as many as an expert has in the mean
gfrag::Shape pick_shape(int m_total, int n_experts, int bits, int group, int dt) {
    using namespace frag;
    const int rows = 2ll * m_total <= n_experts ? 2 : m_total <= 2ll * n_experts ? 4 : 8;
    if (rows == 2) return {S2, 1, dt};
    if (group % 64 != 0) return {S2, rows / 2, dt};
    if (rows == 4) return {S4, 1, dt};
    return bits == 4 || bits == 8 ? gfrag::Shape{G8, 1, dt} : gfrag::Shape{S4, 2, dt};
}

}  // namespace

bool gather_frag_supported(int m_total, int n_out, int K, int n_experts, int bits, int group_size, int dt, const void *w, const void *scales,
                           const void *biases, const void *x) {
    const auto al = [](const void *p, size_t n) { return reinterpret_cast<uintptr_t>(p) % n == 0; };
    if (!(bits == 2 || bits == 3 || bits == 4 || bits == 5 || bits == 6 || bits == 8) || (dt != MTC_F16 && dt != MTC_BF16)) return false;
    if (m_total < 1 || n_out < 1 || K < 32 || K % 32 != 0 || n_experts < 1 || n_experts > 4096) return false;
    if (group_size < 32 || (group_size & (group_size - 1)) != 0 || K % group_size != 0) return false;
    if ((static_cast<long long>(m_total) + n_experts) * ((n_out + 15) / 16 * 2) >= (1ll << 31)) return false;      // tiles are counted in 32 bits
    const gfrag::Shape s = pick_shape(m_total, n_experts, bits, group_size, dt);
    return gfrag::make_plan(K, n_experts, bits, s.mode, s.nt).ks > 0 && al(w, 16) && al(x, 16) && al(scales, 2) && al(biases, 2);
}

// x rows sorted by expert -> mats[i].out [m_total, n_out] for one matrix set or for two that read the same rows; row_src: row m of the
// product reads x[row_src[m]] (x has n_src_rows rows)
cudaError_t launch_gather_frag(Ctx *ctx, cudaStream_t st, const void *x, const uint32_t *row_src, int n_src_rows, const GatherMats *mats, int n_mats,
                               const uint32_t *expert_offsets, int m_total, int n_out, int K, int n_experts, int bits, int group_size, int dt) {
    if (n_mats < 1 || n_mats > 2) return cudaErrorInvalidValue;
    const gfrag::Shape s = pick_shape(m_total, n_experts, bits, group_size, dt);
    const gfrag::Plan p = gfrag::make_plan(K, n_experts, bits, s.mode, s.nt);
    if (p.ks == 0) return cudaErrorInvalidConfiguration;
    GfArgs a{};
    for (int i = 0; i < 2; ++i) {
        const GatherMats &m = mats[i < n_mats ? i : 0];
        a.w[i] = static_cast<const uint32_t *>(m.w);
        a.scales[i] = m.scales;
        a.biases[i] = m.biases;
        a.out[i] = m.out;
    }
    a.x = x;
    a.offsets = expert_offsets;
    a.row_src = row_src;
    a.status = ctx->d_status;
    a.n_src_rows = n_src_rows;
    a.n_experts = n_experts;
    a.m_total = m_total;
    a.n_out = n_out;
    a.K = K;
    while ((1 << a.gs_shift) < group_size) ++a.gs_shift;
    a.wpr = static_cast<int>(static_cast<long long>(K) * bits / 32);
    a.gpr = K / group_size;
    a.steps = (K + 127) / 128;
    a.tpm = (n_out + 15) / 16;
    a.tpe = a.tpm * n_mats;
    a.ks = p.ks;
    a.off_sum = p.off_sum;
    a.off_part = p.off_part;
    a.warp_bytes = p.warp_bytes;
    a.off_red = p.off_red;
    switch (bits) {
        case 2: return launch_gather_frag_b2(st, a, s, p, ctx->sm_count);
        case 3: return launch_gather_frag_b3(st, a, s, p, ctx->sm_count);
        case 4: return launch_gather_frag_b4(st, a, s, p, ctx->sm_count);
        case 5: return launch_gather_frag_b5(st, a, s, p, ctx->sm_count);
        case 6: return launch_gather_frag_b6(st, a, s, p, ctx->sm_count);
        default: return launch_gather_frag_b8(st, a, s, p, ctx->sm_count);
    }
}

}  // namespace mtc
