// Host side of the cluster kernel (qmv_cluster.cuh): which shapes it takes and which of its forms runs.
#include "qmv_cluster.cuh"

namespace mtc {

namespace clu {

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                                  const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                  CUtensorMapFloatOOBfill);

// The words of every projection as lines of 128 bytes: {32 words, lines of a row, rows}, box {32, ub, 16}.  Rows past the end read as zero.
cudaError_t word_maps(CluArgs &a, int row_bytes, int ub) {
    static const EncodeTiledFn encode = [] {
        void *ptr = nullptr;
        cudaDriverEntryPointQueryResult qres;
        const cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres);
        return e == cudaSuccess && qres == cudaDriverEntryPointSuccess ? reinterpret_cast<EncodeTiledFn>(ptr) : nullptr;
    }();
    if (!encode) return cudaErrorNotSupported;
    for (int i = 0; i < a.n_proj; ++i) {
        const cuuint64_t dims[3] = {32, static_cast<cuuint64_t>(row_bytes / 128), static_cast<cuuint64_t>(a.p[i].N)};
        const cuuint64_t strides[2] = {128, static_cast<cuuint64_t>(row_bytes)};
        const cuuint32_t box[3] = {32, static_cast<cuuint32_t>(ub), 16}, estr[3] = {1, 1, 1};
        if (encode(&a.map[i], CU_TENSOR_MAP_DATA_TYPE_UINT32, 3, const_cast<uint32_t *>(a.p[i].w), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return cudaErrorInvalidValue;
    }
    return cudaSuccess;
}

}  // namespace clu

namespace {

bool supported(const mtc_qmv_desc &d) {
    const auto al16 = [](const void *p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; };
    const int G = d.group_size, K = d.K;
    if ((d.bits != 4 && d.bits != 8) || d.M < 1 || d.M > 16 || d.N < 1 || K < 1 || K >= (1 << 24)) return false;
    if (G < 32 || (G & (G - 1)) != 0 || K % G != 0 || static_cast<long long>(d.N) * K >= (1ll << 36)) return false;
    const int esz = static_cast<int>(dtype_size(d.dtype)), unit = clu::lines(d.dtype, d.M, G) * 1024 / d.bits;
    if (K % unit != 0) return false;
    // the scales of a unit and row do not straddle two windows of 16 bytes
    const int bytes = (G < unit ? unit / G : 1) * esz, window = bytes < 16 ? bytes : 16;
    return static_cast<long long>(K / G) * esz % window == 0 && al16(d.w) && al16(d.x) && al16(d.scales) && al16(d.biases);
}

}  // namespace

// Whether one launch of this kernel takes the projections (M >= 2), and is the faster one (us, the kernel it took over from -> this one), among
// those that the entries offer it (cluster_first and frag_rule, runtime.cu): from nine tokens on they keep groups of 32, single 8-bit matrices
// above 20 Mi codes or of K > 5120, and at five to eight 8-bit ones of K > 8192 from 32 Mi codes on for the tcgen05 kernel, unmeasured against this one.
//   f32 activations: always (8-bit 4096 x 4096, 8 / 16 tokens 15.0 -> 10.7 / 28.1 -> 15.2; 8192 x 8192 4-bit 60 -> 21 / 118 -> 35).
//   4-bit: always (4096 x 4096, 8 / 16 tokens 6.3 -> 5.9 / 10.2 -> 9.0, 28672 x 4096 21.8 -> 16.6 / 28.8 -> 25.1, 4096 x 14336 17.4 -> 13.7 / 29.2 ->
//     21.5; groups of 32 4096 x 4096, 8 tokens 9.4 -> 6.9).
//   8-bit, 16-bit activations: from 16 Mi codes on, from nine tokens on from 12 Mi (8192 x 8192, 8 tokens 23.6 -> 17.0, 14336 x 2048 as part of a
//     fused launch, 16 tokens 16.7 -> 11.9; 2048 x 2048 3.8 = 3.9, 5120 x 3072 7.0 against 7.9), with groups of 32 always (2048 x 2048, 8 tokens
//     4.8 -> 4.4).
//   4-bit from nine tokens on where K is an odd multiple of 256 (the fragment kernel had these) and no CTA has more than a tile: not for
//     K = 2304 to 3840, where its few warps walk all of K (477 x 3840 5.3 against 6.3, 865 x 2816 4.5 against 5.1, 2048 x 2304 4.8 against 5.0; 865 x
//     1280 and 4352 and 4096 x 2816 are faster here; K = 1792 is slower by itself, 281 rows 3.7 against 4.0, but faster between the other launches of a
//     decode step: six layers of 1792 / 256 / 1792, 15 tokens 142 -> 131).
// A call costs the host 0.2 us more than the ring kernel before it did (a tensor map a projection): products too small to hide it, 4-bit of 1 Mi
// codes, go from 4.4 to 4.6 us a call, though not in a graph (1247 x 512, 12 tokens 3.37 -> 2.95; 602 x 2560, 5 tokens 3.70 -> 3.43).
static bool takes(const mtc_qmv_desc *d, int n, int sms, clu::Plan &plan) {
    long long codes = 0;
    int tiles = 0;
    for (int i = 0; i < n; ++i) {
        if (d[i].bits != d[0].bits || d[i].group_size != d[0].group_size || !supported(d[i])) return false;
        codes += static_cast<long long>(d[i].N) * d[i].K;
        tiles += (d[i].N + 15) / 16;
    }
    if (d[0].bits == 8 && d[0].dtype != MTC_F32 && d[0].group_size != 32 && codes < ((d[0].M <= 8 ? 16ll : 12ll) << 20)) return false;
    if (d[0].bits == 4 && d[0].dtype != MTC_F32 && d[0].M > 8 && d[0].K % 512 != 0 && d[0].K > 2048 && d[0].K < 4096 && tiles <= sms) return false;
    plan = clu::shape_plan(d[0], tiles, sms);
    return plan.shift >= 0;          // a part of K that shared memory cannot hold: no plan
}

// The form of that launch, for mtc_launch_of; false: not this kernel's shape
bool qmv_cluster_form(const Ctx *ctx, const mtc_qmv_desc *d, int n, mtc_launch_info *info) {
    clu::Plan p;
    if (n < 1 || n > 4 || !takes(d, n, ctx->sm_count, p)) return false;
    *info = mtc_launch_info{"qmv_cluster", p.clusters << p.shift, 1 << p.shift, 1 << p.shift, p.passes};
    return true;
}

// 1 to 4 projections that read the same activations, each writing its own output; false: not this kernel's shape, nothing is launched
bool try_qmv_cluster(Ctx *ctx, cudaStream_t st, const mtc_qmv_desc *d, int n, cudaError_t *e) {
    clu::Plan p;
    if (n < 1 || n > 4 || !takes(d, n, ctx->sm_count, p)) return false;
    const int bits = d[0].bits, G = d[0].group_size;
    CluArgs a{};
    a.M = d[0].M;
    a.K = d[0].K;
    while ((1 << a.gs_shift) < G) ++a.gs_shift;
    a.s_pitch = static_cast<uint32_t>(a.K / G * dtype_size(d[0].dtype));
    a.status = ctx->d_status;
    a.x = d[0].x;
    a.early = early_weights(ctx, st);
    a.n_proj = n;
    for (int i = 0; i < n; ++i) {
        FragProj &p = a.p[i];
        p.w = static_cast<const uint32_t *>(d[i].w);
        p.scales = d[i].scales;
        p.biases = d[i].biases;
        p.out = d[i].outs[0];
        p.N = d[i].N;
        p.tile0 = a.tiles;
        a.tiles += (d[i].N + 15) / 16;
    }
    const clu::Shape s{a.M <= 8 ? 1 : 2, G, d[0].dtype};
    *e = bits == 4 ? launch_cluster_b4(st, a, s, p) : launch_cluster_b8(st, a, s, p);
    return true;
}

}  // namespace mtc
