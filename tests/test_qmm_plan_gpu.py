"""The tcgen05 product on shapes where its copies and its plan can go wrong, against the oracle.

K that is no multiple of a super-block (256), rows of scales that start at any 2-byte offset, 3- and 5-bit rows that start on
8-byte boundaries only, the last scale of the array alone in its word, weight tiles short of 128 rows, K slices of unequal
length with a short last one, one and two chunks per item, chunks of equal width."""
import numpy as np
import pytest

import oracle
from helpers import TOL, dense_case, rel_err, to_dev

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from metaltile_b200 import ops
    return ops.context(0)


@pytest.mark.parametrize("bits", [2, 3, 4, 5, 6, 8])
@pytest.mark.parametrize("m,n,k,gs", [(17, 100, 64, 32),        # one k block
                                      (40, 129, 320, 64),       # five: K / group odd, a tile with one row
                                      (33, 127, 832, 32), (65, 256, 1088, 64), (70, 130, 384, 128),
                                      (257, 96, 2880, 64),      # K slices of two-chunk items
                                      (300, 257, 1152, 128), (530, 64, 192, 64)])
def test_ragged_shapes(ctx, m, n, k, gs, bits):
    import torch
    from metaltile_b200 import ops
    dt = "f16" if (bits + m) % 2 else "bf16"
    w, s, b, x = dense_case(m, n, k, bits, gs, dt, seed=31)
    got = ops.qmm(to_dev(w), to_dev(s, dt), to_dev(b, dt), to_dev(x, dt), bits, gs, ctx=ctx)
    torch.cuda.synchronize()
    assert ctx.status_word() == 0
    got = got.float().cpu().numpy()
    rows = np.unique(np.r_[0:8, m // 2 - 4:m // 2 + 4, m - 8:m])
    ref = oracle.qmm(w, s, b, np.ascontiguousarray(x[rows]), len(rows), n, k, bits, gs)
    assert np.all(np.isfinite(got)) and rel_err(got[rows], ref) <= TOL[dt]


@pytest.mark.parametrize("bits,gs,counts", [(8, 32, (3, 0, 40, 1)), (5, 64, (70, 2, 0, 9)), (4, 64, (300, 1, 33, 0))])
def test_grouped_product_on_ragged_rows(ctx, bits, gs, counts):
    """The same copies with experts: the last row of one is followed by the first of the next, K / group is odd."""
    import torch
    from metaltile_b200 import ops
    e, n, k, dt = len(counts), 136, 320, "f16"
    w, s, b, x = dense_case(sum(counts), e * n, k, bits, gs, dt, seed=32)
    off = np.concatenate([[0], np.cumsum(counts)]).astype(np.uint32)
    ctx.set_option("gather_stream", 0)
    try:
        got = ops.gather_qmm(to_dev(x, dt), to_dev(w).view(e, n, -1), to_dev(s, dt).view(e, n, -1), to_dev(b, dt).view(e, n, -1), bits, gs,
                             expert_offsets=to_dev(off), ctx=ctx)
    finally:
        ctx.set_option("gather_stream", 1)
    torch.cuda.synchronize()
    assert ctx.status_word() == 0
    for i, c in enumerate(counts):
        if c:
            r = slice(off[i], off[i + 1])
            ref = oracle.qmm(w[i * n:(i + 1) * n], s[i * n:(i + 1) * n], b[i * n:(i + 1) * n], x[r], c, n, k, bits, gs)
            assert rel_err(got[r.start:r.stop].float().cpu().numpy(), ref) <= TOL[dt]


@pytest.mark.parametrize("m,n,k,bits,gs,multi", [(300, 1024, 4096, 4, 64, False), (700, 576, 2880, 8, 32, False), (300, 1024, 4096, 4, 64, True)])
def test_capture_without_a_first_run(m, n, k, bits, gs, multi):
    """f16 prompts captured on a fresh context.  The plan for these sizes cuts K into slices, whose partial sums need a block that
    cannot grow during capture: the launch runs without slices instead of failing, and the replay matches the oracle."""
    import torch
    from metaltile_b200 import Context
    from metaltile_b200.ops import _TORCH_DT
    fresh, dt = Context(0), "f16"
    w, s, b, x = dense_case(m, n, k, bits, gs, dt, seed=33)
    wd, sd, bd, xd = to_dev(w), to_dev(s, dt), to_dev(b, dt), to_dev(x, dt)
    outs = [torch.zeros((m, n), dtype=torch.float16, device="cuda") for _ in range(2 if multi else 1)]
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            st = torch.cuda.current_stream().cuda_stream
            if multi:
                fresh.qmm_multi(wd.data_ptr(), sd.data_ptr(), bd.data_ptr(), xd.data_ptr(), [o.data_ptr() for o in outs], n, m, n, k, bits, gs,
                                _TORCH_DT[xd.dtype], stream=st)
            else:
                fresh.qmm(wd.data_ptr(), sd.data_ptr(), bd.data_ptr(), xd.data_ptr(), outs[0].data_ptr(), m, n, k, bits, gs, _TORCH_DT[xd.dtype], stream=st)
    graph.replay()
    torch.cuda.synchronize()
    assert fresh.status_word() == 0
    rows = np.unique(np.r_[0:8, m // 2 - 4:m // 2 + 4, m - 8:m])
    ref = oracle.qmm(w, s, b, np.ascontiguousarray(x[rows]), len(rows), n, k, bits, gs)
    for o in outs:
        assert rel_err(o.float().cpu().numpy()[rows], ref) <= TOL[dt]
    # the same call outside capture takes its slices: the same products, added in another order
    eager = torch.zeros_like(outs[0])
    fresh.qmm(wd.data_ptr(), sd.data_ptr(), bd.data_ptr(), xd.data_ptr(), eager.data_ptr(), m, n, k, bits, gs, _TORCH_DT[xd.dtype],
              stream=torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert rel_err(eager.float().cpu().numpy()[rows], ref) <= TOL[dt]


def test_slices_stay_within_their_bound(ctx):
    """A prompt whose slices would take more than the bound on their partial sums, and lengths that rise: the products are right and
    the block of partial sums (with what it outgrew) stays small beside the outputs."""
    import torch
    from metaltile_b200 import Context, ops
    fresh = Context(0)
    n, k, bits, gs, dt = 576, 4096, 4, 64, "f16"
    w, s, b, x = dense_case(4096, n, k, bits, gs, dt, seed=34)
    wd, sd, bd, xd = to_dev(w), to_dev(s, dt), to_dev(b, dt), to_dev(x, dt)
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    for m in range(300, 4096, 211):
        got = ops.qmm(wd, sd, bd, xd[:m], bits, gs, ctx=fresh)
        rows = np.r_[0:4, m - 4:m]
        ref = oracle.qmm(w, s, b, np.ascontiguousarray(x[rows]), len(rows), n, k, bits, gs)
        assert rel_err(got.float().cpu().numpy()[rows], ref) <= TOL[dt]
        del got
    torch.cuda.empty_cache()
    assert free0 - torch.cuda.mem_get_info()[0] < 3 * (512 << 20) * 1.5 + (64 << 20)


@pytest.mark.parametrize("m,n,k,bits,gs,dt,ld,shift", [
    (70, 576, 2880, 8, 32, "f16", 600, 0), (300, 1024, 4096, 4, 64, "bf16", 4096, 8), (33, 130, 2048, 4, 64, "bf16", 131, 1),
    (700, 192, 5120, 3, 64, "f16", 1000, 3)])
def test_slices_with_several_destinations(ctx, m, n, k, bits, gs, dt, ld, shift):
    """A product cut into K slices whose result is a column block of three wider matrices (rows and blocks that start anywhere): every
    copy equals the plain product bit for bit, and nothing beside the block is written."""
    import torch
    from metaltile_b200 import ops
    from metaltile_b200.ops import _TORCH_DT
    w, s, b, x = dense_case(m, n, k, bits, gs, dt, seed=35)
    wd, sd, bd, xd = to_dev(w), to_dev(s, dt), to_dev(b, dt), to_dev(x, dt)
    ctx.set_option("qmm_mma_chunks", 0)                   # 33 rows: the tensor-core kernel, as for several destinations
    try:
        want = ops.qmm(wd, sd, bd, xd, bits, gs, ctx=ctx)
    finally:
        ctx.set_option("qmm_mma_chunks", 1)
    rows = np.r_[0:4, m - 4:m]
    ref = oracle.qmm(w, s, b, np.ascontiguousarray(x[rows]), len(rows), n, k, bits, gs)
    assert rel_err(want.float().cpu().numpy()[rows], ref) <= TOL[dt]
    outs = [torch.full((m * ld + 16,), 7.0, dtype=xd.dtype, device="cuda") for _ in range(3)]
    ctx.qmm_multi(wd.data_ptr(), sd.data_ptr(), bd.data_ptr(), xd.data_ptr(), [o[shift:].data_ptr() for o in outs], ld, m, n, k, bits, gs,
                  _TORCH_DT[xd.dtype], stream=torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert ctx.status_word() == 0
    for o in outs:
        block = o[shift:shift + m * ld].view(m, ld)
        assert torch.equal(block[:, :n], want)
        block[:, :n] = 7.0
        assert bool((o == 7.0).all())


@pytest.mark.parametrize("m", [256, 257, 300, 432, 433])
@pytest.mark.parametrize("n,k", [(4096, 1024), (3520, 896)])
def test_a_chunk_has_at_most_256_rows(ctx, m, n, k):
    """27 to 33 weight tiles and four super-blocks of K: the rows that one chunk holds, and those that take two."""
    import torch
    from metaltile_b200 import ops
    w, s, b, x = dense_case(m, n, k, 4, 64, "f16", seed=33)
    got = ops.qmm(to_dev(w), to_dev(s, "f16"), to_dev(b, "f16"), to_dev(x, "f16"), 4, 64, ctx=ctx)
    torch.cuda.synchronize()
    assert ctx.status_word() == 0
    rows = np.unique(np.r_[0:2, 255:m][:12])
    ref = oracle.qmm(w, s, b, np.ascontiguousarray(x[rows]), len(rows), n, k, 4, 64)
    assert rel_err(got.float().cpu().numpy()[rows], ref) <= TOL["f16"]
