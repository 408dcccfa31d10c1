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
