"""The fragment kernel (option "qmv_frag" = 2) and the fused launches of the small-M kernels against the oracle.

Sizes where the kernel can go wrong: rows short of and past a 16-row tile, K of one chunk (32), of a partial step (128
codes) and of a partial run (512), slices of K shorter than the eight warps, more tiles than the grid takes in one round,
every token count at which the layout of the columns changes, activations too large for one staged block."""
import numpy as np
import pytest

import oracle
from helpers import dense_case, rel_err, to_dev

pytestmark = pytest.mark.gpu

# |got - oracle| / max(|oracle|, 1).  Rounding a value to a significand of p bits moves it by at most half a unit in the last
# place, 2^-p of the value (bf16: p = 8, f16: p = 11); the f32 sums on both sides add less than 2^-14 at these lengths
# (K <= 14336 products of magnitude ~1 and random sign: sqrt(K) * 2^-24 each way, and the bias term's cancellation)
BOUND = {"bf16": 2.0 ** -8 + 2.0 ** -14, "f16": 2.0 ** -11 + 2.0 ** -14, "f32": 2.0 ** -14}


@pytest.fixture(scope="module")
def ctx():
    from metaltile_b200 import ops
    return ops.context(0)


def _check(ctx, m, n, k, bits, gs, dt, seed=11):
    import torch
    from metaltile_b200 import ops
    w, s, b, x = dense_case(m, n, k, bits, gs, dt, seed=seed)
    ref = oracle.qmm(w, s, b, x, m, n, k, bits, gs)
    ctx.set_option("qmv_frag", 2)
    try:
        got = ops.qmv(to_dev(w), to_dev(s, dt), to_dev(b, dt), to_dev(x, dt), bits, gs, ctx=ctx)
    finally:
        ctx.set_option("qmv_frag", 1)
    torch.cuda.synchronize()
    assert rel_err(got.float().cpu().numpy(), ref) <= BOUND[dt]


@pytest.mark.parametrize("dt", ["bf16", "f16", "f32"])
@pytest.mark.parametrize("bits", [2, 3, 4, 5, 6, 8])
@pytest.mark.parametrize("n,k,gs", [(1, 32, 32), (15, 96, 32), (17, 320, 64), (33, 640, 128), (40, 1536, 64)])
def test_edges_of_tiles_and_runs(ctx, n, k, gs, bits, dt):
    for m in (1, 2, 3, 5):
        _check(ctx, m, n, k, bits, gs, dt)


@pytest.mark.parametrize("m", [1, 2, 3, 4, 5, 7, 8, 9, 16])
@pytest.mark.parametrize("bits,gs,dt", [(4, 64, "bf16"), (4, 128, "f16"), (4, 32, "bf16"), (8, 64, "f32"), (3, 64, "bf16"), (6, 32, "f16")])
def test_every_column_layout(ctx, bits, gs, dt, m):
    _check(ctx, m, 50, 1024, bits, gs, dt)


@pytest.mark.parametrize("m,n,k,bits,gs,dt", [(1, 9600, 512, 4, 64, "bf16"),       # three rounds of tiles
                                              (8, 48, 14336, 4, 64, "bf16"),       # activations staged block by block
                                              (16, 32, 8192, 8, 64, "bf16"), (8, 32, 4096, 8, 64, "f32")])
def test_rounds_and_blocks(ctx, m, n, k, bits, gs, dt):
    _check(ctx, m, n, k, bits, gs, dt)


@pytest.mark.parametrize("m,k,bits,gs", [(1, 1024, 4, 64), (3, 1024, 4, 64), (8, 1024, 4, 128), (16, 512, 4, 64), (4, 1088, 4, 64), (5, 640, 8, 32)])
def test_projections_in_one_launch_equal_separate_ones(ctx, m, k, bits, gs):
    """Rows that end inside a tile in the middle of the launch: every projection has its own tiles.  With so few tiles the launch
    splits K over its warps as each of the separate ones does, so the results are theirs bit for bit (M = 5 to 16 with 4-bit
    codes on the cluster kernel, else the fragment kernel); with more tiles the splits may differ, see the next test."""
    import torch
    from metaltile_b200 import ops
    mats = []
    for i, n in enumerate((100, 17, 48)):
        w, s, b, x = dense_case(m, n, k, bits, gs, "bf16", seed=21, salt=i)
        mats.append((to_dev(w), to_dev(s, "bf16"), to_dev(b, "bf16"), oracle.qmm(w, s, b, dense_case(m, n, k, bits, gs, "bf16", seed=21)[3], m, n, k, bits, gs)))
    xd = to_dev(dense_case(m, 100, k, bits, gs, "bf16", seed=21)[3], "bf16")
    got = ops.qmv_batched([t[:3] for t in mats], xd, bits, gs, ctx=ctx)
    torch.cuda.synchronize()
    if m == 1:
        got = [g for g in torch.split(got, [100, 17, 48], dim=1)]
    for g, t in zip(got, mats):
        assert rel_err(g.float().cpu().numpy().reshape(m, -1), t[3]) <= BOUND["bf16"]
        assert torch.equal(g.reshape(m, -1), ops.qmv(*t[:3], xd, bits, gs, ctx=ctx).reshape(m, -1))


@pytest.mark.parametrize("m,k,bits,gs,dt", [(1, 4096, 4, 64, "bf16"), (8, 4096, 4, 64, "f16"), (16, 2048, 4, 128, "bf16"), (4, 2048, 8, 64, "f16")])
def test_projections_in_one_launch_at_size(ctx, m, k, bits, gs, dt):
    """Launches whose tiles fill the device, where the fused launch may split K otherwise than the separate ones: every product is
    right, the call repeats itself bit for bit, and it differs from the separate launches by single roundings of the output."""
    import torch
    from metaltile_b200 import ops
    ns, mats = (4096, 1024, 1040), []
    for i, n in enumerate(ns):
        w, s, b, _ = dense_case(m, n, k, bits, gs, dt, seed=22, salt=i)
        mats.append((to_dev(w), to_dev(s, dt), to_dev(b, dt), w, s, b))
    x = dense_case(m, 16, k, bits, gs, dt, seed=22)[3]
    xd = to_dev(x, dt)
    got, again = (ops.qmv_batched([t[:3] for t in mats], xd, bits, gs, ctx=ctx) for _ in range(2))
    if m == 1:
        got, again = torch.split(got, list(ns), dim=1), torch.split(again, list(ns), dim=1)
    for n, t, g, a in zip(ns, mats, got, again):
        assert torch.equal(g, a)
        alone = ops.qmv(*t[:3], xd, bits, gs, ctx=ctx)
        ref = oracle.qmm(t[3], t[4], t[5], x, m, n, k, bits, gs, rows=(0, 64))[:, :64]
        assert rel_err(g[:, :64].float().cpu().numpy(), ref) <= BOUND[dt]
        assert rel_err(g.float().cpu().numpy(), alone.float().cpu().numpy()) <= 2 * BOUND[dt]


@pytest.mark.parametrize("m,gs,dt", [(1, 64, "bf16"), (1, 32, "f32"), (2, 64, "f16"), (4, 32, "bf16"), (7, 32, "f16"), (7, 64, "bf16")])
@pytest.mark.parametrize("k", [8320, 8576, 14464])
def test_long_lanes_past_a_staged_block(ctx, m, gs, dt, k):
    """3-bit rows that start on 16 bytes (K a multiple of 128, so that lanes take consecutive chunks), a last run of K that is not full,
    and - at several tokens - activations that are staged block by block."""
    _check(ctx, m, 50, k, 3, gs, dt)


@pytest.mark.parametrize("bits,gs,dt,m", [(4, 64, "bf16", 1), (4, 32, "f16", 4), (8, 64, "f32", 5), (8, 64, "bf16", 7), (2, 64, "f16", 2)])
def test_infinite_scales(ctx, bits, gs, dt, m):
    """One group with an infinite scale in some rows, before a last run of K that is not full: lanes past the end of the row must
    not multiply their zeros by what the run before left in their registers (inf * 0), and the other rows stay finite.  The
    weights' codes are not zero, so the sum of the group is not, and the result is the infinity that the CUDA cores get."""
    import torch
    from metaltile_b200 import ops
    n, k = 40000, 1088
    w, s, b, x = dense_case(m, n, k, bits, gs, dt, seed=5)
    w |= np.uint32({2: 0x55555555, 4: 0x11111111, 8: 0x01010101}[bits])
    x = np.abs(x)
    bad = np.arange(0, n, 97)
    s[bad, 640 // gs] = np.inf                     # of the second run of 512 codes, in steps that the third one does not reach
    s[bad[::2], 960 // gs] = np.inf
    want = np.zeros(n, dtype=bool)
    want[bad] = True
    for frag in (0, 2):
        ctx.set_option("qmv_frag", frag)
        try:
            got = ops.qmv(to_dev(w), to_dev(s, dt), to_dev(b, dt), to_dev(x, dt), bits, gs, ctx=ctx)
        finally:
            ctx.set_option("qmv_frag", 1)
        got = got.float().cpu().numpy()
        assert (np.isposinf(got) == want).all() and np.isfinite(got[:, ~want]).all(), frag


@pytest.mark.parametrize("bits,dt,m", [(8, "f32", 5), (4, "f32", 16), (4, "bf16", 1), (8, "bf16", 4), (4, "f16", 2)])
def test_infinite_activations(ctx, bits, dt, m):
    """x = inf against weights that are all positive is inf (a CUDA-core product of the same inputs says so too), x = nan is nan, and
    the other tokens know nothing of either."""
    import torch
    from metaltile_b200 import ops
    n, k, gs = 64, 512, 64
    w, s, b, x = dense_case(m, n, k, bits, gs, dt, seed=6)
    w |= np.uint32(0x11111111 if bits == 4 else 0x01010101)             # no code is zero
    b = np.abs(b)
    x[0, 100] = np.inf
    if m > 2:
        x[2, 300] = np.nan
    for frag in (2, 0):
        ctx.set_option("qmv_frag", frag)
        try:
            got = ops.qmv(to_dev(w), to_dev(s, dt), to_dev(b, dt), to_dev(x, dt), bits, gs, ctx=ctx).float().cpu().numpy()
        finally:
            ctx.set_option("qmv_frag", 1)
        assert (got[0] == np.inf).all(), frag
        if m > 2:
            assert np.isnan(got[2]).all()
        assert np.isfinite(got[[i for i in range(m) if i not in (0, 2)]]).all()
