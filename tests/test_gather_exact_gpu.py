"""The exact grouped 4-bit bf16 kernel (csrc/gather_exact.cu): edges of its columns, k blocks, stages, halves and rows of scales against 64-bit sums,
powers of two of rows and tokens at the ends of their ranges, infinities, what stays inside its token, what it reports, and the fused layer against the
separate entries."""
import pytest

from test_gather_frag_gpu import _codes, _offsets, _stack

pytestmark = pytest.mark.gpu


def _product(torch, ops, ctx, counts, n, k, g, change=None, x_change=None, seed=0):
    """(got, ref, bound) of one product; mags: what the bound is in terms of."""
    gen = torch.Generator(device="cuda").manual_seed(seed + 31 * n + k)
    e, m = len(counts), sum(counts)
    w, s, b = _stack(torch, e, n, k, 4, g, torch.bfloat16, gen)
    x = torch.randn((m, k), device="cuda", generator=gen).to(torch.bfloat16)
    if change:
        s, b = change(s, b)
    if x_change:
        x = x_change(x)
    out = torch.full((m + 1, n), 7.0, dtype=torch.bfloat16, device="cuda")
    ops.gather_qmm(x, w, s, b, 4, g, expert_offsets=_offsets(torch, counts), out=out[:m], ctx=ctx)
    again = ops.gather_qmm(x, w, s, b, 4, g, expert_offsets=_offsets(torch, counts), ctx=ctx)
    torch.cuda.synchronize()
    assert ctx.status_word() == 0 and bool((out[m] == 7.0).all())
    assert torch.equal(out[:m].nan_to_num(3.0), again.nan_to_num(3.0))
    refs, bounds, row = [], [], 0
    steps = k // 16 + 4 * ((k // 64 + 7) // 8)
    for i, c in enumerate(counts):
        sd, bd = (t[i].double().repeat_interleave(g, 1) for t in (s, b))
        xs = x[row:row + c].double()
        wd = _codes(torch, w[i], 4, k).double() * sd + bd
        mag = xs.abs() @ (16 * sd.abs() + bd.abs()).T
        # rounded to bf16 once; a chain of steps, each truncated to 24 bits
        refs.append(xs @ wd.T)
        bounds.append(2.0 ** -8 * refs[-1].abs() + 2.0 ** -23 * steps * mag + 2.0 ** -133)
        row += c
    return out[:m], torch.cat(refs), torch.cat(bounds)


CASES = [([1, 15, 16, 17], 64, 64, 64), ([31, 0, 32, 33], 72, 128, 64), ([47, 48, 49], 200, 192, 64), ([63, 64, 65, 0, 130], 128, 320, 64),
         ([9, 300], 136, 256, 128), ([40, 7, 25], 64, 640, 128), ([20, 21], 264, 1088, 64), ([5, 36], 320, 2048, 64), ([30], 8, 448, 64),
         ([12, 6, 44], 96, 4096, 64), ([18] * 40, 64, 128, 128),
         # long rows of scales: the most for 64 columns, one more, the most for 48, one more, the most for 32
         ([64, 41], 64, 4032, 64), ([64, 41], 64, 4096, 64), ([48, 49], 64, 5568, 64), ([48, 49], 64, 5632, 64), ([33, 64], 64, 7104, 64)]


@pytest.mark.parametrize("counts,n,k,g", CASES)
def test_products(counts, n, k, g):
    import torch
    from metaltile_b200 import ops

    ctx = ops.context()
    assert ctx.gather_qmm_route(sum(counts), n, k, len(counts), 4, g, "bf16") == "gather_qmm_exact"
    got, ref, bound = _product(torch, ops, ctx, counts, n, k, g)
    assert bool(((got.double() - ref).abs() <= bound).all())


@pytest.mark.parametrize("g,k", [(64, 512), (64, 320), (128, 640)])            # rows of scales on boundaries of 16 bytes, of 2, of 2
@pytest.mark.parametrize("what", ["rows", "groups", "zeros", "biases", "negative", "most", "outlier 9", "outlier 14", "outlier 29", "outlier 30", "outlier 60"])
def test_scales_of_every_size(what, g, k):
    """Also of one row: as far apart as either form of the operands holds, and farther."""
    import torch
    from metaltile_b200 import ops

    def change(s, b):
        e, n, g = s.shape
        if what == "rows":                                   # a power of two a row, from 2^-40 to 2^40
            p = torch.exp2(torch.linspace(-40, 40, n, device="cuda").round())[None, :, None]
        elif what == "groups":                               # within a row up to 2^14 apart
            p = torch.exp2((torch.arange(g, device="cuda") * 7 % 15).float())[None, None, :]
        else:
            p = torch.ones((), device="cuda")
        s, b = s.float() * p, b.float() * p
        if what == "zeros":
            s[:, ::3] = 0
            b[:, ::6] = 0
            s[:, 1::4, 1] = 0
        if what == "biases":
            b = b * 4096
        if what == "negative":
            s = -s
        if what == "most":                                   # biases of rows without scales, and with scales far below them
            s[:, 1::2] *= 2.0 ** -20
            s[:, ::4] = 0
        if what.startswith("outlier"):                       # a group of some rows, where the tokens are zero: what is left is the others'
            s[:, ::5, 1] *= 2.0 ** int(what[8:])
            b[:, ::7, 1] *= 2.0 ** int(what[8:])
        return s.to(torch.bfloat16), b.to(torch.bfloat16)

    def no_outlier(x):
        x = x.clone()
        if what.startswith("outlier"):
            x[::2, g:2 * g] = 0
        return x

    got, ref, bound = _product(torch, ops, ops.context(), [20, 0, 37], 192, k, g, change, no_outlier)
    assert bool(torch.isfinite(got).all()) and bool(((got.double() - ref).abs() <= bound).all())


def test_tokens_of_every_size():
    """Rows of x from 2^-100 to 2^100; an infinity and a NaN stay in their tokens."""
    import torch
    from metaltile_b200 import ops

    m = 45
    p = torch.exp2(torch.linspace(-100, 100, m, device="cuda").round())[:, None]
    got, ref, bound = _product(torch, ops, ops.context(), [m], 64, 256, 64, x_change=lambda x: (x.float() * p).to(torch.bfloat16))
    assert bool(((got.double() - ref).abs() <= bound).all())

    def odd(x):
        x = x.clone()
        x[3, 17], x[20, 200] = float("inf"), float("nan")
        x[30] = 0
        return x

    got, ref, bound = _product(torch, ops, ops.context(), [30, 15], 64, 256, 64, x_change=odd)
    keep = [i for i in range(m) if i not in (3, 20)]
    assert not bool(torch.isfinite(got[3]).any()) and bool(got[20].isnan().all()) and bool((got[30] == 0).all())
    assert bool(((got.double() - ref).abs() <= bound)[keep].all())


@pytest.mark.parametrize("g,k", [(64, 256), (128, 640)])
def test_infinities_are_what_the_definition_gives(g, k):
    """An infinite activation, bias or scale: infinities of the products' signs, NaN where two signs meet (or a weight of zero); others are as without it."""
    import torch
    from metaltile_b200 import ops

    inf = float("inf")

    def odd(x):
        x = x.clone()
        x[3, 17], x[7, 130], x[20, 200], x[20, 3] = inf, -inf, float("nan"), inf
        x[33, 5], x[33, k - 1] = inf, -inf
        return x

    def change(s, b):
        s, b = s.clone(), b.clone()
        b[0, 9, 1], b[1, 70, 0], s[1, 71, 2] = inf, -inf, inf
        return s, b

    got, ref, bound = _product(torch, ops, ops.context(), [30, 15], 136, k, g, change, odd)
    finite = torch.isfinite(ref)
    assert bool(((got.double() - ref).abs() <= bound)[finite].all())
    assert torch.equal(got[~finite].double().nan_to_num(7.0, 1.0, -1.0), ref[~finite].nan_to_num(7.0, 1.0, -1.0))
    assert bool(finite[8].any()) and bool((ref[3] == inf).any()) and bool((ref[3] == -inf).any()) and not bool(finite[[3, 7, 20, 33]].any())


@pytest.mark.parametrize("tokens,e,top,hidden,inter,g", [(40, 8, 2, 512, 320, 64), (90, 16, 8, 384, 256, 128), (100, 8, 4, 448, 200 * 8, 64),
                                                               (40, 4, 4, 4096, 320, 64),       # passes of 48 rows, then of 64
                                                               (6, 4, 2, 8192, 256, 64), (40, 4, 2, 8192, 256, 64), (30, 4, 2, 7168, 320, 64)])      # down alone
@pytest.mark.parametrize("odd", [False, True])
def test_layer_equals_the_separate_entries(tokens, e, top, hidden, inter, g, odd):
    """odd: infinite tokens, rows of gate, up and down with scales far apart and farther: what is added up from the definition, on both sides of the pair."""
    import torch
    from metaltile_b200 import ops

    gen = torch.Generator(device="cuda").manual_seed(tokens)
    gate, up, down = (_stack(torch, e, n, k, 4, g, torch.bfloat16, gen) for n, k in ((inter, hidden), (inter, hidden), (hidden, inter)))
    x = torch.randn((tokens, hidden), device="cuda", generator=gen).to(torch.bfloat16)
    if odd:
        x[1, 5], x[3, hidden - 1], x[4, 0] = float("inf"), -float("inf"), float("nan")
        for m, far in ((gate, 40), (up, 35), (down, 60)):
            m[1][:, ::9, 1] *= 2.0 ** far
            m[1][:, 1::7, 0] *= 2.0 ** -20
            m[2][:, 3, 1] = float("inf")
    idx, _ = ops.moe_router_topk(torch.randn((tokens, e), device="cuda", generator=gen).to(torch.bfloat16), top)
    order, _, off, _ = ops.moe_sort(idx, e)
    fused = ops.moe_experts(x, gate, up, down, 4, g, off, sort_token_idx=order)
    rows = ops.moe_permute(x, order)
    act = ops.swiglu(ops.gather_qmm(rows, *gate, 4, g, expert_offsets=off), ops.gather_qmm(rows, *up, 4, g, expert_offsets=off))
    separate = ops.gather_qmm(act, *down, 4, g, expert_offsets=off)
    assert torch.equal(fused.nan_to_num(7.0), separate.nan_to_num(7.0)) and (odd or bool(torch.isfinite(fused).all()))
    assert ops.context().status_word() == 0


def test_reports_what_does_not_exist():
    """Offsets past the rows or backwards: clamped, 0x901.  A row index past x: row 0 is read instead, 0x903."""
    import torch
    from metaltile_b200 import Context, MetalTileError, ops

    ctx = Context(0)
    gen = torch.Generator(device="cuda").manual_seed(5)
    e, n, k, g, m = 3, 200, 320, 64, 60
    assert ctx.gather_qmm_route(m, n, k, e, 4, g, "bf16") == ctx.gather_qmm_route(m, k, n * 8, e, 4, g, "bf16") == "gather_qmm_exact"
    w, s, b = _stack(torch, e, n, k, 4, g, torch.bfloat16, gen)
    x = torch.randn((m, k), device="cuda", generator=gen).to(torch.bfloat16)

    def reported(code):
        with pytest.raises(MetalTileError):
            ctx.sync(torch.cuda.current_stream().cuda_stream)
        assert ctx.status_word() == code
        ctx.status_clear()

    for off, same in (([0, 20, 1000, 1001], [0, 20, 60, 60]), ([0, 40, 10, 60], None)):
        out = torch.full((m + 1, n), 7.0, dtype=torch.bfloat16, device="cuda")
        ops.gather_qmm(x, w, s, b, 4, g, expert_offsets=torch.tensor(off, dtype=torch.int32, device="cuda"), out=out[:m], ctx=ctx)
        reported(0x901)
        assert bool((out[m] == 7.0).all())
        if same:
            assert torch.equal(out[:m], ops.gather_qmm(x, w, s, b, 4, g, expert_offsets=torch.tensor(same, dtype=torch.int32, device="cuda"), ctx=ctx))
    gate, up, down = (_stack(torch, e, a, c, 4, g, torch.bfloat16, gen) for a, c in ((192, k), (192, k), (k, 192)))
    order, off = torch.arange(m, dtype=torch.int32, device="cuda") % 50, _offsets(torch, [25, 20, 15])
    order[7], order[33] = 50, -1                             # not rows of the first 50
    got = ops.moe_experts(x[:50], gate, up, down, 4, g, off, sort_token_idx=order, ctx=ctx)
    reported(0x903)
    order[7] = order[33] = 0
    assert torch.equal(got, ops.moe_experts(x[:50], gate, up, down, 4, g, off, sort_token_idx=order, ctx=ctx)) and ctx.status_word() == 0


def test_long_rows_of_scales_take_narrower_passes():
    from metaltile_b200 import _lib
    from metaltile_b200.context import _dt

    route = lambda k, rows, dt="bf16": _lib.load().mtc_gather_qmm_route(8 * rows, 1536, k, 8, 4, 64, _dt(dt)).decode()  # noqa: E731
    assert {route(64 * g, 300) for g in (63, 64, 87, 88, 111)} == {"gather_qmm_exact"}
    assert route(64 * 112, 300) == route(64 * 112, 300, "f16") == "gather_qmm_tcgen05"


def test_rule():
    from metaltile_b200 import _lib
    from metaltile_b200.context import _dt

    def route(m, n, k, e, bits=4, g=64, dt="bf16"):
        return _lib.load().mtc_gather_qmm_route(m, n, k, e, bits, g, _dt(dt)).decode()

    frag, exact, tc = "gather_qmm_frag", "gather_qmm_exact", "gather_qmm_tcgen05"
    assert [route(m, 768, 1088, 32) for m in (48, 49, 512 * 32, 512 * 32 + 1)] == [frag, exact, exact, tc]
    assert [route(m, 832, 2112, 128) for m in (32, 33)] == [frag, exact]
    # where the streaming kernel takes the shape, rows an expert by the size of an expert's matrix
    for n, k, e, rows in ((1024, 512, 128, 8), (512, 768, 64, 0.5), (1536, 512, 128, 8), (768, 2048, 128, 6), (1536, 2048, 64, 5)):
        assert [route(m, n, k, e) for m in (int(rows * e), int(rows * e) + 1)] == [frag if rows < 1 else "gather_qmm_stream", exact], (n, k, e)
    assert [route(m, 832, 2112, 128, dt="f16") for m in (33, 1300)] == [frag, tc]
