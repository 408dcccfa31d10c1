"""Calls issued back to back give what the same calls give with the GPU waited for between them.

The kernels of the library are launched while the kernel before them drains and wait on the device for what it writes.  Here a
consumer follows its producer at once, over buffers that are rewritten with other values every time, so that a value read
before it is written is one of the round before."""
import numpy as np
import pytest

from helpers import dense_case, to_dev

pytestmark = pytest.mark.gpu
ROUNDS = 40


@pytest.fixture(scope="module")
def ctx():
    from metaltile_b200 import ops
    return ops.context(0)


def _same_without_waiting(step, rounds=ROUNDS):
    """``step(i)`` enqueues round i and returns its results: all rounds at once against one at a time."""
    import torch
    want = []
    for i in range(rounds):
        want.append([t.clone() for t in step(i)])
        torch.cuda.synchronize()
    got = [[t.clone() for t in step(i)] for i in range(rounds)]
    torch.cuda.synchronize()
    for i in range(rounds):
        for a, b in zip(got[i], want[i]):
            assert torch.equal(a, b), i


@pytest.mark.parametrize("by_rows", [False, True])
@pytest.mark.parametrize("dt", ["f16", "bf16"])
def test_work_list_of_a_grouped_product(ctx, dt, by_rows):
    """The list of work items and its length are written by the kernel in front of the product (bf16: with the row conversion in
    between): offsets that name 4 rows and 900 in turn."""
    import torch
    from metaltile_b200 import ops
    e, n, k, rows = 8, 256, 512, 900
    w, s, b, x = dense_case(rows, e * n, k, 8, 64, dt, seed=41)
    wd, sd, bd, xd = to_dev(w).view(e, n, -1), to_dev(s, dt).view(e, n, -1), to_dev(b, dt).view(e, n, -1), to_dev(x, dt)
    rng = np.random.default_rng(3)
    lists = []
    for i in range(ROUNDS):
        m = 4 if i % 2 else rows
        owner = np.sort(rng.integers(0, e, size=m))
        off = np.searchsorted(owner, np.arange(e + 1)).astype(np.uint32)
        lists.append((m, to_dev(owner.astype(np.uint32)), to_dev(off)))
    torch.cuda.synchronize()

    def step(i):
        m, owner, off = lists[i]
        kw = dict(indices=owner) if by_rows else dict(expert_offsets=off)
        return [ops.gather_qmm(xd[:m], wd, sd, bd, 8, 64, ctx=ctx, **kw)]

    _same_without_waiting(step)
    assert ctx.status_word() == 0


def _dense(n, k, bits, gs, dt, seed):
    w, s, b, _ = dense_case(1, n, k, bits, gs, dt, seed=seed)
    return to_dev(w), to_dev(s, dt), to_dev(b, dt)


@pytest.mark.parametrize("m,bits,dt", [(1, 4, "bf16"), (1, 5, "f16"), (1, 4, "f32"), (4, 8, "f16"), (8, 4, "bf16"), (8, 8, "f32"), (16, 4, "f16"),
                                       (64, 4, "bf16"), (300, 8, "bf16"), (300, 4, "f16")])
def test_products_behind_swiglu_and_each_other(ctx, m, bits, dt):
    """x of every product is what the launch before it stores: SwiGLU, a product, the row conversion of a prompt in bf16."""
    import torch
    from metaltile_b200 import ops
    n, k = 2048, 1024
    up, down = _dense(n, k, bits, 64, dt, 1), _dense(k, n, bits, 64, dt, 2)
    gen = torch.Generator(device="cuda").manual_seed(m)
    xs = [(torch.randn(m, k, device="cuda", generator=gen) * 0.05).to(up[1].dtype) for _ in range(ROUNDS)]
    act, mid, out = torch.empty_like(xs[0]), xs[0].new_empty(m, n), torch.empty_like(xs[0])

    def step(i):
        ops.swiglu(xs[i], xs[i], out=act, ctx=ctx)
        ops.qmm(*up, act, bits, 64, out=mid, ctx=ctx)
        ops.qmm(*down, mid, bits, 64, out=out, ctx=ctx)
        return [mid, out]

    _same_without_waiting(step)


@pytest.mark.parametrize("kernel", ["stream", "mma", "tc", "cuda"])
@pytest.mark.parametrize("m", [1, 4])
def test_other_small_m_kernels_behind_swiglu(ctx, kernel, m):
    import torch
    from metaltile_b200 import ops
    options = dict(stream=[("qmv_stream", 2)], mma=[("qmv_stream", 0), ("qmv_small_m_mma", 2)], tc=[("qmv_tc", 1)], cuda=[("qmv_stream", 0), ("qmv_small_m_mma", 0)])[kernel]
    mat = _dense(2048, 1024, 4, 64, "bf16", 3)
    xs = [torch.randn(m, 1024, device="cuda").to(torch.bfloat16) for _ in range(ROUNDS)]
    act, out = torch.empty_like(xs[0]), xs[0].new_empty(m, 2048)
    ctx.set_option("qmv_frag", 0)
    for name, v in options:
        ctx.set_option(name, v)
    try:
        def step(i):
            ops.swiglu(xs[i], xs[i], out=act, ctx=ctx)
            return [ops.qmv(*mat, act, 4, 64, out=out, ctx=ctx)]

        _same_without_waiting(step)
    finally:
        for name, v in (("qmv_frag", 1), ("qmv_stream", 1), ("qmv_small_m_mma", 1), ("qmv_tc", 0)):
            ctx.set_option(name, v)


@pytest.mark.parametrize("m,bits,dt", [(1, 4, "bf16"), (1, 3, "f32"), (4, 4, "f16"), (2, 8, "bf16")])
def test_qvm_behind_swiglu(ctx, m, bits, dt):
    import torch
    from metaltile_b200 import ops, synth
    k, n = 2048, 4096
    w = to_dev(synth.words(k * n * bits // 32, seed=4).reshape(k, -1))
    s = (torch.rand(k // 64, n, device="cuda") * 0.01).to(getattr(torch, dict(f32="float32", f16="float16", bf16="bfloat16")[dt]))
    xs = [torch.randn(m, k, device="cuda").to(s.dtype) for _ in range(ROUNDS)]
    act, out = torch.empty_like(xs[0]), xs[0].new_empty(m, n)

    def step(i):
        ops.swiglu(xs[i], xs[i], out=act, ctx=ctx)
        return [ops.qvm(w, s, s, act, bits, 64, out=out, ctx=ctx)]

    _same_without_waiting(step)


@pytest.mark.parametrize("tokens", [4, 200])
def test_a_layer_of_experts(ctx, tokens):
    """Router, sort, experts and unpermute over buffers of their own that every round rewrites; the logits are a SwiGLU's result."""
    import torch
    from metaltile_b200 import ops
    e, h, i_dim = 16, 512, 256
    mats = [tuple(t.view(e, -1, t.shape[-1]) for t in _dense(e * o, k, 4, 64, "bf16", 5 + j)) for j, (o, k) in enumerate(((i_dim, h), (i_dim, h), (h, i_dim)))]
    xs = [torch.randn(tokens, h, device="cuda").to(torch.bfloat16) for _ in range(ROUNDS)]
    raw = [torch.randn(tokens, e, device="cuda").to(torch.bfloat16) for _ in range(ROUNDS)]
    logits, x, y, out = torch.empty_like(raw[0]), torch.empty_like(xs[0]), xs[0].new_empty(tokens * 4, h), torch.empty_like(xs[0])

    def step(i):
        ops.swiglu(xs[i], xs[i], out=x, ctx=ctx)
        ops.swiglu(raw[i], raw[i], out=logits, ctx=ctx)
        idx, wts = ops.moe_router_topk(logits, 4, ctx=ctx)
        order, inverse, offsets, _ = ops.moe_sort(idx, e, ctx=ctx)
        ops.moe_experts(x, *mats, 4, 64, offsets, sort_token_idx=order, out=y, ctx=ctx)
        return [idx, wts, ops.moe_unpermute(y, inverse, wts, out=out, ctx=ctx)]

    _same_without_waiting(step)


@pytest.mark.parametrize("bits,dt", [(4, "bf16"), (3, "f16"), (8, "f32")])
def test_codec_behind_swiglu_and_itself(ctx, bits, dt):
    """Values just computed are quantized, read back and quantized again."""
    import torch
    from metaltile_b200 import ops
    dtype = dict(f32=torch.float32, f16=torch.float16, bf16=torch.bfloat16)[dt]
    xs = [torch.randn(512, 1024, device="cuda").to(dtype) for _ in range(ROUNDS)]
    act = torch.empty_like(xs[0])

    def step(i):
        ops.swiglu(xs[i], xs[i], out=act, ctx=ctx)
        q = ops.affine_quantize(act, bits, 64, ctx=ctx)
        back = ops.affine_dequantize(*q, bits, 64, ctx=ctx)
        return [*q, back, *ops.affine_quantize(back, bits, 64, ctx=ctx)]

    _same_without_waiting(step)


PRODUCTS = {
    # kernel: (m, n, k, bits, dt, options)
    "frag": (1, 1024, 2048, 4, "bf16", {}), "frag_8bit": (4, 1024, 2048, 8, "f16", {}), "frag_f32": (8, 1024, 2048, 4, "f32", {}),
    "stream": (1, 4096, 2048, 4, "bf16", dict(qmv_frag=0)), "ring": (8, 1024, 2048, 4, "bf16", {}), "mma": (8, 1024, 2048 - 64, 4, "f16", dict(qmv_frag=0)),
    "cuda": (1, 1024, 2048, 5, "bf16", dict(qmv_frag=0)), "tc": (2, 1024, 2048, 4, "bf16", dict(qmv_tc=1)),
    "qmm": (200, 1024, 2048, 4, "f16", {}), "qmm_bf16": (200, 1024, 2048, 8, "bf16", {}), "grouped": (64, 2048, 1024, 4, "f16", {}),
    "qvm": (1, 2048, 1024, 4, "bf16", {}), "qvm_mma": (4, 4096, 2048, 4, "f16", {}),
}


@pytest.mark.parametrize("early", [1, 0])
@pytest.mark.parametrize("between", [False, True])
@pytest.mark.parametrize("kind", sorted(PRODUCTS))
def test_products_of_weights_just_quantized(ctx, kind, between, early):
    """Packed words, scales and biases are rewritten in place by the quantizer and used at once: by the product behind it, by a second
    one behind that, and with another kernel (which lets the product start while the quantizer may still run) in between."""
    import torch
    from metaltile_b200 import ops
    from metaltile_b200.ops import _TORCH_DT
    m, n, k, bits, dt, options = PRODUCTS[kind]
    dtype = dict(f32=torch.float32, f16=torch.float16, bf16=torch.bfloat16)[dt]
    rounds = 16
    gen = torch.Generator(device="cuda").manual_seed(7)
    # qvm: groups along K of a transposed matrix; its words are those of [k, n] and its scales are made separately
    qvm = kind.startswith("qvm")
    shape = (k, n) if qvm else (n, k)
    ws = [torch.randn(shape, device="cuda", generator=gen).to(dtype) for _ in range(rounds)]
    q = [t.clone() for t in ops.affine_quantize(ws[0], bits, 64, ctx=ctx)]
    t_s = torch.rand(k // 64, n, device="cuda", generator=gen).to(dtype)
    x = torch.randn(m, k, device="cuda", generator=gen).to(dtype)
    junk = torch.empty_like(x)
    offsets = torch.tensor([0, m // 2, m // 2, m], dtype=torch.int32, device="cuda")

    def product():
        if qvm:
            return ops.qvm(q[0], t_s, t_s, x, bits, 64, ctx=ctx)
        if kind == "grouped":
            return ops.gather_qmm(x, *(t[:n // 3 * 3].view(3, n // 3, -1) for t in q), bits, 64, expert_offsets=offsets, ctx=ctx)
        return ops.qmm(*q, x, bits, 64, ctx=ctx)

    def step(i):
        ctx.affine_quantize(ws[i].data_ptr(), q[0].data_ptr(), q[1].data_ptr(), q[2].data_ptr(), ws[i].numel(), bits, 64, _TORCH_DT[dtype],
                            stream=torch.cuda.current_stream().cuda_stream)
        if between:
            ops.swiglu(x, x, out=junk, ctx=ctx)
        return [product(), product()]

    for name, v in dict(options, pdl_early_weights=early).items():
        ctx.set_option(name, v)
    try:
        _same_without_waiting(step, rounds)
    finally:
        for name, v in dict(qmv_frag=1, qmv_tc=0, pdl_early_weights=1).items():
            ctx.set_option(name, v)
