"""The grouped fragment kernel (csrc/gather_frag.cuh): every width and form against 64-bit sums, experts without rows and with several passes,
ragged weight rows and K, both sides of its rule, what it reports, and the fused layer against the separate entries."""
import pytest

pytestmark = pytest.mark.gpu


def _codes(torch, w, bits, k):
    shift = torch.arange(k, device=w.device) * bits
    v = w.to(torch.int64) & 0xFFFFFFFF
    nxt = torch.clamp(shift // 32 + 1, max=w.shape[-1] - 1)
    q = v[..., shift // 32] >> (shift % 32)
    return torch.where(shift % 32 + bits > 32, q | (v[..., nxt] << (32 - shift % 32)), q) & ((1 << bits) - 1)


def _stack(torch, e, n, k, bits, g, td, gen):
    w = torch.randint(-2 ** 31, 2 ** 31, (e, n, k * bits // 32), dtype=torch.int32, device="cuda", generator=gen)
    s = (0.002 + 0.018 * torch.rand((e, n, k // g), device="cuda", generator=gen)) * (16.0 / 2 ** bits)
    return w, s.to(td), (-(2.0 ** (bits - 1)) * s + 1e-3 * torch.randn((e, n, k // g), device="cuda", generator=gen)).to(td)


def _offsets(torch, counts):
    return torch.tensor([sum(counts[:i]) for i in range(len(counts) + 1)], dtype=torch.int32, device="cuda")


CASES = [(b, g, dt, counts, n, k) for b, dt in ((2, "bf16"), (3, "f16"), (4, "bf16"), (5, "bf16"), (6, "f16"), (8, "bf16"))
         for g, counts, n, k in ((32, [1] + [0] * 6 + [1, 0], 33, 96), (64, [3, 0, 1, 5], 16, 192), (32, [9, 0, 2], 48, 1056), (128, [0, 17, 8, 1, 1], 130, 640),
                                 (32, [6, 3], 24, 64))]


@pytest.mark.parametrize("bits,g,dt,counts,n,k", CASES)
def test_grouped_products(bits, g, dt, counts, n, k):
    import torch
    from metaltile_b200 import ops

    gen = torch.Generator(device="cuda").manual_seed(bits * 100 + k)
    td = dict(bf16=torch.bfloat16, f16=torch.float16)[dt]
    ctx, e, m = ops.context(), len(counts), sum(counts)
    assert ctx.gather_qmm_route(m, n, k, e, bits, g, dt) == "gather_qmm_frag"
    w, s, b = _stack(torch, e, n, k, bits, g, td, gen)
    x = torch.randn((m, k), device="cuda", generator=gen).to(td)
    out = torch.full((m + 1, n), 7.0, dtype=td, device="cuda")
    ops.gather_qmm(x, w, s, b, bits, g, expert_offsets=_offsets(torch, counts), out=out[:m])
    torch.cuda.synchronize()
    assert ctx.status_word() == 0 and bool((out[m] == 7.0).all())
    row = 0
    for i, c in enumerate(counts):
        q = _codes(torch, w[i], bits, k).double() * s[i].double().repeat_interleave(g, 1)
        bias, xs = b[i].double().repeat_interleave(g, 1), x[row:row + c].double()
        ref, mag = xs @ (q + bias).T, xs.abs() @ (q.abs() + bias.abs()).T
        # rounded to the output type once; a group's chain of truncated MMA steps, the groups and the warps' parts in 32 bits
        bound = (2.0 ** -8 if dt == "bf16" else 2.0 ** -11) * ref.abs() + 2.0 ** -23 * (24 + (k // g) ** 0.5) * mag
        assert bool(((out[row:row + c].double() - ref).abs() <= bound).all())
        row += c


@pytest.mark.parametrize("tokens,e,top,hidden,inter,bits,g,dt", [
    (5, 16, 2, 512, 256, 8, 64, "bf16"), (40, 8, 2, 320, 224, 6, 32, "f16"), (3, 32, 1, 512, 256, 4, 64, "bf16"), (12, 8, 4, 512, 320, 4, 64, "f16")])
def test_layer_equals_the_separate_entries(tokens, e, top, hidden, inter, bits, g, dt):
    """Also where the streaming kernel takes some of the products and this one the others."""
    import torch
    from metaltile_b200 import ops

    gen = torch.Generator(device="cuda").manual_seed(tokens)
    td = dict(bf16=torch.bfloat16, f16=torch.float16)[dt]
    gate, up, down = (_stack(torch, e, n, k, bits, g, td, gen) for n, k in ((inter, hidden), (inter, hidden), (hidden, inter)))
    x = torch.randn((tokens, hidden), device="cuda", generator=gen).to(td)
    idx, _ = ops.moe_router_topk(torch.randn((tokens, e), device="cuda", generator=gen).to(td), top)
    order, _, off, _ = ops.moe_sort(idx, e)
    fused = ops.moe_experts(x, gate, up, down, bits, g, off, sort_token_idx=order)
    rows = ops.moe_permute(x, order)
    act = ops.swiglu(ops.gather_qmm(rows, *gate, bits, g, expert_offsets=off), ops.gather_qmm(rows, *up, bits, g, expert_offsets=off))
    assert torch.equal(fused, ops.gather_qmm(act, *down, bits, g, expert_offsets=off))
    assert ops.context().status_word() == 0


def test_bad_offsets_and_rows_are_reported():
    import torch
    from metaltile_b200 import MetalTileError, ops

    gen = torch.Generator(device="cuda").manual_seed(9)
    ctx, mats = ops.context(), [_stack(torch, 4, n, k, 8, 32, torch.bfloat16, gen) for n, k in ((64, 128), (64, 128), (128, 64))]
    x = torch.randn((4, 128), device="cuda", generator=gen).to(torch.bfloat16)
    good, order = torch.tensor([0, 1, 2, 3, 4], dtype=torch.int32, device="cuda"), torch.tensor([2, 0, 3, 1], dtype=torch.int32, device="cuda")
    for off, src, code in ((torch.tensor([0, 2, 900, 4, 4], dtype=torch.int32, device="cuda"), order, 0x901), (good, order + 2, 0x903)):
        try:
            ops.moe_experts(x, *mats, 8, 32, off, sort_token_idx=src)
            with pytest.raises(MetalTileError):
                ctx.sync(torch.cuda.current_stream().cuda_stream)
            assert ctx.status_word() == code
        finally:
            ctx.status_clear()


def test_rule():
    from metaltile_b200 import _lib
    from metaltile_b200.context import _dt

    def route(m, n, k, e, bits, g, dt="bf16"):
        return _lib.load().mtc_gather_qmm_route(m, n, k, e, bits, g, _dt(dt)).decode()

    frag, stream, tc = "gather_qmm_frag", "gather_qmm_stream", "gather_qmm_tcgen05"
    assert [route(m, 768, 2048, 128, 4, 64) for m in (64, 65)] == [frag, stream]
    assert [route(m, 512, 1024, 16, 4, 64) for m in (64, 65)] == [frag, "gather_qmm_exact"]
    assert [route(m, 768, 2048, 128, 8, 64) for m in (512, 513)] == [frag, tc]
    assert [route(m, 768, 1024, 32, 6, 32) for m in (320, 321)] == [frag, tc]
    assert route(8, 768, 2048, 128, 8, 64, "f32") == "gather_qmm_cuda_core"
