"""The tensor-memory product on both of its ways to an operand (packed halves; through f32 for scales and biases beyond their range), on each way that
scales reach the chip, at the edges of its tiles and rings: against the float64 product of the dequantised weights."""
import pytest

pytestmark = pytest.mark.gpu

CASES = [
    # m, n, k, bits, group, type, factor of the scales, elements that the scale arrays are off a 16-byte boundary, options
    (64, 130, 1088, 4, 64, "bf16", 1.0, 0, {}), (65, 256, 2048, 4, 128, "f16", 16.0, 0, {}), (200, 100, 2048, 3, 32, "bf16", 1.0, 2, {}), (200, 136, 1024, 4, 64, "f16", 1.0, 1, {}),
    (257, 128, 1024, 8, 64, "f16", 1.0, 0, {}), (129, 640, 960, 5, 32, "f16", 1.0, 8, {}), (300, 72, 1472, 6, 64, "bf16", 64.0, 2, {}),
    (192, 384, 4096, 2, 64, "bf16", 2.0 ** -12, 0, {}), (333, 200, 2880, 8, 32, "f16", 8.0, 0, {}), (100, 96, 1024, 4, 256, "bf16", 1.0, 0, {}),
    (300, 260, 1536, 4, 64, "f16", 1.0, 0, {"qmm_max_stages": 1}), (300, 260, 1536, 8, 32, "bf16", 1.0, 0, {"qmm_max_stages": 2}),
] + [(513, 20000, 512, 4, 64, "bf16", 1.0, 0, {"qmm_tile_tokens": tn}) for tn in (16, 128, 144, 192, 208, 256)]


@pytest.mark.parametrize("m,n,k,bits,g,dt,factor,off,options", CASES)
def test_product_against_float64(m, n, k, bits, g, dt, factor, off, options):
    import torch
    from metaltile_b200 import Context, ops
    from test_gather_frag_gpu import _codes

    gen = torch.Generator(device="cuda").manual_seed(m + n)
    td = dict(bf16=torch.bfloat16, f16=torch.float16)[dt]

    def placed(v):
        room = torch.zeros(v.numel() + 8, dtype=td, device="cuda")[off:off + v.numel()].view(v.shape)
        return room.copy_(v)

    w = torch.randint(-2 ** 31, 2 ** 31, (n, k * bits // 32), dtype=torch.int32, device="cuda", generator=gen)
    s = (0.002 + 0.018 * torch.rand((n, k // g), device="cuda", generator=gen)) * (16.0 / 2 ** bits) * factor
    b = -(2.0 ** (bits - 1)) * s * (1 + 0.1 * torch.randn((n, k // g), device="cuda", generator=gen))
    s[0], s[1], b[2] = 0.0, -s[1], 0.0                     # a row of biases, one of negative scales, one without biases
    s[3, 0] = 200.0 / 2 ** bits                            # one group of a row beyond what packed halves take
    s, b = placed(s), placed(b)
    x = torch.randn((m, k), device="cuda", generator=gen).to(td)
    ctx = Context(0)
    for name, value in options.items():
        ctx.set_option(name, value)
    assert ctx.launch_of(m, [n], k, bits, g, dt)["kernel"] == "qmm_tcgen05"
    got = ops.qmm(w, s, b, x, bits, g, ctx=ctx)
    torch.cuda.synchronize()
    assert ctx.status_word() == 0
    weights = _codes(torch, w, bits, k).double() * s.double().repeat_interleave(g, 1) + b.double().repeat_interleave(g, 1)
    want = x.double() @ weights.T
    # a weight is rounded twice at most (the bias, then the sum: 2^-11 of each, or half of the least subnormal), the sum has 32 bits, the result one
    # rounding of its type
    per_weight = 2.0 ** -11 * (weights.abs() + b.double().abs().repeat_interleave(g, 1)) + 2.0 ** -25
    mag = x.double().abs() @ weights.abs().T
    bound = x.double().abs() @ per_weight.T + (k / 16 + 16) * 2.0 ** -24 * mag + (2.0 ** -8 if dt == "bf16" else 2.0 ** -11) * want.abs() + 2.0 ** -25
    assert bool(((got.double() - want).abs() <= bound).all())


@pytest.mark.parametrize("g", [32, 64])
@pytest.mark.parametrize("bits", [2, 3, 5, 6])
def test_a_weight_is_rounded_once(bits, g):
    """Scale and bias just below half of the least f16, codes of one: their sum is that f16, and each alone would be rounded to nothing."""
    import torch
    from metaltile_b200 import ops

    m, n, k = 40, 136, 512
    row = 0
    for i in range(k):
        row |= 1 << (i * bits)
    words = [(row >> (32 * i)) & 0xFFFFFFFF for i in range(k * bits // 32)]
    w = torch.tensor(words, dtype=torch.int64, device="cuda").to(torch.int32).expand(n, -1).contiguous()
    s = torch.full((n, k // g), 255 * 2.0 ** -33, dtype=torch.bfloat16, device="cuda")
    x = torch.full((m, k), 1024.0, dtype=torch.bfloat16, device="cuda")
    assert ops.context().launch_of(m, [n], k, bits, g, "bf16")["kernel"] == "qmm_tcgen05"
    assert bool((ops.qmm(w, s, s, x, bits, g).double() == k * 1024 * 2.0 ** -24).all())
