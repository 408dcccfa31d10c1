"""The vector-matrix product of one token whose codes pass through shared memory, against the float64 product of the dequantised weights: column
counts that end inside a tile and inside a copy's row of lanes, chunks and ranges of K that end inside a group, groups of one unit and longer than a
warp's range, one column tile whose K is spread over 32 CTAs, the first sizes on both sides of the rule.  On random operands, where the bound of the longest
sums is wide, and on ones whose sums are exact."""
import pytest

pytestmark = pytest.mark.gpu


SHAPES = [
    (2080, 2064, 4, 16, "bf16"), (1056, 4128, 4, 48, "f32"), (4128, 1024, 4, 1024, "f16"), (32, 131104, 4, 32, "bf16"), (1024, 4096, 4, 64, "f32"),
    (1024, 4080, 4, 16, "f32"), (528, 24000, 8, 64, "f32"), (2064, 6144, 8, 128, "bf16"), (32, 393216, 8, 32, "f16"), (19024, 672, 8, 16, "f16"),
    (37920, 128, 4, 64, "bf16"), (1028, 16384, 8, 64, "f32"),
]


@pytest.mark.parametrize("n,k,bits,g,dt", SHAPES)
def test_every_code_counts_once(n, k, bits, g, dt):
    """Operands whose sums are exact in 32 bits, so that the result is the exact one, rounded once: a row, a unit, a range or a chunk left out, taken twice or
    met with other scales would show in nearly every column."""
    import torch
    from metaltile_b200 import ops

    gen = torch.Generator(device="cuda").manual_seed(n + 1)
    td = dict(bf16=torch.bfloat16, f16=torch.float16, f32=torch.float32)[dt]
    w = torch.randint(-2 ** 31, 2 ** 31, (k, n * bits // 32), dtype=torch.int32, device="cuda", generator=gen)
    # x is zero but in about a thousand rows, the first and the last of each range of 16 units among them; |sums| < 2^24 in units of 2^-10
    x = torch.randint(1, 4, (1, k), device="cuda", generator=gen) * (2 * torch.randint(0, 2, (1, k), device="cuda", generator=gen) - 1)
    x = x * (torch.rand((1, k), device="cuda", generator=gen) < min(1.0, 700 / k))
    x[:, ::max(16, k // 512 // 16 * 16)] = 1
    x[:, -1] = 2
    s = 2.0 ** -torch.randint(0, 4, (k // g, n), device="cuda", generator=gen)
    b = torch.randint(-4, 5, (k // g, n), device="cuda", generator=gen).double()
    if bits == 8:
        s, b = s * 2.0 ** -4, b * 0.5
    if dt == "f16":                                           # within the type's range
        s, b = s * 2.0 ** -4, b * 2.0 ** -4
    got = ops.qvm(w, s.to(td), b.to(td), x.to(td), bits, g)
    q = torch.stack([(w >> (i * bits)) & (2 ** bits - 1) for i in range(32 // bits)], -1).reshape(k, n)
    rows = x[0].nonzero()[:, 0]
    xr, of = x[:, rows].double(), rows // g
    weights = q[rows].double() * s.double()[of] + b[of]
    mag = xr.abs() @ (q[rows].double() * s.double()[of] + b.abs()[of])
    assert float(mag.max()) < 2.0 ** 24 * float((2.0 ** -3 * (2.0 ** -4 if bits == 8 else 1.0) * (2.0 ** -4 if dt == "f16" else 1.0)))
    assert torch.equal(got, (xr @ weights).to(td))


@pytest.mark.parametrize("dt", ["bf16", "f16", "f32"])
def test_sums_are_those_of_units(dt):
    """One group as long as 32 warps' ranges: units of 16 rows add up by themselves, then the units, the warps, the chunks, each in order.  Columns of sums that
    cancel, so that the order shows in the result."""
    import torch
    from metaltile_b200 import ops

    n, k, chunks, warps = 256, 1 << 18, 32, 16
    gen = torch.Generator(device="cuda").manual_seed(3)
    td = dict(bf16=torch.bfloat16, f16=torch.float16, f32=torch.float32)[dt]
    w = torch.randint(-2 ** 31, 2 ** 31, (k, n // 8), dtype=torch.int32, device="cuda", generator=gen)
    w[k // 2:] = w[:k // 2].roll(208, 0)
    x = (0.0625 + 1.9 * torch.rand(k, device="cuda", generator=gen)).to(td if dt != "f32" else torch.float16)
    x[k // 2:] = -x[:k // 2].roll(208)
    one, zero = torch.ones((k // 16384, n), dtype=td, device="cuda"), torch.zeros((k // 16384, n), dtype=td, device="cuda")
    got = ops.qvm(w, one, zero, x.to(td)[None], 4, 16384)
    q = torch.stack([(w >> (4 * i)) & 15 for i in range(8)], -1).reshape(k, n)
    units = (x.double()[:, None] * q.double()).view(k // 16, 16, n).sum(1)
    assert torch.equal(units.float().double(), units)         # those of 16 rows are exact in 32 bits

    def in_order(v, dim):
        total = torch.zeros_like(v.select(dim, 0))
        for i in range(v.shape[dim]):
            total = total + v.select(dim, i)
        return total

    want = in_order(in_order(in_order(units.float().view(chunks, warps, -1, n), 2), 1), 0)
    assert torch.equal(got[0], want.to(td)) and float((want.double() - units.sum(0)).abs().max()) > 0


@pytest.mark.parametrize("n,k,bits,g,dt", SHAPES)
def test_against_float64(n, k, bits, g, dt):
    import torch
    from metaltile_b200 import ops

    gen = torch.Generator(device="cuda").manual_seed(n)
    td = dict(bf16=torch.bfloat16, f16=torch.float16, f32=torch.float32)[dt]
    w = torch.randint(-2 ** 31, 2 ** 31, (k, n * bits // 32), dtype=torch.int32, device="cuda", generator=gen)
    s = ((0.002 + 0.018 * torch.rand((k // g, n), device="cuda", generator=gen)) * (16.0 / 2 ** bits)).to(td)
    b = (-(2.0 ** (bits - 1)) * s.float() * (1 + 0.1 * torch.randn((k // g, n), device="cuda", generator=gen))).to(td)
    x = torch.randn((1, k), device="cuda", generator=gen).to(td)
    got, again = ops.qvm(w, s, b, x, bits, g), ops.qvm(w, s, b, x, bits, g)
    torch.cuda.synchronize()
    assert torch.equal(got, again)
    q = torch.stack([(w >> (i * bits)) & (2 ** bits - 1) for i in range(32 // bits)], -1).reshape(k, n).double()
    want = mag = 0
    for r in range(0, k, 65536 // g * g):
        r1 = min(k, r + 65536 // g * g)
        xr, sr, br = x[:, r:r1].double(), s[r // g:r1 // g].double().repeat_interleave(g, 0), b[r // g:r1 // g].double().repeat_interleave(g, 0)
        want = want + xr @ (q[r:r1] * sr + br)
        mag = mag + xr.abs() @ (q[r:r1] * sr.abs() + br.abs())
    # 32-bit sums: a range of a warp (k / 16 rows where one CTA has all of them, 32 chunks at most), 16 warps and 32 chunks one after the other, each
    # addition half a unit in the last place of at most the sum of magnitudes; then one rounding to the type
    bound = (k / 16 + 64) * 2.0 ** -24 * mag + dict(bf16=2.0 ** -8, f16=2.0 ** -11, f32=2.0 ** -24)[dt] * want.abs()
    assert bool(((got.double() - want).abs() <= bound).all())
