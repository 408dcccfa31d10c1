"""The vector-matrix product of one token whose codes pass through shared memory, against the float64 product of the dequantised weights: column
counts that end inside a tile and inside a copy's row of lanes, chunks and ranges of K that end inside a group, groups of one unit and longer than a
warp's range, one column tile whose K is spread over 32 CTAs, the first sizes on both sides of the rule."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k,bits,g,dt", [
    (2080, 2064, 4, 16, "bf16"), (1056, 4128, 4, 48, "f32"), (4128, 1024, 4, 1024, "f16"), (32, 131104, 4, 32, "bf16"), (1024, 4096, 4, 64, "f32"),
    (1024, 4080, 4, 16, "f32"), (528, 24000, 8, 64, "f32"), (2064, 6144, 8, 128, "bf16"), (32, 393216, 8, 32, "f16"), (19024, 672, 8, 16, "f16"),
    (37920, 128, 4, 64, "bf16"), (1028, 16384, 8, 64, "f32"),
])
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
