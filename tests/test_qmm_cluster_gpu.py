"""K slices of the tensor-memory product that add up inside a cluster, against the same product without slices: the same f16 weights, 32-bit
sums in another order, one rounding each."""
import pytest

pytestmark = pytest.mark.gpu

CASES = [
    (256, 4096, 4096, 4, 64, "bf16"), (250, 4001, 4096, 4, 64, "f16"),       # four CTAs; rows that are no multiple of a tile, outputs that do not pair
    (558, 1152, 2752, 4, 64, "f16"),                                         # K of 43 blocks: slices of different length
    (512, 4096, 4096, 4, 128, "bf16"), (1024, 1000, 4096, 4, 64, "bf16"),    # two and more token chunks a tile
    (300, 6400, 5760, 8, 32, "f16"), (285, 6400, 3072, 2, 128, "bf16"),      # pairs of two-chunk items
]


@pytest.mark.parametrize("m,n,k,bits,g,dt", CASES)
def test_cluster_slices_equal_the_unsliced_product(m, n, k, bits, g, dt):
    import torch
    from metaltile_b200 import Context, ops

    gen = torch.Generator(device="cuda").manual_seed(m)
    td = dict(bf16=torch.bfloat16, f16=torch.float16)[dt]
    w = torch.randint(-2 ** 31, 2 ** 31, (n, k * bits // 32), dtype=torch.int32, device="cuda", generator=gen)
    s = ((0.002 + 0.018 * torch.rand((n, k // g), device="cuda", generator=gen)) * (16.0 / 2 ** bits)).to(td)
    b = (-(2.0 ** (bits - 1)) * s.float()).to(td)
    x = torch.randn((m, k), device="cuda", generator=gen).to(td)
    ctx = Context(0)
    form = ctx.launch_of(m, [n], k, bits, g, dt)
    assert form["kernel"] == "qmm_tcgen05" and form["cluster"] == form["k_slices"] >= 2
    got = torch.full((m + 1, n), 7.0, dtype=td, device="cuda")
    ops.qmm(w, s, b, x, bits, g, out=got[:m], ctx=ctx)
    again = ops.qmm(w, s, b, x, bits, g, ctx=ctx)
    ctx.set_option("qmm_ksplit", 0)
    assert ctx.launch_of(m, [n], k, bits, g, dt)["k_slices"] == 1
    whole = ops.qmm(w, s, b, x, bits, g, ctx=ctx)
    torch.cuda.synchronize()
    assert ctx.status_word() == 0
    assert bool((got[m] == 7.0).all()) and torch.equal(got[:m], again)
    # both rounded to the output type once: where the sums straddle a boundary they land a unit in the last place apart, 2^-7 (2^-10) of the value
    # at most; the sums themselves have terms of at most 2^(bits - 1) * max scale * |x| and differ by their order in 32 bits
    unit = 2.0 ** -7 if dt == "bf16" else 2.0 ** -10
    mag = x.float().abs().sum(1, keepdim=True) * (2.0 ** (bits - 1)) * float(s.float().max())
    bound = unit * whole.float().abs() + 2.0 ** -23 * 16 * mag
    assert bool(((got[:m].float() - whole.float()).abs() <= bound).all())
