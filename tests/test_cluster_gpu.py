"""The cluster kernel (csrc/qmv_cluster.cuh) against 64-bit sums, at the sizes where it can go wrong: one unit a row, rows past a tile, uneven
units over the CTAs of a cluster, several passes, every group form, windows of scales cut by the end of the matrix."""
import pytest

pytestmark = pytest.mark.gpu

EPS = {"bf16": 2.0 ** -8, "f16": 2.0 ** -11, "f32": 2.0 ** -24}


def _matrix(torch, n, k, bits, g, dt, gen):
    w = torch.randint(-2 ** 31, 2 ** 31, (n, k * bits // 32), dtype=torch.int32, device="cuda", generator=gen)
    s = (0.002 + 0.018 * torch.rand((n, k // g), device="cuda", generator=gen)) * (16.0 / 2 ** bits)
    b = -(2.0 ** (bits - 1)) * s + 1e-3 * torch.randn((n, k // g), device="cuda", generator=gen)
    return w, s.to(dt), b.to(dt)


def _codes(torch, w, bits):
    return torch.stack([(w >> (bits * i)) & ((1 << bits) - 1) for i in range(32 // bits)], dim=-1).reshape(w.shape[0], -1)


def _check(torch, got, mat, x, bits, g, dt):
    w, s, b = mat
    weights = _codes(torch, w, bits).double() * s.double().repeat_interleave(g, 1) + b.double().repeat_interleave(g, 1)
    ref, mag = x.double() @ weights.T, x.double().abs() @ (_codes(torch, w, bits).double() * s.double().repeat_interleave(g, 1)).T
    mag += x.double().abs() @ b.double().abs().repeat_interleave(g, 1).T
    # rounded to the output type once; sums of 32 bits: a group's chain of up to 16 truncated MMA steps, K / g groups, the warps' parts
    bound = EPS[dt] * ref.abs() + 2.0 ** -23 * (16 + s.shape[1] ** 0.5 + 16) * mag
    assert bool(((got.double() - ref).abs() <= bound).all()), float(((got.double() - ref).abs() / bound).max())


CASES = [
    # one unit of a row, rows that are no whole tile, both token tiles
    ((1,), 512, 5, 4, 64, "bf16"), ((17,), 512, 8, 4, 64, "f16"), ((15,), 256, 9, 4, 64, "bf16"), ((33,), 256, 16, 4, 32, "f32"),
    ((4099,), 128, 16, 8, 32, "f32"), ((4099,), 256, 7, 8, 32, "f32"),
    # units that do not divide over warps or ranks; several projections, one of them a single row
    ((1000, 520, 17), 1536, 7, 4, 64, "bf16"), ((96, 1, 300, 16), 2560, 13, 4, 128, "f16"), ((640, 128), 1536, 12, 4, 256, "bf16"),
    # long rows: the parts of K of two, four and eight CTAs
    ((200,), 8192, 8, 4, 64, "bf16"), ((600, 24), 14336, 8, 4, 64, "f16"), ((513,), 14336, 16, 4, 64, "bf16"), ((300,), 7168, 16, 4, 64, "f32"),
    # many tiles a CTA
    ((28672,), 4096, 16, 4, 64, "bf16"), ((40000,), 1024, 8, 4, 64, "f16"), ((9000,), 4096, 8, 4, 32, "f32"),
    # scales of a unit shorter than a window, down to one of two bytes, at the end of the matrix
    ((31,), 512, 8, 4, 512, "bf16"), ((47,), 1024, 11, 4, 512, "bf16"), ((18,), 512, 6, 4, 256, "f16"), ((5,), 1024, 6, 4, 128, "f32"),
    # eight bits: from the size on where it takes over
    ((4112,), 4096, 8, 8, 64, "bf16"), ((8200, 100), 2048, 16, 8, 128, "f16"), ((3400,), 4096, 9, 8, 256, "bf16"), ((100,), 1280, 5, 8, 64, "f32"),
    ((777,), 1024, 6, 8, 32, "bf16"), ((4100,), 4096, 5, 8, 512, "f16"),
]


@pytest.mark.parametrize("ns,k,m,bits,g,dt", CASES)
def test_products(ns, k, m, bits, g, dt):
    import torch
    from metaltile_b200 import ops

    gen = torch.Generator(device="cuda").manual_seed(k + m)
    td = dict(bf16=torch.bfloat16, f16=torch.float16, f32=torch.float32)[dt]
    mats = [_matrix(torch, n, k, bits, g, td, gen) for n in ns]
    x = torch.randn((m, k), device="cuda", generator=gen).to(td)
    ctx = ops.context()
    assert ctx.launch_of(m, list(ns), k, bits, g, dt)["kernel"] == "qmv_cluster"
    outs = [torch.full((m * n + 64,), 7.0, dtype=td, device="cuda") for n in ns]
    ctx.qmv_batched([dict(w=w.data_ptr(), scales=s.data_ptr(), biases=b.data_ptr(), x=x.data_ptr(), outs=[o.data_ptr()], M=m, N=n, K=k, bits=bits,
                          group_size=g, dtype=dt) for (w, s, b), o, n in zip(mats, outs, ns)], torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert ctx.status_word() == 0
    for mat, o, n in zip(mats, outs, ns):
        assert bool((o[m * n:] == 7.0).all())
        _check(torch, o[:m * n].reshape(m, n), mat, x, bits, g, dt)


# rows (or parts of rows) of fewer staged pieces than a CTA has warps, and so many tiles that the warps without a piece have two units and more:
# the whole ring of every warp is requested all the same
SHORT = [
    ((16384,), 512, 8, 8, 64, "f32"), ((12288,), 768, 8, 8, 64, "f32"), ((16384,), 896, 5, 8, 64, "f32"), ((50257,), 768, 8, 4, 64, "f32"),
    ((16384,), 384, 16, 8, 64, "f32"), ((50257,), 512, 5, 4, 64, "bf16"), ((40000,), 256, 16, 4, 64, "bf16"), ((40001,), 256, 6, 4, 32, "bf16"),
    ((32000,), 768, 8, 8, 64, "bf16"), ((33000,), 512, 7, 8, 64, "f16"), ((30000, 9000, 1000), 512, 6, 4, 64, "f16"),
    ((2576,), 3072, 8, 8, 64, "f32"), ((2000, 576), 3072, 6, 8, 128, "f32"),                                       # K split over four CTAs
]


# tiles of a cluster whose partial sums do not fit at once: two, three and four passes over them
PASSES = [
    ((988,), 13824, 11, 4, 256, "bf16"), ((1001, 24), 13568, 14, 4, 128, "f16"), ((262,), 9472, 12, 8, 256, "f32"), ((514,), 9472, 13, 8, 64, "f32"),
    ((742,), 10240, 10, 8, 128, "f32"), ((16937,), 11520, 9, 4, 64, "bf16"),
]


@pytest.mark.parametrize("ns,k,m,bits,g,dt", SHORT + PASSES)
def test_short_rows_and_passes(ns, k, m, bits, g, dt):
    test_products(ns, k, m, bits, g, dt)


@pytest.mark.parametrize("bits,dt", [(4, "bf16"), (4, "f16"), (4, "f32"), (8, "f32")])
def test_infinity_and_nan_stay_in_their_token_and_row(bits, dt):
    import torch
    from metaltile_b200 import ops

    gen = torch.Generator(device="cuda").manual_seed(3)
    td = dict(bf16=torch.bfloat16, f16=torch.float16, f32=torch.float32)[dt]
    w, s, b = _matrix(torch, 100, 2048, bits, 64, td, gen)
    w |= 0x11111111 if bits == 4 else 0x01010101                  # no code is zero: 0 * inf would be NaN
    b = b.abs()
    x = torch.randn((11, 2048), device="cuda", generator=gen).to(td)
    clean = ops.qmv(w, s, b, x, bits, 64)
    x[3, 1000], x[9, 17] = float("inf"), float("nan")
    s[50, 7] = float("inf")
    got = ops.qmv(w, s, b, x, bits, 64)
    rows, toks = [n for n in range(100) if n != 50], [t for t in range(11) if t not in (3, 9)]
    assert bool((got[3][rows] == float("inf")).all()) and bool(got[9].isnan().all())
    assert not bool(got[toks, 50].isfinite().any())
    assert torch.equal(got[toks][:, rows], clean[toks][:, rows])


def test_a_call_repeats_itself_and_follows_the_stream():
    """Captured and replayed with the activations rewritten in between: the sums are added in a fixed order."""
    import torch
    from metaltile_b200 import ops

    gen = torch.Generator(device="cuda").manual_seed(4)
    mat = _matrix(torch, 3000, 14336, 4, 64, torch.bfloat16, gen)
    x = torch.randn((8, 14336), device="cuda", generator=gen).to(torch.bfloat16)
    y = torch.randn((8, 14336), device="cuda", generator=gen).to(torch.bfloat16)
    want = [ops.qmv(*mat, v, 4, 64) for v in (x, y)]
    buf = x.clone()
    ops.qmv(*mat, buf, 4, 64)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = ops.qmv(*mat, buf, 4, 64)
    for _ in range(3):
        for v, ref in zip((x, y), want):
            buf.copy_(v)
            graph.replay()
            assert torch.equal(out, ref)
