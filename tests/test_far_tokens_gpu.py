"""Activations outside the range of products with codes in place (csrc/far_tokens.cuh): tokens of very large and very small values, zeros and
infinities beside ordinary ones, against 64-bit sums, on the kernels that took over from ones without those limits."""
import pytest

from test_cluster_gpu import EPS, _matrix
from test_gather_frag_gpu import _codes, _offsets, _stack

pytestmark = pytest.mark.gpu

TYPES = {"bf16": "bfloat16", "f16": "float16", "f32": "float32"}


def _far(torch, x, dt):
    """Rows in turn: as they are, times 2^70, 2^-90, zero, one value of 2^66, an infinity, times 2^32, 2^-66 (f16: as they are, zero, an infinity)."""
    kinds = ("usual", "zero", "inf") if dt == "f16" else ("usual", 70, -90, "zero", "one", "inf", 32, -66)
    for i in range(x.shape[0]):
        kind = kinds[i % len(kinds)]
        if isinstance(kind, int):
            x[i] *= 2.0 ** kind
        elif kind == "zero":
            x[i] = 0.0
        elif kind != "usual":
            x[i, x.shape[1] - 1 - i] = 2.0 ** 66 if kind == "one" else float("inf")
    return [i for i in range(x.shape[0]) if kinds[i % len(kinds)] == "usual"]


def _check(torch, got, x, q, b, groups, dt):
    ref, mag = x.double() @ (q + b).T, x.double().abs() @ (q.abs() + b.abs()).T
    fin = ref.isfinite()
    assert torch.equal(got[~fin].double().nan_to_num(nan=7.0), ref[~fin].nan_to_num(nan=7.0))      # infinities of the same sign; 0 * inf is NaN
    # rounded to the output type once; 32-bit sums in chains of at most 32 and K / 32 of them
    bound = EPS[dt] * ref.abs() + 2.0 ** -23 * (24 + groups ** 0.5) * mag
    assert bool(((got.double() - ref).abs() <= bound)[fin].all())


@pytest.mark.parametrize("n,k,m,bits,g,dt", [
    (100, 2048, 8, 4, 64, "bf16"), (601, 14336, 7, 4, 64, "bf16"), (3999, 2816, 12, 4, 256, "bf16"), (9000, 4096, 16, 4, 128, "bf16"), (777, 1024, 6, 8, 32, "bf16"),
    (300, 7168, 16, 4, 64, "f32"), (100, 1280, 7, 8, 64, "f32"), (2100, 5888, 16, 4, 64, "bf16"), (100, 1024, 6, 4, 512, "bf16")])
def test_cluster_kernel(n, k, m, bits, g, dt):
    import torch
    from metaltile_b200 import ops

    gen = torch.Generator(device="cuda").manual_seed(n)
    td = getattr(torch, TYPES[dt])
    w, s, b = _matrix(torch, n, k, bits, g, td, gen)
    assert ops.context().launch_of(m, [n], k, bits, g, dt)["kernel"] == "qmv_cluster"
    x = torch.randn((m, k), device="cuda", generator=gen).to(td)
    clean = ops.qmv(w, s, b, x, bits, g)
    usual = _far(torch, x, dt)
    got = ops.qmv(w, s, b, x, bits, g)
    torch.cuda.synchronize()
    assert ops.context().status_word() == 0
    assert torch.equal(got[usual], clean[usual])
    q = _codes(torch, w, bits, k).double() * s.double().repeat_interleave(g, 1)
    _check(torch, got, x, q, b.double().repeat_interleave(g, 1), k // 32, dt)


@pytest.mark.parametrize("counts", [[1, 0, 1, 1] + [0] * 9, [3, 0, 1, 5], [7, 8, 9, 12, 1]])
@pytest.mark.parametrize("bits,g,dt", [(4, 64, "bf16"), (8, 128, "bf16"), (3, 64, "bf16"), (6, 32, "bf16"), (2, 32, "bf16"), (5, 64, "f16"), (8, 64, "f16")])
def test_grouped_kernel(bits, g, dt, counts):
    import torch
    from metaltile_b200 import ops

    gen = torch.Generator(device="cuda").manual_seed(bits)
    td, e, m, n, k = getattr(torch, TYPES[dt]), len(counts), sum(counts), 130, 640
    ctx = ops.context()
    assert ctx.gather_qmm_route(m, n, k, e, bits, g, dt) == "gather_qmm_frag"
    w, s, b = _stack(torch, e, n, k, bits, g, td, gen)
    x = torch.randn((m, k), device="cuda", generator=gen).to(td)
    off = _offsets(torch, counts)
    clean = ops.gather_qmm(x, w, s, b, bits, g, expert_offsets=off)
    usual = _far(torch, x, dt)
    got = ops.gather_qmm(x, w, s, b, bits, g, expert_offsets=off)
    torch.cuda.synchronize()
    assert ctx.status_word() == 0 and torch.equal(got[usual], clean[usual])
    row = 0
    for i, c in enumerate(counts):
        if c:
            q = _codes(torch, w[i], bits, k).double() * s[i].double().repeat_interleave(g, 1)
            _check(torch, got[row:row + c], x[row:row + c], q, b[i].double().repeat_interleave(g, 1), k // 32, dt)
        row += c
