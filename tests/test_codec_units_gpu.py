"""The codec kernels that give a lane 8 consecutive values, four times: every group size that a warp reduces in its own
way (4 to 32 lanes of a unit, two and four units), a tail that ends inside a warp's 1024 values, and a group size that
is not a power of two.  Codes, scales, biases and values are compared for equality."""
import numpy as np
import pytest

import oracle
from helpers import ODT, to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", ["f32", "f16", "bf16"])
@pytest.mark.parametrize("bits", [2, 3, 4, 5, 6, 8])
@pytest.mark.parametrize("gs", [32, 64, 96, 128, 256, 512, 1024])
def test_codec_is_exact(bits, gs, dt):
    import torch
    from metaltile_b200 import ops
    rng = np.random.default_rng(gs * 10 + bits)
    n = 1024 // gs * 3 + 1 if gs <= 512 else 3            # groups: one row each, total not a multiple of 1024 values
    wf = rng.standard_normal((n, gs)) * np.exp2(rng.integers(-12, 8, size=(n, 1)))
    wf[0] = 0.25                                          # a constant group: the scale is 1
    if n > 1:
        wf[1, :] = np.linspace(-1.0, 1.0, gs)             # values that fall on code boundaries
    wf = oracle.round_through(wf.astype(np.float32), ODT[dt])
    q, s, b = ops.affine_quantize(to_dev(wf, dt), bits, gs)
    back = ops.affine_dequantize(q, s, b, bits, gs)
    torch.cuda.synchronize()
    oq, osc, obi = oracle.affine_quantize(wf, bits, gs)
    assert np.array_equal(q.cpu().numpy().view(np.uint32).reshape(-1), oq)
    s_h, b_h = s.float().cpu().numpy().reshape(-1), b.float().cpu().numpy().reshape(-1)
    assert np.array_equal(s_h, oracle.round_through(osc, ODT[dt]))
    assert np.array_equal(b_h, oracle.round_through(obi, ODT[dt]))
    ref = oracle.round_through(oracle.affine_dequantize(oq, s_h, b_h, n * gs, bits, gs), ODT[dt])
    assert np.array_equal(back.float().cpu().numpy().reshape(-1), ref)


def _awkward_groups(gs, dt):
    """Groups of values that are not ordinary numbers: all NaN, partly NaN, both infinities, one of them, nothing but one
    infinity, a span past the largest f32 (or the type's largest values), and one whose 1 / scale is subnormal."""
    big = {"f32": 3.4e38, "f16": 65504.0, "bf16": 3.38e38}[dt]
    g = np.random.default_rng(gs).standard_normal((9, gs)).astype(np.float32)
    g[0, :] = np.nan
    g[1, ::3] = np.nan
    g[2, 0], g[2, gs - 1] = np.inf, -np.inf
    g[3, 5] = np.inf
    g[4, 7] = -np.inf
    g[5, :] = np.inf
    g[6, 0], g[6, 1] = big, -big
    g[7, :] = 0.0
    g[7, 2] = big                                         # 2- and 3-bit f32: the scale is above 2^126
    g[8, :gs - 1] = np.nan                                # one number among NaN: the scale is 1
    return oracle.round_through(g, ODT[dt])


@pytest.mark.parametrize("dt", ["f32", "f16", "bf16"])
@pytest.mark.parametrize("bits", [2, 3, 4, 8])
@pytest.mark.parametrize("gs,shift", [(32, 0), (64, 0), (256, 0), (512, 0), (1024, 0), (64, 1), (96, 0)])
def test_values_that_are_not_numbers(gs, shift, bits, dt):
    """The same codes, scales and biases as the scalar formula whatever kernel runs: the vector form (whole warps of units), the
    warp-per-group form (``shift``: an input that is not 16-byte aligned; 96: no power of two)."""
    import torch
    from metaltile_b200 import ops
    wf = _awkward_groups(gs, dt)
    src = to_dev(wf, dt)
    room = torch.empty(src.numel() + 8, dtype=src.dtype, device="cuda")
    src = room[shift:shift + src.numel()].view(src.shape).copy_(src)
    q, s, b = ops.affine_quantize(src, bits, gs)
    torch.cuda.synchronize()
    with np.errstate(all="ignore"):
        oq, osc, obi = oracle.affine_quantize(wf, bits, gs)
        osc, obi = oracle.round_through(osc, ODT[dt]), oracle.round_through(obi, ODT[dt])
    assert np.array_equal(s.float().cpu().numpy().reshape(-1), osc, equal_nan=True)
    assert np.array_equal(b.float().cpu().numpy().reshape(-1), obi, equal_nan=True)
    assert np.array_equal(q.cpu().numpy().view(np.uint32).reshape(-1), oq)
