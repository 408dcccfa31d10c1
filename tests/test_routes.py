"""Which kernel a product runs on, at both sides of every line of the rules (mtc_qmm_kernel: the function mtc_qmm and mtc_qmv decide by;
without a context: the default options, no GPU needed), and which kernel family the selector names without the fragment kernel."""
import pytest

from metaltile_b200 import _lib
from metaltile_b200.context import _dt

FRAG, RING, TC, CUDA = "qmv_frag", "qmv_mma_sync", "qmm_tcgen05", "qmv_cuda_core"


def kernel(m, n, k, bits, group, dt):
    return _lib.load().mtc_qmm_kernel(None, m, n, k, bits, group, _dt(dt)).decode()


@pytest.mark.parametrize("args,want", [
    # one token: 4 and 8 bits at any size, 2 / 3 / 6 up to 64 Mi codes, 5 never, f32 never
    ((1, 4096, 4096, 4, 64, "bf16"), FRAG), ((1, 16384, 16384, 4, 64, "f16"), FRAG), ((1, 64, 512, 8, 32, "bf16"), FRAG),
    ((1, 8192, 8192, 3, 64, "bf16"), FRAG), ((1, 8224, 8192, 3, 64, "bf16"), CUDA), ((1, 16384, 16384, 2, 64, "f16"), CUDA),
    ((1, 4096, 4096, 6, 128, "f16"), FRAG), ((1, 4096, 4096, 5, 64, "bf16"), CUDA), ((1, 4096, 4096, 4, 64, "f32"), CUDA),
    # 4 bits, K % 512 == 0: up to four tokens, groups of 64 and 128
    ((2, 4096, 4096, 4, 64, "bf16"), FRAG), ((4, 4096, 4096, 4, 128, "bf16"), FRAG), ((5, 4096, 4096, 4, 64, "bf16"), RING),
    ((16, 4096, 4096, 4, 64, "bf16"), RING), ((2, 4096, 4096, 4, 256, "bf16"), RING),
    # ... and where that kernel does not go: K % 512, groups of 32
    ((8, 2880, 2880, 4, 64, "bf16"), FRAG), ((8, 4096, 4096, 4, 32, "bf16"), FRAG), ((16, 4096, 4096, 4, 32, "bf16"), TC),
    ((16, 2880, 2880, 4, 64, "bf16"), FRAG), ((16, 2880, 2880, 4, 32, "bf16"), TC),
    # other widths: up to four tokens always; to eight while K <= 8192 or below 32 Mi codes; from nine on groups of 64 and more with K <= 5120 up
    # to 20 Mi codes
    ((4, 16384, 16384, 8, 64, "bf16"), FRAG), ((4, 4096, 4096, 5, 32, "f16"), FRAG), ((8, 16384, 8192, 8, 64, "bf16"), FRAG),
    ((8, 4096, 8256, 8, 64, "bf16"), TC), ((8, 4032, 8256, 8, 64, "bf16"), FRAG), ((9, 4096, 5120, 8, 64, "bf16"), FRAG), ((9, 4112, 5120, 8, 64, "bf16"), TC),
    ((9, 4096, 5184, 8, 64, "bf16"), TC), ((9, 4096, 4096, 8, 32, "bf16"), TC), ((16, 512, 512, 8, 64, "bf16"), FRAG),
    ((16, 512, 512, 8, 32, "bf16"), CUDA),
    # f32 activations: three pieces a value, from five tokens on
    ((4, 4096, 4096, 8, 64, "f32"), CUDA), ((5, 4096, 4096, 8, 64, "f32"), FRAG), ((16, 4096, 4096, 4, 32, "f32"), FRAG),
    # outside the fragment kernel's shapes
    ((1, 64, 96, 4, 48, "bf16"), CUDA), ((2, 64, 480, 4, 24, "bf16"), CUDA), ((2, 64, 48, 8, 16, "bf16"), CUDA),
    # more than 16 tokens
    ((17, 4096, 4096, 4, 64, "bf16"), RING), ((32, 4096, 4096, 4, 64, "bf16"), RING), ((33, 4096, 4096, 4, 64, "bf16"), TC),
    ((17, 4096, 4096, 8, 64, "bf16"), TC), ((2048, 14336, 4096, 4, 64, "f32"), CUDA), ((64, 256, 96, 4, 32, "bf16"), CUDA),
    # nothing takes these
    ((0, 64, 64, 4, 64, "bf16"), ""), ((1, 64, 64, 4, 0, "bf16"), ""),
])
def test_kernel_of_a_product(args, want):
    assert kernel(*args) == want


@pytest.mark.gpu
def test_options_change_the_kernel():
    from metaltile_b200 import Context
    ctx = Context(0)
    shape = (1, 4096, 4096, 4, 64, "bf16")
    assert ctx.qmm_kernel(*shape) == kernel(*shape) == FRAG
    ctx.set_option("qmv_frag", 0)
    assert ctx.qmm_kernel(*shape) == ctx.qmm_route(*shape) == "qmv_stream"
    for args in ((8, 4096, 4096, 4, 64, "bf16"), (1, 4096, 4096, 3, 64, "bf16"), (16, 4096, 4096, 8, 64, "bf16"), (1, 1024, 1024, 4, 64, "f16"),
                 (8, 4096, 4096, 8, 64, "f32"), (20, 4096, 4096, 4, 64, "bf16"), (300, 4096, 4096, 3, 64, "f16")):
        assert ctx.qmm_kernel(*args) == ctx.qmm_route(*args)
    ctx.set_option("qmv_stream", 0)
    assert ctx.qmm_kernel(*shape) == CUDA
    ctx.set_option("qmv_tc", 1)
    assert ctx.qmm_kernel(*shape) == "qmv_tcgen05_decode"
    ctx.set_option("qmv_tc", 0)
    ctx.set_option("qmv_frag", 2)
    assert ctx.qmm_kernel(16, 8192, 8192, 3, 32, "bf16") == FRAG
