"""What a product launches (mtc_launch_of: the functions the entries go by; without a context the default options and 148 SMs, no GPU needed):
the kernel's name and form on both sides of the rules, and that the GPU tests of a kernel name shapes that it takes."""
import random

import pytest

from metaltile_b200 import MetalTileError, _lib
from metaltile_b200.context import _dt, launch_of
from test_cluster_gpu import CASES, PASSES, SHORT
from test_qmm_cluster_gpu import CASES as SLICED

WARPS = 16


@pytest.mark.parametrize("args,want", [
    ((1, [4096], 4096, 4, 64, "bf16"), "qmv_frag"), ((4, [4096], 4096, 4, 64, "bf16"), "qmv_frag"), ((5, [4096], 4096, 4, 64, "bf16"), "qmv_cluster"),
    ((16, [4096], 4096, 4, 256, "f16"), "qmv_cluster"), ((8, [2880], 2880, 4, 64, "bf16"), "qmv_frag"), ((8, [4096], 4096, 4, 32, "bf16"), "qmv_cluster"),
    ((2, [4096], 4096, 4, 256, "bf16"), "qmv_cluster"), ((4, [4096], 4096, 8, 64, "f32"), "qmv_cuda_core"), ((5, [4096], 4096, 8, 64, "f32"), "qmv_cluster"),
    ((5, [4096], 4096, 3, 64, "f32"), "qmv_frag"), ((8, [4096], 4096, 8, 64, "bf16"), "qmv_cluster"), ((8, [4095], 4096, 8, 64, "bf16"), "qmv_frag"),
    ((9, [3072], 4096, 8, 64, "bf16"), "qmv_cluster"), ((9, [3071], 4096, 8, 64, "bf16"), "qmv_frag"), ((16, [8192], 8192, 8, 64, "bf16"), "qmm_tcgen05"),
    ((16, [4096], 4096, 4, 32, "bf16"), "qmm_tcgen05"), ((20, [4096], 4096, 4, 64, "bf16"), "qmv_cluster"), ((2048, [4096], 4096, 4, 64, "bf16"), "qmm_tcgen05"),
    # from nine tokens on, K an odd multiple of 256, a tile a CTA
    ((9, [2368], 2304, 4, 64, "bf16"), "qmv_frag"), ((9, [2369], 2304, 4, 64, "bf16"), "qmv_cluster"), ((16, [865], 1792, 4, 256, "f16"), "qmv_cluster"),
    ((16, [865], 1280, 4, 64, "f16"), "qmv_cluster"), ((16, [865], 3840, 4, 64, "bf16"), "qmv_frag"), ((16, [865], 4352, 4, 64, "bf16"), "qmv_cluster"),
    ((8, [865], 2816, 4, 64, "bf16"), "qmv_frag"), ((16, [865], 2816, 4, 64, "f32"), "qmv_cluster"), ((9, [1000, 400], 2304, 4, 64, "bf16"), "qmv_frag"),
    # projections that share x: one launch, or "" where they run one by one
    ((1, [4096, 1024, 1024], 4096, 4, 64, "bf16"), "qmv_frag"), ((8, [4096, 1024, 1024], 4096, 4, 64, "bf16"), "qmv_cluster"),
    ((16, [14336, 14336], 4096, 8, 64, "bf16"), "qmv_cluster"), ((16, [4096, 4096], 4096, 8, 32, "bf16"), ""), ((2, [64, 64], 480, 4, 24, "bf16"), ""),
    ((0, [64], 64, 4, 64, "bf16"), ""), ((1, [64], 64, 4, 0, "bf16"), ""), ((1, [64, 0], 64, 4, 64, "bf16"), ""),
])
def test_names(args, want):
    assert launch_of(*args)["kernel"] == want


def test_forms():
    assert launch_of(8, [4096], 14336, 4, 64, "bf16") == dict(kernel="qmv_cluster", ctas=132, cluster=4, k_slices=4, passes=1)
    assert launch_of(2048, [4096], 4096, 4, 64, "bf16") == dict(kernel="qmm_tcgen05", ctas=144, cluster=1, k_slices=1, passes=0)
    for m, n, k, bits, g, dt in SLICED:
        form = launch_of(m, [n], k, bits, g, dt)
        assert form["kernel"] == "qmm_tcgen05" and form["cluster"] == form["k_slices"] >= 2 and form["ctas"] % form["cluster"] == 0
    # K slices: in clusters where that was measured to be faster than whole items, or than slices that add up through memory (us, this form against the next:
    # 202 x 5760 x 6208 29.1, in three slices through memory 30.8; 699 x 832 x 3072 16.9, six through memory 18.3; 186 x 4096 x 1024 as four items 9.7, in
    # clusters of four 12.5; 333 x 7616 x 2880 as two items 22.2, in pairs 23.6; 800 x 4352 x 3904 as four items 26.0, in pairs 30.2)
    for args, slices, cluster in (((364, [6144], 2560, 8, 128, "bf16"), 1, 1), ((800, [4352], 3904, 4, 32, "f16"), 1, 1), ((202, [5760], 6208, 8, 32, "bf16"), 2, 2),
                                  ((212, [5376], 5120, 4, 64, "f16"), 3, 3), ((699, [832], 3072, 4, 128, "bf16"), 4, 4), ((186, [4096], 1024, 4, 64, "bf16"), 1, 1),
                                  ((333, [7616], 2880, 8, 32, "f16"), 1, 1)):
        form = launch_of(*args)
        assert (form["k_slices"], form["cluster"]) == (slices, cluster), args
    with pytest.raises(MetalTileError):
        launch_of(1, [64] * 5, 64, 4, 64, "bf16")


@pytest.mark.parametrize("bits,group,most", [(8, 64, 512), (6, 128, 512), (8, 32, 256), (4, 32, 384), (3, 32, 384)])
def test_rows_an_expert_of_the_grouped_fragment_kernel(bits, group, most):
    route = lambda m, n, k, e: _lib.load().mtc_gather_qmm_route(m, n, k, e, bits, group, _dt("bf16")).decode()  # noqa: E731
    assert [route(m, 768, 2048, 128) for m in (most, most + 1)] == ["gather_qmm_frag", "gather_qmm_tcgen05"]
    assert [route(m, 768, 1024, 32) for m in (320, 321)] == ["gather_qmm_frag", "gather_qmm_tcgen05"]      # up to 32 Mi codes


def _walk(ns, k, m, bits, g, dt):
    """The units of each warp of the first and the last cluster, and the staged pieces of its CTA: the arithmetic of qmv_cluster.cuh."""
    form = launch_of(m, list(ns), k, bits, g, dt)
    assert form["kernel"] == "qmv_cluster"
    unit = (1 if dt == "f32" or m > 8 or g == 32 else 2) * 1024 // bits
    units, cs, tiles = k // unit, form["cluster"], sum((n + 15) // 16 for n in ns)
    clusters, pieces = form["ctas"] // cs, unit // (32 if g == 32 else 64) * (1 if m <= 8 else 2)
    for cid in (0, clusters - 1):
        mine = tiles // clusters + (cid < tiles % clusters)
        for rank in range(cs):
            nu = (rank + 1) * units // cs - rank * units // cs
            assert nu >= 1
            totals = [(mine * (i + 1) // form["passes"] - mine * i // form["passes"]) * nu for i in range(form["passes"])]
            share = [[t * w // WARPS if t >= WARPS else min(w, t) for w in range(WARPS + 1)] for t in totals]
            held = [sum(s[w + 1] - s[w] for s in share) for w in range(WARPS)]
            assert sum(held) == sum(totals)
            yield held, nu * pieces


@pytest.mark.parametrize("case", SHORT)
def test_short_rows_leave_warps_without_a_piece_but_with_units(case):
    assert any(held[w] >= 2 for held, pieces in _walk(*case) for w in range(pieces, WARPS))


@pytest.mark.parametrize("case", PASSES)
def test_passes(case):
    ns, k, m, bits, g, dt = case
    assert launch_of(m, list(ns), k, bits, g, dt)["passes"] >= 2


def test_every_unit_has_a_warp():
    rng, seen = random.Random(1), 0
    for case in CASES + SHORT + PASSES:
        list(_walk(*case))
    while seen < 2000:
        m, bits, g, dt = rng.randint(2, 16), rng.choice((4, 8)), rng.choice((32, 64, 128, 256, 512)), rng.choice(("bf16", "f16", "f32"))
        ns = [int(2 ** rng.uniform(0, 16)) + 1 for _ in range(rng.choice((1, 1, 2, 3, 4)))]
        k = rng.choice((128, 256, 512)) * rng.randint(1, 40)
        if k % g == 0 and launch_of(m, ns, k, bits, g, dt)["kernel"] == "qmv_cluster":
            list(_walk(ns, k, m, bits, g, dt))
            seen += 1
