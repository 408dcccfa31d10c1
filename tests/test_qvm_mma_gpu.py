"""The tensor-core form of the vector-matrix product (several tokens, or 2-bit codes) against the oracle: column counts that
end inside a tile and inside a lane quad, ranges of K that do not fill the last batch, groups of one, three and four slabs
of 32 rows, every token count at which the split of the MMA columns changes, one tile whose K is spread over 32 CTAs."""
import numpy as np
import pytest

import oracle
from helpers import ODT, rel_err, to_dev

pytestmark = pytest.mark.gpu

# rounding to a significand of p bits (2^-p of the value: bf16 8, f16 11) and the f32 sums on both sides (below 2^-14 at these lengths)
BOUND = {"bf16": 2.0 ** -8 + 2.0 ** -14, "f16": 2.0 ** -11 + 2.0 ** -14}


@pytest.mark.parametrize("n,k,bits,gs,dt", [
    (1056, 7968, 4, 96, "bf16"), (2080, 4096, 4, 128, "f16"), (1024, 8224, 4, 32, "bf16"), (4128, 2112, 4, 64, "bf16"),
    (1040, 4064, 8, 32, "f16"), (1024, 4096, 8, 256, "bf16"), (544, 1952, 2, 32, "bf16"), (32, 33024, 2, 128, "f16"),
])
def test_against_the_oracle(n, k, bits, gs, dt):
    import torch
    from metaltile_b200 import ops, synth
    rng = np.random.default_rng(n + bits)
    w = synth.words(k * n * bits // 32, seed=n).reshape(k, -1)
    sc = oracle.round_through(((0.002 + 0.018 * rng.random((k // gs, n))) * 16 / 2 ** bits).astype(np.float32), ODT[dt])
    bi = oracle.round_through((-(2.0 ** (bits - 1)) * sc).astype(np.float32), ODT[dt])
    wd, sd, bd = to_dev(w), to_dev(sc, dt), to_dev(bi, dt)
    for m in (1, 2, 3, 4, 5):
        x = oracle.round_through(synth.activations(m, k, seed=m), ODT[dt])
        xd = to_dev(x, dt)
        got, again = ops.qvm(wd, sd, bd, xd, bits, gs), ops.qvm(wd, sd, bd, xd, bits, gs)
        torch.cuda.synchronize()
        assert torch.equal(got, again)                          # the chunks of K are added in a fixed order
        assert rel_err(got.float().cpu().numpy(), oracle.qvm(w, sc, bi, x, m, n, k, bits, gs)) <= BOUND[dt]
