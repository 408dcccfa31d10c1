"""The expert sort on both sides of its rules: rows stored directly and through shared memory, experts told apart by matches and by votes, walks of one
warp, of held ids and of more than those.  Integers: equal to a stable sort."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_tokens,k", [(32, 8), (33, 8), (341, 3), (512, 8), (513, 8), (1536, 8), (1537, 8)])
@pytest.mark.parametrize("n_experts", [1, 16, 17, 64, 1024])
def test_equal_to_a_stable_sort(n_tokens, k, n_experts):
    import torch
    from metaltile_b200 import ops

    rng = np.random.default_rng(n_tokens + n_experts)
    idx = (rng.integers(0, n_experts, (n_tokens, k)) ** 2 // max(n_experts - 1, 1)).astype(np.int32)      # a biased router; the last expert too
    sti, inv, off, row = ops.moe_sort(torch.from_numpy(idx).cuda(), n_experts)
    torch.cuda.synchronize()
    flat = idx.reshape(-1)
    order = np.argsort(flat, kind="stable")
    assert np.array_equal(sti.cpu().numpy(), order // k)
    assert np.array_equal(row.cpu().numpy(), flat[order])
    assert np.array_equal(inv.cpu().numpy().reshape(-1)[order], np.arange(flat.size))
    assert np.array_equal(off.cpu().numpy(), np.concatenate([[0], np.cumsum(np.bincount(flat, minlength=n_experts))]))
