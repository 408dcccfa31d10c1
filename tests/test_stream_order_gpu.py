"""Calls issued back to back give what the same calls give with the GPU waited for between them.

The kernels of the library are launched while the kernel before them drains and wait on the device for what it writes.  Here a
consumer follows its producer at once, over buffers that are rewritten with other values every time, so that a value read
before it is written is one of the round before."""
import numpy as np
import pytest

from helpers import dense_case, to_dev

pytestmark = pytest.mark.gpu
ROUNDS = 40


@pytest.fixture(scope="module")
def ctx():
    from metaltile_b200 import ops
    return ops.context(0)


def _same_without_waiting(step, rounds=ROUNDS):
    """``step(i)`` enqueues round i and returns its results: all rounds at once against one at a time."""
    import torch
    want = []
    for i in range(rounds):
        want.append([t.clone() for t in step(i)])
        torch.cuda.synchronize()
    got = [[t.clone() for t in step(i)] for i in range(rounds)]
    torch.cuda.synchronize()
    for i in range(rounds):
        for a, b in zip(got[i], want[i]):
            assert torch.equal(a, b), i


@pytest.mark.parametrize("by_rows", [False, True])
@pytest.mark.parametrize("dt", ["f16", "bf16"])
def test_work_list_of_a_grouped_product(ctx, dt, by_rows):
    """The list of work items and its length are written by the kernel in front of the product (bf16: with the row conversion in
    between): offsets that name 4 rows and 900 in turn."""
    import torch
    from metaltile_b200 import ops
    e, n, k, rows = 8, 256, 512, 900
    w, s, b, x = dense_case(rows, e * n, k, 8, 64, dt, seed=41)
    wd, sd, bd, xd = to_dev(w).view(e, n, -1), to_dev(s, dt).view(e, n, -1), to_dev(b, dt).view(e, n, -1), to_dev(x, dt)
    rng = np.random.default_rng(3)
    lists = []
    for i in range(ROUNDS):
        m = 4 if i % 2 else rows
        owner = np.sort(rng.integers(0, e, size=m))
        off = np.searchsorted(owner, np.arange(e + 1)).astype(np.uint32)
        lists.append((m, to_dev(owner.astype(np.uint32)), to_dev(off)))
    torch.cuda.synchronize()

    def step(i):
        m, owner, off = lists[i]
        kw = dict(indices=owner) if by_rows else dict(expert_offsets=off)
        return [ops.gather_qmm(xd[:m], wd, sd, bd, 8, 64, ctx=ctx, **kw)]

    _same_without_waiting(step)
    assert ctx.status_word() == 0
