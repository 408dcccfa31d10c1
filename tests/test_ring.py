"""The barrier protocol of the tcgen05 kernels' rings, played on the CPU: the rules of csrc/ring.h, compiled by the host compiler, against a model of
mbarriers in which every role may be held back for as long as another can go on."""
import ctypes
import os
import random
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(__file__), os.pardir, "metaltile_b200", "csrc")


@pytest.fixture(scope="module")
def ring(tmp_path_factory):
    d = tmp_path_factory.mktemp("ring")
    src = d / "ring.cpp"
    src.write_text('#include "ring.h"\nusing namespace mtc::ring;\nextern "C" {\n'
                   "int fills_(int tma, int w) { return fills(tma, w); }\n"
                   "int fill_arrivals_(int tma) { return fill_arrivals(tma); }\n"
                   "}\n")
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", CSRC, str(src), "-o", str(d / "ring.so")], check=True)
    return ctypes.CDLL(str(d / "ring.so"))


class Barrier:
    """An mbarrier: a phase is complete when its arrivals have come."""

    def __init__(self, count):
        self.count = self.pending = count
        self.done = 0                       # phases that are complete

    def arrive(self, n=1):
        self.pending -= n
        assert self.pending >= 0, "more arrivals than a phase takes"
        if self.pending == 0:
            self.done, self.pending = self.done + 1, self.count

    def passed(self, parity):               # what try_wait.parity says
        return self.done % 2 != parity


def play(roles, last, rng):
    """Runs the roles (generators of conditions) to their ends; the one at ``last`` only where no other can go on.  False: some role waits for good."""
    waiting = [next(r, None) for r in roles]
    while any(w is not None for w in waiting):
        ready = [i for i, w in enumerate(waiting) if w is not None and w()]
        if not ready:
            return False
        held = [i for i in ready if i != last] or ready
        i = rng.choice(held)
        waiting[i] = next(roles[i], None)
    return True


def _copies(ring, buffers, blocks, tma, by_rule):
    """The two copy warps and a few dequantising warps over one kind of buffer; ``by_rule``: as fills() says, else both copy warps wait always."""
    readers = 4
    full = [Barrier(ring.fill_arrivals_(tma)) for _ in range(buffers)]
    empty = [Barrier(readers) for _ in range(buffers)]

    def copy(w):
        if by_rule and not ring.fills_(tma, w):
            return
        for i in range(blocks):
            b, par = i % buffers, i // buffers % 2
            yield lambda b=b, par=par: empty[b].passed(par ^ 1)
            if not tma:
                full[b].arrive(32)
            elif w == 0:
                full[b].arrive()

    def read():
        for i in range(blocks):
            b, par = i % buffers, i // buffers % 2
            yield lambda b=b, par=par: full[b].passed(par)
            empty[b].arrive()

    return [copy(0), copy(1)] + [read() for _ in range(readers)]


@pytest.mark.parametrize("tma", [0, 1])
@pytest.mark.parametrize("buffers", [2, 3, 4])
def test_no_copy_warp_is_overtaken(ring, buffers, tma):
    rng = random.Random(buffers)
    for blocks in (1, buffers, buffers + 1, 2 * buffers, 2 * buffers + 1, 23):
        for last in range(6):
            for _ in range(5):
                assert play(_copies(ring, buffers, blocks, tma, True), last, rng), (blocks, last)


def test_a_warp_that_nobody_waits_for_is():
    """What the rule is for: the model does find a second copy warp that waits for buffers which the first fills alone."""
    class Both:
        fills_ = staticmethod(lambda tma, w: 1)
        fill_arrivals_ = staticmethod(lambda tma: 1)

    assert not play(_copies(Both, 2, 2, 1, False), 1, random.Random(0))
