"""The barrier protocol of the tcgen05 kernels' rings, played on the CPU: the rules of csrc/ring.cuh, compiled by the host compiler, against a model of
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
    src.write_text('#include "ring.cuh"\nusing namespace mtc::ring;\nextern "C" {\n'
                   "int fills_(int tma, int w) { return fills(tma, w); }\n"
                   "int fill_arrivals_(int tma) { return fill_arrivals(tma); }\n"
                   "int last_parity_(unsigned n, int slots, int slot) { return last_parity(n, slots, slot); }\n"
                   "int owed_(unsigned use, int teams, int team) { return owed(use, teams, team); }\n"
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


def _gives_up(ring, slots, teams, uses, steps, rng):
    """Copies, teams that convert and MMAs over one ring; after ``steps`` steps every wait fails.  Returns what leaving has to put right: the barriers, the
    copies still on their way, the uses that were issued, how far each warp came."""
    per = 4                                                  # warps of a team; MMAs as in the kernel: full takes the copy's arrival and theirs
    full = [Barrier(1 + per) for _ in range(slots)]
    empty = [Barrier(1) for _ in range(slots)]
    landing, state = [], dict(issued=0, converted=[0] * (per * teams))

    def producer():
        for u in range(uses):
            yield lambda b=u % slots, par=u // slots % 2: empty[b].passed(par ^ 1)
            landing.append(u % slots)                        # the copy's bytes hold the phase open as an arrival does
            state["issued"] = u + 1

    def convert(w):
        for u in range(uses):
            if u % teams == w // per:
                yield lambda b=u % slots, par=u // slots % 2: empty[b].passed(par ^ 1)
                full[u % slots].arrive()
            state["converted"][w] = u + 1

    def mma():
        for u in range(uses):
            yield lambda b=u % slots, par=u // slots % 2: full[b].passed(par)
            empty[u % slots].arrive()

    roles = [producer(), mma()] + [convert(w) for w in range(per * teams)]
    waiting = [next(r, None) for r in roles]
    for _ in range(steps):
        ready = [i for i, w in enumerate(waiting) if w is not None and w()]
        if landing and (not ready or rng.random() < 0.3):
            full[landing.pop(rng.randrange(len(landing)))].arrive()
        elif ready:
            i = rng.choice(ready)
            waiting[i] = next(roles[i], None)
    return full, landing, state


@pytest.mark.parametrize("slots,teams", [(1, 1), (2, 2), (3, 3), (4, 3), (8, 3)])
def test_leaving_waits_for_every_copy(ring, slots, teams):
    """Wherever the roles stop: with the arrivals that are owed every issued copy's phase completes when the copy lands, not before, and takes no other."""
    rng = random.Random(slots)
    for trial in range(300):
        full, landing, state = _gives_up(ring, slots, teams, 20, rng.randrange(400), rng)
        issued = state["issued"]
        for w, done in enumerate(state["converted"]):
            for u in range(done, issued):
                if ring.owed_(u, teams, w // 4):
                    full[u % slots].arrive()
        parity = [ring.last_parity_(issued, slots, b) for b in range(slots)]
        for b in range(slots):
            if parity[b] >= 0:
                assert full[b].passed(parity[b]) == (b not in landing)
        for b in landing:
            full[b].arrive()
        assert all(full[b].passed(p) for b, p in enumerate(parity) if p >= 0)
        assert [p for p in parity if p < 0] == [-1] * max(0, slots - issued)
