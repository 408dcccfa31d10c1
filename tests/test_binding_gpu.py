"""The native binding of the typed ops and of the name-keyed call, from Python's side: threads, and the forms of host buffers
and sizes that the call takes."""
import _thread
import sys
import threading

import pytest

from helpers import dense_case, to_dev

pytestmark = pytest.mark.gpu


def _ops_to_call():
    """Every op that takes ``out``: nothing but the library's entry runs between the checks and the return (making or freeing a
    tensor may let go of the interpreter lock by itself)."""
    import torch
    from metaltile_b200 import ops
    w, s, b, x = (to_dev(a) if i == 0 else to_dev(a, "bf16") for i, a in enumerate(dense_case(4, 256, 512, 4, 64, "bf16", seed=1)))
    wt, st, bt = ops.affine_quantize(torch.randn(512, 512, device="cuda").to(torch.bfloat16), 4, 64)
    t_s, t_b = torch.ones(8, 512, dtype=torch.bfloat16, device="cuda"), torch.zeros(8, 512, dtype=torch.bfloat16, device="cuda")
    idx, wts = ops.moe_router_topk(torch.randn(4, 16, device="cuda"), 2)
    wts = wts.to(torch.bfloat16)
    order, inverse, offsets, _ = ops.moe_sort(idx, 16)
    we, se, be = w.view(16, 16, -1), s.view(16, 16, -1), b.view(16, 16, -1)
    rows = x.repeat(2, 1)
    mats = [ops.affine_quantize(torch.randn(16, o, i, device="cuda").to(torch.bfloat16), 4, 64) for o, i in ((256, 512), (256, 512), (512, 256))]
    new = lambda *size: torch.empty(size, dtype=torch.bfloat16, device="cuda")  # noqa: E731
    o256, o512, o1, o2, o16, y, x1 = new(4, 256), new(4, 512), new(1, 256), new(1, 512), new(8, 16), new(8, 512), x[:1].clone()
    return {
        "qmv": lambda: ops.qmv(w, s, b, x, 4, 64, out=o256), "qmm": lambda: ops.qmm(w, s, b, x, 4, 64, out=o256),
        "qmv_batched": lambda: ops.qmv_batched([(w, s, b), (w, s, b)], x1, 4, 64, out=o2),
        "qvm": lambda: ops.qvm(wt, t_s, t_b, x, 4, 64, out=o512), "swiglu": lambda: ops.swiglu(x, x, out=o512),
        "rms_norm_qmv": lambda: ops.rms_norm_qmv(w, s, b, x1, x1, 1e-5, 4, 64, out=o1),
        "permute": lambda: ops.moe_permute(x, order, out=y), "unpermute": lambda: ops.moe_unpermute(rows, inverse, wts, out=o512),
        "gather": lambda: ops.gather_qmm(rows, we, se, be, 4, 64, expert_offsets=offsets, out=o16),
        "experts": lambda: ops.moe_experts(x, *mats, 4, 64, offsets, sort_token_idx=order, out=y),
    }


def test_other_threads_run_during_a_call():
    """The library is called without the interpreter lock (a call may wait for the GPU's queue, an allocation or the first load
    of a kernel, and another thread may drive another GPU meanwhile).  With a switch interval that never comes, a second
    thread gets to run only when the first one lets go of the lock inside the call."""
    import torch
    calls = _ops_to_call()
    missing = []
    for name, call in calls.items():
        call()                                                       # loads its kernel
        torch.cuda.synchronize()
        old = sys.getswitchinterval()
        ran, stop = threading.Event(), threading.Event()

        def other():
            ran.set()
            stop.wait()

        sys.setswitchinterval(1000.0)
        try:
            _thread.start_new_thread(other, ())                      # (Thread.start() would wait for it and so let it run)
            assert not ran.is_set()
            for _ in range(20000):
                call()
                if ran.is_set():
                    break
            if not ran.is_set():
                missing.append(name)
        finally:
            sys.setswitchinterval(old)
            stop.set()
    torch.cuda.synchronize()
    assert not missing


def test_threads_with_contexts_of_their_own():
    """Two threads, each with its own Context and stream, call at the same time; an error raised in one stays in it."""
    import torch
    from metaltile_b200 import Context, ops
    w, s, b, x = (to_dev(a) if i == 0 else to_dev(a, "f16") for i, a in enumerate(dense_case(300, 256, 512, 8, 64, "f16", seed=2)))
    want = [ops.qmm(w, s, b, x[:m], 8, 64) for m in (3, 40, 300)]
    torch.cuda.synchronize()
    wrong = []

    def work(seed):
        own = Context(0)
        with torch.cuda.stream(torch.cuda.Stream()):
            for i in range(200):
                k = (i + seed) % 3
                got = ops.qmm(w, s, b, x[:(3, 40, 300)[k]], 8, 64, ctx=own)
                try:
                    ops.qmm(w, s, b, x, 8, 48, ctx=own)
                    wrong.append("accepted")
                except ValueError:
                    pass
                torch.cuda.current_stream().synchronize()
                if not torch.equal(got, want[k]):
                    wrong.append((seed, i))

    threads = [threading.Thread(target=work, args=(t,)) for t in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
