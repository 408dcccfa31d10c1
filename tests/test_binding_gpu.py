"""The native binding of the typed ops and of the name-keyed call, from Python's side: threads, and the forms of host buffers
and sizes that the call takes."""
import _thread
import sys
import threading

import numpy as np
import pytest

from helpers import bytes_to_f32, dense_case, dt_bytes, to_dev

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


def test_threads_that_quantize_and_multiply():
    """Two threads on streams of their own and one Context: weights are packed and used at once in both (no shared scratch block)."""
    import torch
    from metaltile_b200 import ops
    ctx = ops.context(0)
    gen = torch.Generator(device="cuda").manual_seed(1)
    ws = [torch.randn(512, 1024, device="cuda", generator=gen).to(torch.bfloat16) for _ in range(8)]
    x = torch.randn(4, 1024, device="cuda", generator=gen).to(torch.bfloat16)
    want = []
    for w in ws:
        want.append(ops.qmv(*ops.affine_quantize(w, 8, 64, ctx=ctx), x, 8, 64, ctx=ctx))
        torch.cuda.synchronize()
    wrong = []

    def work(seed):
        with torch.cuda.stream(torch.cuda.Stream()):
            for i in range(400):
                k = (i * 3 + seed) % len(ws)
                got = ops.qmv(*ops.affine_quantize(ws[k], 8, 64, ctx=ctx), x, 8, 64, ctx=ctx)
                if not torch.equal(got, want[k]):
                    wrong.append((seed, i))

    threads = [threading.Thread(target=work, args=(t,)) for t in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong


def _qmv_call(ctx, n, k, dt="f32", form=bytes, grid=(1, 1, 1), extra=0):
    w, s, b, x = dense_case(1, n, k, 4, 64, dt, seed=3)
    esz = 4 if dt == "f32" else 2
    bufs = dict(w=form(w.tobytes()), scales=form(dt_bytes(s, dt)), biases=form(dt_bytes(b, dt)), x=form(dt_bytes(x, dt)), out=form(bytes(n * esz + extra)))
    return ctx.dispatch_with_grid("mt_qmv_b4", bufs, dict(k=k, n=n, group_size=64), grid, (64, 1, 1), dtype=dt)


def _strided(raw):
    a = np.zeros((len(raw), 2), dtype=np.uint8)
    a[:, 0] = np.frombuffer(raw, dtype=np.uint8)
    return a[:, 0]


def test_forms_of_host_buffers_and_sizes():
    """Whatever bytes() takes: bytes, bytearray, memoryview, an array, a strided array, a list; sizes that int() takes, three at most."""
    from metaltile_b200 import ops
    ctx = ops.context(0)
    want = _qmv_call(ctx, 64, 512).outputs["out"]
    for form in (bytearray, memoryview, lambda r: np.frombuffer(r, dtype=np.uint8), _strided, list):
        assert _qmv_call(ctx, 64, 512, form=form).outputs["out"] == want
    for grid in ((8.0, 1.0, 1.0), (np.int64(8), 1, True), (8,)):
        assert _qmv_call(ctx, 64, 512, grid=grid).outputs["out"] == want
    with pytest.raises(IndexError):
        _qmv_call(ctx, 64, 512, grid=(8, 1, 1, 1))
    with pytest.raises(TypeError):
        _qmv_call(ctx, 64, 512, form=lambda r: "text")


@pytest.mark.parametrize("k", [4096, 16384, 65536])
def test_staging_at_its_limits(k):
    """Inputs below, at and above the size up to which they travel together (64 KiB), outputs below and past the block they come back
    through (1 MiB), outputs with bytes behind the result, and a call after one that failed with its uploads under way."""
    from metaltile_b200 import MetalTileError, ops
    ctx = ops.context(0)
    for n in {4096: (8, 32, 4096, 300000), 16384: (8, 9, 64), 65536: (2, 3, 16)}[k]:
        got = _qmv_call(ctx, n, k, extra=12)
        assert len(got.outputs["out"]) == n * 4 + 12 and got.outputs["out"][-12:] == bytes(12)
        w, s, b, x = dense_case(1, n, k, 4, 64, "f32", seed=3)
        dev = ops.qmv(to_dev(w), to_dev(s, "f32"), to_dev(b, "f32"), to_dev(x, "f32"), 4, 64, ctx=ctx).cpu().numpy().reshape(-1)
        assert np.array_equal(bytes_to_f32(got.outputs["out"][:n * 4], "f32"), dev)
        with pytest.raises(MetalTileError):              # k > 32 experts a token: refused by the entry, after the uploads
            ctx.dispatch_with_grid("mt_moe_router_topk", dict(router_logits=bytes(4 * 64 * 64), indices_out=bytes(64 * 160), weights_out=bytes(64 * 160)),
                                   dict(n_experts=64, k=40), (1, 1, 1), (32, 1, 1), dtype="f32", outputs=("indices_out", "weights_out"))
        assert _qmv_call(ctx, n, k, extra=12).outputs["out"] == got.outputs["out"]
