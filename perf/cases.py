"""The work a user of this package has it do, as cases that can be timed and compared.

Every case goes through the public entry points (``metaltile_b200.ops`` and ``Context``).  Kinds:

``proj``      one quantized projection issued by itself (``ops.qmv`` / ``ops.qvm``): where a call costs more than its bytes
``decode``    the projections of one decode step over all layers (q/k/v and gate/up share a launch, SwiGLU before down),
              replayed from a CUDA graph, as a server keeps it
``prefill``   the projections of one layer over a whole prompt (``ops.qmm``), issued call by call
``moe``       one mixture-of-experts layer: router, sort, expert MLP, unpermute
``codec``     a float weight matrix quantized at load time and dequantized again
``dispatch``  the name-keyed call on host buffers, the boundary the reference's own runtime has

Values follow the benchmark definition: codes uniform, scale ~ U(0.002, 0.02) * 16 / 2^bits,
bias = -2^(bits-1) * scale + N(0, 1e-3), activations and router logits ~ N(0, 1).
"""
import math

import numpy as np
import torch

from metaltile_b200 import ops

_DT = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}
_SIZE = {"bf16": 2, "f16": 2, "f32": 4}


# ---- the cases ---------------------------------------------------------------------------------------------------
def listed():
    return [
        # One attention projection for one token, the smallest call there is in earnest: launch and host time count.
        dict(name="proj_m1", kind="proj", op="qmv", m=1, n=4096, k=4096, bits=4, group=64, dtype="bf16"),
        # Four draft tokens verified on a 3-bit model with fine groups: a width whose codes straddle words.
        dict(name="proj_3bit_m4", kind="proj", op="qmv", m=4, n=8192, k=8192, bits=3, group=32, dtype="f16"),
        # A small batch kept in 32-bit activations on 8-bit weights (evaluation runs, final heads), odd row count.
        dict(name="proj_8bit_f32_m16", kind="proj", op="qmv", m=16, n=4099, k=4096, bits=8, group=64, dtype="f32"),
        # The other direction of the product, weights stored transposed (x @ W): one token.
        dict(name="qvm_m1", kind="proj", op="qvm", m=1, n=4096, k=14336, bits=4, group=64, dtype="bf16"),
        # Single-user generation with the Llama-3-8B-shaped set: every projection of all layers for one token.
        dict(name="decode_m1", kind="decode", m=1, layers=32, hidden=4096, kv=1024, ffn=14336, bits=4, group=64, dtype="bf16"),
        # The same model serving a batch of eight.
        dict(name="decode_m8", kind="decode", m=8, layers=32, hidden=4096, kv=1024, ffn=14336, bits=4, group=64, dtype="bf16"),
        # A long prompt through one layer of that model.
        dict(name="prefill_2048", kind="prefill", m=2048, hidden=4096, kv=1024, ffn=14336, bits=4, group=64, dtype="bf16"),
        # A short prompt of no round length on a small 8-bit model whose sizes are multiples of 64 only.
        dict(name="prefill_ragged", kind="prefill", m=333, hidden=2880, kv=576, ffn=7616, bits=8, group=32, dtype="f16"),
        # A prompt or a large batch through a layer of many small experts.
        dict(name="moe_512", kind="moe", tokens=512, hidden=2048, inter=768, experts=128, top_k=8, bits=4, group=64, dtype="bf16"),
        # The same layer while four users decode: few experts are hit, each by a row or two.
        dict(name="moe_4", kind="moe", tokens=4, hidden=2048, inter=768, experts=128, top_k=8, bits=4, group=64, dtype="bf16"),
        # Packing one feed-forward matrix while a model is loaded, and reading it back.
        dict(name="codec_4bit", kind="codec", n=14336, k=4096, bits=4, group=64, dtype="bf16"),
        # One kernel by its name on host buffers, as a test bench or a first integration calls it.
        dict(name="dispatch_qmv", kind="dispatch", n=2048, k=2048, group=64, dtype="bf16"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _mult(rng, lo, hi, step):
    """A multiple of ``step`` between lo and hi, spread over the logarithm; round sizes about half of the time."""
    if rng.random() < 0.5:
        step = max(step, 512)
    return max(step, _log(rng, lo, hi) // step * step)


def _format(rng):
    bits = rng.choice((4, 4, 4, 4, 8, 8, 6, 5, 3, 2))
    group = rng.choice((64, 64, 64, 128, 32))
    return dict(bits=bits, group=group)


def draw(rng):
    kind = rng.choice(("proj", "proj", "proj", "decode", "decode", "prefill", "prefill", "moe", "moe", "codec", "dispatch"))
    f = _format(rng)
    step = max(64, f["group"])
    if kind == "proj":
        op = rng.choice(("qmv", "qmv", "qmv", "qvm"))
        n = _log(rng, 512, 16384) if op == "qmv" else _mult(rng, 512, 16384, 64)
        m = rng.choice((1, 1, rng.randint(2, 4), rng.randint(5, 8), rng.randint(9, 16))) if op == "qmv" else rng.choice((1, 1, 2, 4))
        return dict(kind=kind, op=op, m=m, n=n, k=_mult(rng, 512, 16384, step), dtype=rng.choice(("bf16", "bf16", "f16", "f32")), **f)
    if kind in ("decode", "prefill"):
        hidden = _mult(rng, 1024, 4096, step)
        kv = max(step, hidden // rng.choice((1, 4, 8)) // step * step)
        ffn = max(step, int(hidden * rng.uniform(1.5, 3.5)) // step * step)
        dims = dict(hidden=hidden, kv=kv, ffn=ffn, dtype=rng.choice(("bf16", "bf16", "f16")), **f)
        if kind == "decode":
            return dict(kind=kind, m=rng.choice((1, 1, rng.randint(2, 8), rng.randint(9, 16))), layers=rng.randint(2, 8), **dims)
        return dict(kind=kind, m=_log(rng, 17, 2048), **dims)
    if kind == "moe":
        experts = rng.choice((8, 16, 32, 64, 128))
        hidden, inter = _mult(rng, 512, 2048, step), _mult(rng, 256, 1536, step)
        return dict(kind=kind, tokens=_log(rng, 1, 512), hidden=hidden, inter=inter, experts=experts,
                    top_k=rng.choice((1, 2, 4, 6, 8)), dtype=rng.choice(("bf16", "bf16", "f16")), **f)
    if kind == "codec":
        return dict(kind=kind, n=_log(rng, 256, 14336), k=_mult(rng, 512, 4096, step), dtype=rng.choice(("bf16", "f16", "f32")), **f)
    return dict(kind=kind, n=_mult(rng, 256, 4096, 64), k=_mult(rng, 512, 4096, step), group=f["group"],
                dtype=rng.choice(("bf16", "f16", "f32")))


# ---- inputs ------------------------------------------------------------------------------------------------------
class _Maker:
    """Seeded inputs on the GPU."""

    def __init__(self, seed, dtype):
        self.gen = torch.Generator(device="cuda")
        self.gen.manual_seed(int(seed))
        self.dt = _DT[dtype]

    def normal(self, *shape):
        return torch.randn(shape, device="cuda", generator=self.gen).to(self.dt)

    def words(self, *shape):
        return torch.randint(-2 ** 31, 2 ** 31, shape, dtype=torch.int32, device="cuda", generator=self.gen)

    def matrix(self, shape, k, bits, group, transposed=False):
        """(w, scales, biases) of ``shape + (k,)`` codes; ``transposed``: k rows of shape[0] codes, groups along k."""
        if transposed:
            w, s_shape = self.words(k, shape[0] * bits // 32), (k // group, shape[0])
        else:
            w, s_shape = self.words(*shape, k * bits // 32), tuple(shape) + (k // group,)
        scales = (0.002 + 0.018 * torch.rand(s_shape, device="cuda", generator=self.gen)) * (16.0 / 2 ** bits)
        biases = -(2.0 ** (bits - 1)) * scales + 1e-3 * torch.randn(s_shape, device="cuda", generator=self.gen)
        return w, scales.to(self.dt), biases.to(self.dt)


def _prepare_proj(c, mk):
    mat = mk.matrix((c["n"],), c["k"], c["bits"], c["group"], transposed=c["op"] == "qvm")
    return dict(mat=mat, x=mk.normal(c["m"], c["k"]))


def _prepare_decode(c, mk):
    m, h, kv, ffn, n_layers = c["m"], c["hidden"], c["kv"], c["ffn"], c["layers"]
    fmt = (c["bits"], c["group"])
    layers = [dict(q=mk.matrix((h,), h, *fmt), k=mk.matrix((kv,), h, *fmt), v=mk.matrix((kv,), h, *fmt), o=mk.matrix((h,), h, *fmt),
                   gate=mk.matrix((ffn,), h, *fmt), up=mk.matrix((ffn,), h, *fmt), down=mk.matrix((h,), ffn, *fmt))
              for _ in range(n_layers)]
    xs = dict(qkv=mk.normal(m, h), o=mk.normal(m, h), mlp=mk.normal(m, h))
    outs = {name: torch.empty((n_layers, m, n), dtype=mk.dt, device="cuda")
            for name, n in (("q", h), ("k", kv), ("v", kv), ("o", h), ("gate", ffn), ("up", ffn), ("act", ffn), ("down", h))}
    ctx = ops.context()

    def project(layer, i, names, x):
        ctx.qmv_batched([dict(w=layer[n][0].data_ptr(), scales=layer[n][1].data_ptr(), biases=layer[n][2].data_ptr(), x=x.data_ptr(),
                              outs=[outs[n][i].data_ptr()], M=m, N=outs[n].shape[2], K=x.shape[1], bits=c["bits"],
                              group_size=c["group"], dtype=c["dtype"]) for n in names], torch.cuda.current_stream().cuda_stream)

    def step():
        for i, layer in enumerate(layers):
            project(layer, i, ("q", "k", "v"), xs["qkv"])
            project(layer, i, ("o",), xs["o"])
            project(layer, i, ("gate", "up"), xs["mlp"])
            ops.swiglu(outs["gate"][i], outs["up"][i], out=outs["act"][i])
            project(layer, i, ("down",), outs["act"][i])

    step()                       # blocks that the library keeps reach their size before the capture
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        step()
    return dict(graph=graph, layers=layers, xs=xs, outs=outs)


def _prepare_prefill(c, mk):
    m, h, kv, ffn = c["m"], c["hidden"], c["kv"], c["ffn"]
    fmt = (c["bits"], c["group"])
    mats = dict(q=mk.matrix((h,), h, *fmt), k=mk.matrix((kv,), h, *fmt), v=mk.matrix((kv,), h, *fmt), o=mk.matrix((h,), h, *fmt),
                gate=mk.matrix((ffn,), h, *fmt), up=mk.matrix((ffn,), h, *fmt), down=mk.matrix((h,), ffn, *fmt))
    return dict(mats=mats, xs=dict(qkv=mk.normal(m, h), o=mk.normal(m, h), mlp=mk.normal(m, h)))


def _prepare_moe(c, mk):
    e, h, i = c["experts"], c["hidden"], c["inter"]
    fmt = (c["bits"], c["group"])
    return dict(gate=mk.matrix((e, i), h, *fmt), up=mk.matrix((e, i), h, *fmt), down=mk.matrix((e, h), i, *fmt),
                x=mk.normal(c["tokens"], h), logits=mk.normal(c["tokens"], e))


def _prepare_codec(c, mk):
    return dict(w=mk.normal(c["n"], c["k"]) * 0.02)


def _prepare_dispatch(c, mk):
    w, s, b = mk.matrix((c["n"],), c["k"], 4, c["group"])
    x = mk.normal(1, c["k"])
    raw = lambda t: t.contiguous().view(torch.uint8).cpu().numpy().tobytes()  # noqa: E731
    bufs = dict(w=raw(w), scales=raw(s), biases=raw(b), x=raw(x), out=bytes(c["n"] * _SIZE[c["dtype"]]))
    return dict(bufs=bufs, consts=dict(k=c["k"], gs_per_row=c["k"] // c["group"]), ctx=ops.context())


def prepare(case, seed):
    made = globals()["_prepare_" + case["kind"]](case, _Maker(seed, case.get("dtype", "bf16")))
    return dict(made, case=case)


# ---- one pass ----------------------------------------------------------------------------------------------------
def _run_proj(c, s):
    op = ops.qvm if c["op"] == "qvm" else ops.qmv
    return op(*s["mat"], s["x"], c["bits"], c["group"])


def _run_decode(c, s):
    s["graph"].replay()
    return {n: s["outs"][n] for n in ("q", "k", "v", "o", "act", "down")}


def _run_prefill(c, s):
    def project(name, x):
        return ops.qmm(*s["mats"][name], x, c["bits"], c["group"])

    out = {n: project(n, s["xs"]["qkv"]) for n in ("q", "k", "v")}
    out["o"] = project("o", s["xs"]["o"])
    out["act"] = ops.swiglu(project("gate", s["xs"]["mlp"]), project("up", s["xs"]["mlp"]))
    out["down"] = project("down", out["act"])
    return out


def _run_moe(c, s):
    idx, weights = ops.moe_router_topk(s["logits"], c["top_k"])
    order, inverse, offsets, _ = ops.moe_sort(idx, c["experts"])
    y = ops.moe_experts(s["x"], s["gate"], s["up"], s["down"], c["bits"], c["group"], offsets, sort_token_idx=order)
    return dict(idx=idx, weights=weights, offsets=offsets, y=ops.moe_unpermute(y, inverse, weights))


def _run_codec(c, s):
    w, scales, biases = ops.affine_quantize(s["w"], c["bits"], c["group"])
    return dict(w=w, scales=scales, biases=biases, back=ops.affine_dequantize(w, scales, biases, c["bits"], c["group"]))


def _run_dispatch(c, s):
    got = s["ctx"].dispatch_with_grid("mt_qmv", s["bufs"], s["consts"], (c["n"] // 8, 1, 1), (64, 1, 1), dtype=c["dtype"])
    bits = np.frombuffer(got.outputs["out"], dtype=np.uint8)
    return torch.from_numpy(bits.copy()).view(_DT[c["dtype"]])


def run(state):
    case = state["case"]
    return globals()["_run_" + case["kind"]](case, state)


# ---- what a pass cannot do without ---------------------------------------------------------------------------------
def _product(c, m, n, k, bits=None, mats=1, reads_x=True):
    """Bytes and operations of ``mats`` products that share x: packed words, scales and biases, x once, the outputs."""
    size = _SIZE[c["dtype"]]
    weights = n * k * (bits or c["bits"]) / 8 + 2 * n * (k // c["group"]) * size
    return mats * (weights + m * n * size) + (m * k * size if reads_x else 0), 2.0 * mats * m * n * k


def work(case):
    c, kind, parts = case, case["kind"], []
    if kind == "proj":
        parts = [_product(c, c["m"], c["n"], c["k"])]
    elif kind in ("decode", "prefill"):
        m, h, kv, ffn = c["m"], c["hidden"], c["kv"], c["ffn"]
        parts = [_product(c, m, h, h), _product(c, m, kv, h, mats=2, reads_x=False), _product(c, m, h, h),
                 _product(c, m, ffn, h, mats=2), (3 * m * ffn * _SIZE[c["dtype"]], 0), _product(c, m, h, ffn)] * c.get("layers", 1)
    elif kind == "moe":
        rows, size = c["tokens"] * c["top_k"], _SIZE[c["dtype"]]
        hit = c["experts"] * (1 - (1 - c["top_k"] / c["experts"]) ** c["tokens"])      # experts that get a row, on average
        per_row = size * (2 * c["hidden"] + 4 * c["inter"])
        codes = 3 * c["hidden"] * c["inter"]
        weights = hit * (codes * c["bits"] / 8 + 2 * codes / c["group"] * size)
        parts = [(weights + rows * per_row + c["tokens"] * size * (2 * c["hidden"] + c["experts"]), 2.0 * rows * codes)]
    elif kind == "codec":
        n, size = c["n"] * c["k"], _SIZE[c["dtype"]]
        packed = n * c["bits"] / 8 + 2 * n / c["group"] * size
        parts = [(2 * n * size + 2 * packed, 6.0 * n)]
    elif kind == "dispatch":
        parts = [_product(c, 1, c["n"], c["k"], bits=4)]
    return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}


def tolerance(case):
    if case["kind"] == "codec":
        return "exact"           # every float operation of the codec is rounded on its own, by definition
    # 32-bit sums; results (and, in the tensor-core kernels, dequantized weights) rounded to the activations' type
    return {"rel": {"f32": 1e-5, "f16": 2e-3, "bf16": 1e-2}[case["dtype"]]}
