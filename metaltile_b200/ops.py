"""Typed ops on tensors that already live on the GPU.

PyTorch is used only as the owner of device memory and streams: every function hands raw device pointers and the
current CUDA stream to ``libmtcuda.so``.  The argument checks, the output allocation and the call itself are in the
native binding (``csrc/binding.cpp``): through ctypes they cost 12-18 us a call, more than most decode kernels.
"""
from __future__ import annotations

import torch

from . import _lib
from ._lib import BF16, F16, F32
from .context import Context

_lib.load()                                  # checks that the library exports what the header declares
try:
    from . import _native
except ImportError as e:
    raise ImportError(f"the native binding of the typed ops is missing ({e}): build it with `python -m metaltile_b200.build` "
                      "(there is no CPU or PyTorch fallback for these ops)") from e

if _native.torch_version != torch.__version__:
    raise ImportError(f"the native binding of the typed ops was compiled against PyTorch {_native.torch_version}, this is {torch.__version__}: "
                      "build it again with `python -m metaltile_b200.build`")

_TORCH_DT = {torch.float32: F32, torch.float16: F16, torch.bfloat16: BF16}

_ctx_cache = {}


def context(device=None) -> Context:
    """The process-wide Context of a device (created on first use)."""
    idx = torch.cuda.current_device() if device is None else torch.device(device).index or 0
    if idx not in _ctx_cache:
        _ctx_cache[idx] = Context(idx)
    return _ctx_cache[idx]


_native.set_context(context)


def _check_dense(w, scales, biases, x, bits, group_size):
    if not (w.is_cuda and scales.is_cuda and biases.is_cuda and x.is_cuda):
        raise ValueError("all operands must be CUDA tensors")
    if w.dtype not in (torch.int32, torch.uint32):
        raise TypeError("w must hold packed 32-bit words (torch.int32 / torch.uint32)")
    if x.dtype not in _TORCH_DT or scales.dtype != x.dtype or biases.dtype != x.dtype:
        raise TypeError("x, scales and biases must share one dtype in {f32, f16, bf16}")
    x2 = x.reshape(-1, x.shape[-1])
    M, K = x2.shape
    N = w.shape[0]
    if w.shape[1] * 32 != K * bits:
        raise ValueError(f"w has {w.shape[1]} words per row, expected K*bits/32 = {K * bits / 32}")
    if scales.shape != (N, K // group_size) or biases.shape != scales.shape:
        raise ValueError("scales/biases must be [N, K/group_size]")
    for t in (w, scales, biases, x2):
        if not t.is_contiguous():
            raise ValueError("operands must be contiguous")
    return x2, M, N, K


def _check_out(out, M, N, like):
    """A caller-supplied output must be the dense row-major [M, N] block the kernels write."""
    if out.device != like.device or out.dtype != like.dtype:
        raise TypeError("out must live on the same device and have the dtype of x")
    if out.numel() != M * N or not out.is_contiguous():
        raise ValueError(f"out must be a contiguous block of M*N = {M * N} elements "
                         "(a column slice of a wider tensor with M > 1 is not)")


def qmv(w, scales, biases, x, bits: int, group_size: int, out=None, ctx: Context = None):
    """out[M, N] = x[M, K] @ dequant(w)[N, K]^T (decode, M <= 16 tuned); ``Context.launch_of`` names the kernel."""
    return _native.dense(0, w, scales, biases, x, bits, group_size, out, ctx)


def qmm(w, scales, biases, x, bits: int, group_size: int, out=None, ctx: Context = None):
    """Like ``qmv`` but routed by M as the reference's ``mt_qmm_for`` does (prefill -> tensor cores)."""
    return _native.dense(1, w, scales, biases, x, bits, group_size, out, ctx)


def _projection(w, scales, biases, x, bits, group_size, outs, phase=0):
    x2, M, N, K = _check_dense(w, scales, biases, x, bits, group_size)
    for o in outs:
        _check_out(o, M, N, x)
    return {"w": w.data_ptr(), "scales": scales.data_ptr(), "biases": biases.data_ptr(), "x": x2.data_ptr(),
            "outs": [o.data_ptr() for o in outs], "M": M, "N": N, "K": K, "bits": bits, "group_size": group_size,
            "dtype": _TORCH_DT[x.dtype], "phase": phase}


def qmv_batched(mats, x, bits: int, group_size: int, out=None, ctx: Context = None):
    """Several projections of the same activations in one launch: ``mats`` = [(w, scales, biases), ...] (1 to 4).

    Returns ``out[M, sum(N_i)]`` with the results side by side - for M = 1 the concatenated vector of
    ``ffai_batched_qkv_qgemv`` (crates/metaltile-std/src/ffai/batched_qkv_qgemv.rs:1-35).  For M > 1 every
    projection writes its own contiguous [M, N_i] tile and the tiles are returned as a list instead.  The f32 sums of a fused
    projection may be added in another order than ``qmv`` of it alone adds them (the last bit of an output may differ); the
    same call always gives the same bits."""
    return _native.qmv_batched(mats, x, bits, group_size, out, ctx)


def unpack_codes(w, K: int, bits: int, ctx: Context = None):
    """u8[N, K] integer codes of a packed matrix (for bit-exact checks)."""
    return _native.unpack_codes(w, K, bits, ctx)


# ---- MoE -----------------------------------------------------------------------------------------
def moe_router_topk(logits, k: int, norm_topk_prob: int = 1, ctx: Context = None):
    """(indices int32[rows, k], weights T[rows, k]) of ``mt_moe_router_topk``."""
    return _native.moe_router_topk(logits, k, norm_topk_prob, ctx)


def moe_sort(topk_idx, n_experts: int, ctx: Context = None):
    """Stable expert sort: (sort_token_idx[T*k], inv_perm[T, k], expert_offsets[E+1], row_expert[T*k]), int32."""
    return _native.moe_sort(topk_idx, n_experts, ctx)


def moe_permute(tokens, sort_token_idx, out=None, ctx: Context = None):
    return _native.moe_permute(tokens, sort_token_idx, out, ctx)


def moe_unpermute(expert_outputs, inv_perm, weights, out=None, ctx: Context = None):
    return _native.moe_unpermute(expert_outputs, inv_perm, weights, out, ctx)


def swiglu(gate, up, out=None, ctx: Context = None):
    return _native.swiglu(gate, up, out, ctx)


def gather_qmm(x, w, scales, biases, bits: int, group_size: int, expert_offsets=None, indices=None, out=None,
               ctx: Context = None):
    """out[t, n] = sum_k x[t, k] * dequant(w[E(t)])[n, k]; x rows sorted by expert; w [E, n_out, k*bits/32]."""
    return _native.gather_qmm(x, w, scales, biases, bits, group_size, expert_offsets, indices, out, ctx)


def moe_experts(x, gate, up, down, bits: int, group_size: int, expert_offsets, sort_token_idx=None, out=None, ctx: Context = None):
    """y[r] = down_e(silu(gate_e(x_r)) * up_e(x_r)) for rows sorted by expert; gate / up / down are (w, scales, biases)
    with w [E, inter, hidden*bits/32] (gate, up) and [E, hidden, inter*bits/32] (down).  ``sort_token_idx`` folds the
    permutation in: row r reads ``x[sort_token_idx[r]]``."""
    return _native.moe_experts(x, gate, up, down, bits, group_size, expert_offsets, sort_token_idx, out, ctx)


def rms_norm_qmv(w, scales, biases, x, norm_weight, eps: float, bits: int, group_size: int, out=None, ctx: Context = None):
    """``qmv(rms_norm(x) * norm_weight)`` in one launch (``ffai_rms_norm_qgemv``,
    crates/metaltile-std/src/ffai/rms_norm_qgemv.rs:51-107): x and norm_weight are vectors of length K, out [1, N]."""
    return _native.rms_norm_qmv(w, scales, biases, x, norm_weight, eps, bits, group_size, out, ctx)


def affine_quantize(w, bits: int, group_size: int, ctx: Context = None):
    """Float tensor ``w [..., K]`` (K a multiple of the group size) -> (packed int32 ``[..., K*bits/32]``, scales, biases
    ``[..., K/group_size]``) in the layout the quantized matmuls read (``mt_affine_quantize_int*``,
    crates/metaltile-std/src/mlx/quantized.rs:3629-3667).  A product of them may follow on the same stream at once: the
    context keeps it from requesting its weights before they are written (other writers: option ``pdl_early_weights``)."""
    return _native.affine_quantize(w, bits, group_size, ctx)


def affine_dequantize(w, scales, biases, bits: int, group_size: int, ctx: Context = None):
    """The inverse of ``affine_quantize``: ``scale * q + bias`` in the type of ``scales`` (``mt_affine_dequantize_int*``)."""
    return _native.affine_dequantize(w, scales, biases, bits, group_size, ctx)


def dequant_gather(weight, scales, biases, indices, bits: int, group_size: int, ctx: Context = None):
    """Rows ``indices`` (int32) of a quantized table ``weight [vocab, hidden*bits/32]`` dequantized: ``[n_tokens, hidden]``
    in the type of ``scales`` (``dequant_gather_int*``, crates/metaltile-std/src/ffai/dequant_gather.rs:44-101)."""
    return _native.dequant_gather(weight, scales, biases, indices, bits, group_size, ctx)


def qvm(w, scales, biases, x, bits: int, group_size: int, out=None, ctx: Context = None):
    """``x @ W`` with W stored transposed and quantized along K: w [K, N*bits/32], scales / biases [K/group_size, N],
    x [M, K] -> out [M, N] (``mt_qvm_*``, crates/metaltile-std/src/mlx/quantized.rs:4397-4530).  Like the other dense products
    it requests its first weights while the previous kernel of the stream drains (option ``pdl_early_weights``)."""
    return _native.qvm(w, scales, biases, x, bits, group_size, out, ctx)
