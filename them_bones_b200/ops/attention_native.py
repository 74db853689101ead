"""Autograd wrapper of the sm_100a attention kernels (``csrc/attention.cu``, ``csrc/attention_bwd_split.cu``).

Forward: RoPE + QK-norm pre-pass into a ``[B*T, 2*H*D]`` buffer, then the persistent tcgen05 flash-attention kernel
reading the values in place from the packed ``qkv``.  Saved for backward: ``qkv``, the rotated/normalised ``qk``, the
output and ``lse``.  Backward (``ops/attention_bwd.py``): a statistics pre-pass, the dK/dV kernel and the dQ kernel
(every accumulator in TMEM, bf16 outputs, no atomics), then the pre-pass backward that applies the norm Jacobian and
the inverse rotation and writes one packed ``[B, T, 3*H*D]`` gradient (reference: the fused backward emits one packed
gradient, round2/source/kernels/nki_attn_bandpro.py:1-134).
"""
from __future__ import annotations

import ctypes

import torch

from . import _lib as L
from .attention_bwd import _aligned

_I, _L, _F = ctypes.c_int, ctypes.c_longlong, ctypes.c_float
SUPPORTED_HEAD_DIMS = (128, 64)


def why_not(qkv, n_head, head_dim, window=0) -> str:
    """Empty when the kernels cover the call, else the reason."""
    from . import attention_bwd as AB
    if qkv.dtype != torch.bfloat16:
        return f"dtype {qkv.dtype} (bf16 only)"
    if head_dim not in SUPPORTED_HEAD_DIMS:
        return f"head_dim {head_dim} (supported: {SUPPORTED_HEAD_DIMS})"
    if qkv.shape[1] % AB.length_multiple(head_dim):
        return f"sequence length {qkv.shape[1]} is not a multiple of 128"
    if window % 128:
        return f"window {window} is not a multiple of 128"
    return ""


def applies(qkv, n_head, head_dim) -> bool:
    return not why_not(qkv, n_head, head_dim)


def _lse_buffer(b, t, n_head, dev):
    """The log-sum-exp rows ``[b, n_head, t]`` and, behind them, the int the forward kernel draws its work items from."""
    n = b * n_head * t
    buf = torch.empty(n + 1, dtype=torch.float32, device=dev)
    return buf, buf.data_ptr() + 4 * n


def rope_qknorm(qkv2, cos, sin, t, n_head, head_dim):
    m = qkv2.shape[0]
    qk = torch.empty(m, 2 * n_head * head_dim, dtype=qkv2.dtype, device=qkv2.device)
    L.call("bones_rope_qknorm_fwd", L.ptr(qkv2), L.ptr(cos), L.ptr(sin), L.ptr(qk), L.ptr(None), _L(m), _I(t), _I(n_head), _I(head_dim),
           L.stream())
    return qk


def attn_forward(qk, qkv2, doc_start, b, t, n_head, scale, window, head_dim=128):
    """The attention kernel alone, on rotated and normalised ``qk``; returns ``y`` and ``lse [b, n_head, t]``."""
    y = torch.empty(b * t, n_head * head_dim, dtype=qkv2.dtype, device=qkv2.device)
    lse = torch.empty(b, n_head, t, dtype=torch.float32, device=qkv2.device)
    counter = torch.zeros(1, dtype=torch.int32, device=qkv2.device)
    L.call("bones_attn_fwd", L.ptr(qk), L.ptr(qkv2), L.ptr(y), L.ptr(lse), L.ptr(doc_start), L.ptr(counter), _I(b), _I(t), _I(n_head),
           _I(head_dim), _F(scale), _I(window // 128), L.stream())
    return y, lse


class _AttnFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, qkv, cos, sin, n_head, head_dim, scale, doc_start, window):
        b, t, _ = qkv.shape
        a = n_head * head_dim
        # a tensor may begin anywhere in its storage (one sequence of a packed batch); document starts are read one by one
        qkv2 = _aligned(qkv).view(b * t, -1)
        cos, sin = _aligned(cos.float()), _aligned(sin.float())
        ds = doc_start.to(torch.int32).contiguous() if doc_start is not None else None
        dev = qkv2.device
        qk = torch.empty(b * t, 2 * a, dtype=qkv2.dtype, device=dev)
        y = torch.empty(b, t, a, dtype=qkv2.dtype, device=dev)
        lse, counter = _lse_buffer(b, t, n_head, dev)
        L.call("bones_attention_fwd", qkv2.data_ptr(), cos.data_ptr(), sin.data_ptr(), qk.data_ptr(), y.data_ptr(), lse.data_ptr(),
               0 if ds is None else ds.data_ptr(), counter, b, t, n_head, head_dim, scale, window // 128, L.raw_stream(), launches=2)
        ctx.save_for_backward(qkv2, qk, y, lse, cos, sin, ds)
        ctx.meta = (b, t, n_head, head_dim, scale, window)
        return y

    @staticmethod
    def backward(ctx, dy):
        qkv2, qk, y, lse, cos, sin, ds = ctx.saved_tensors
        b, t, n_head, head_dim, scale, window = ctx.meta
        from . import attention_bwd as AB
        dqkv = AB.backward(dy, qkv2, qk, y, lse, cos, sin, ds, b, t, n_head, head_dim, scale, window)
        return dqkv.view(b, t, -1), None, None, None, None, None, None, None


def attention(qkv, cos, sin, n_head, head_dim, scale, doc_start, window):
    return _AttnFn.apply(qkv, cos, sin, n_head, head_dim, scale, doc_start, window)
