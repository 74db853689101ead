"""Backward of the native attention: statistics pre-pass, tcgen05 backward kernels, RoPE/QK-norm backward."""
from __future__ import annotations

import ctypes
import os

import torch

from . import COUNTS
from . import _lib as L

_I, _L, _F = ctypes.c_int, ctypes.c_longlong, ctypes.c_float
# split: two kernels (dK/dV, then dQ), every accumulator and every intermediate in TMEM, bf16 outputs;
# fused: one kernel with dQ through fp32 atomics
_IMPL = os.environ.get("BONES_ATTN_BWD", "split")


# The dK / dV kernel leaves dS for the dQ kernel (32 KB per pair of 128-token tiles) while that scratch stays below this, 2 % of the
# device, and can be had; otherwise the dQ kernel computes S, P and dP again, which gives the same bits.  It is given back when the
# call returns.  With it the two kernels take 398 instead of 486 us at 16 x 2048 tokens, 10 heads of 128 (0.71 GB); the gain per pair
# does not depend on the size.
DS_LIMIT = 4 << 30


def ds_tiles(t: int, window: int) -> int:
    """Tile pairs of a (sequence, head) that causality and the band allow."""
    n, w = -(-t // 128), window // 128
    return n * (n + 1) // 2 if w <= 0 or n <= w else w * (w + 1) // 2 + (n - w) * w


# From this size on the scratch is the largest allocation of the call (dqkv takes a third of it at 2048 tokens), and whether it
# fits is looked up first: an allocation that fails makes the allocator give back all it has cached, layer after layer on a device
# that is nearly full.  The allocator's own figures, about 60 us of host time, leave DS_OTHERS for what it does not know of.  Asking the
# driver (cudaMemGetInfo) takes as long on a quiet machine and took milliseconds on a busy one.
DS_ASK = 256 << 20
DS_OTHERS = 2 << 30


def _fits(nbytes, device) -> bool:
    if torch.cuda.is_current_stream_capturing():         # a graph's memory comes from its own pool
        return True
    stats = torch.cuda.memory_stats(device)
    reserved = stats["reserved_bytes.all.current"]
    cached, unused = reserved - stats["allocated_bytes.all.current"], torch.cuda.get_device_properties(device).total_memory - reserved
    return nbytes <= max(cached, unused - DS_OTHERS)


def _ds_scratch(nbytes, device):
    if nbytes > DS_LIMIT or nbytes >= DS_ASK and not _fits(nbytes, device):
        return None
    try:
        return torch.empty(nbytes, dtype=torch.uint8, device=device)
    except torch.OutOfMemoryError:               # the other route needs none
        return None


def _aligned(x):
    """Contiguous and 16-byte aligned (what the kernels' tensor maps and vector loads need)."""
    x = x if x.is_contiguous() else x.contiguous()
    return x if x.data_ptr() % 16 == 0 else x.clone()


def length_multiple(head_dim: int) -> int:
    """The sequence length has to be a multiple of this: the split kernels take any length, the fused one whole tiles."""
    return 128 if _IMPL == "fused" and head_dim == 128 else 1


def backward(dy, qkv2, qk, y, lse, cos, sin, ds, b, t, n_head, head_dim, scale, window):
    m, a = b * t, n_head * head_dim
    dev = dy.device
    dy2 = _aligned(dy).view(m, a)
    dqkv = torch.empty(m, 3 * a, dtype=torch.bfloat16, device=dev)
    if _IMPL != "fused" or head_dim != 128:
        # statistics of whole 128-query tiles, and behind them the two kernels' work-item counters
        n = b * n_head * (-(-t // 128) * 128) * 2
        stats = torch.empty(n + 2, dtype=torch.float32, device=dev)
        dqk = torch.empty(m, 2 * a, dtype=torch.bfloat16, device=dev)
        scratch = _ds_scratch(b * n_head * ds_tiles(t, window) * 32768, dev)
        COUNTS["attention_dq_again" if scratch is None else "attention_dq_stored"] += 1
        # dV goes straight into its third of dqkv, rows 3a apart
        L.call("bones_attention_bwd", dy2.data_ptr(), qkv2.data_ptr(), qk.data_ptr(), y.data_ptr(), lse.data_ptr(), cos.data_ptr(), sin.data_ptr(),
               0 if ds is None else ds.data_ptr(), stats.data_ptr(), stats.data_ptr() + 4 * n, 0 if scratch is None else scratch.data_ptr(), dqk.data_ptr(),
               dqkv.data_ptr(), b, t, n_head, head_dim, scale, window // 128, L.raw_stream(), launches=4)
        return dqkv
    delta = torch.empty(b, n_head, t, dtype=torch.float32, device=dev)
    L.call("bones_attn_delta", L.ptr(dy2), L.ptr(y), L.ptr(delta), _L(m), _I(t), _I(n_head), L.stream())
    dqk = torch.empty(m, 2 * a, dtype=torch.float32, device=dev)
    dv = torch.empty(m, a, dtype=torch.bfloat16, device=dev)
    L.call("bones_attn_bwd", L.ptr(qk), L.ptr(qkv2), L.ptr(dy2), L.ptr(lse), L.ptr(delta), L.ptr(dqk), L.ptr(dv), L.ptr(ds),
           _I(b), _I(t), _I(n_head), _F(scale), _I(window // 128), L.stream())
    L.call("bones_rope_qknorm_bwd", L.ptr(qkv2), L.ptr(cos), L.ptr(sin), L.ptr(dqk), L.ptr(dv), L.ptr(dqkv), _L(m), _I(t),
           _I(n_head), _I(head_dim), L.stream())
    return dqkv
