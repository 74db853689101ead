"""Native (sm_100a) operator bodies: autograd ``Function``s around the C entry points of ``libbones_b200.so``.

Conventions: activations are bf16, contiguous, flattened to ``[M, C]``; weights are bf16 replicas ``[out, in]``.  A weight
that carries ``main_grad`` (the optimizer's fp32 reduce-scatter slab view) receives its gradient by accumulation inside
the weight-gradient GEMM's epilogue and autograd sees ``None`` for it (reference: dW written straight into the
optimizer's buffer, ``GradFoldIn`` round2/source/train.py:4677-4723 and ``_LinearAccum`` round1/source/train.py:8484).
"""
from __future__ import annotations

import ctypes
import functools
import os

import torch
import torch.nn.functional as F

from . import _lib as L
from . import COUNTS

_I, _L, _F = ctypes.c_int, ctypes.c_longlong, ctypes.c_float
BF16 = torch.bfloat16
_LIBRARY_OPS = os.environ.get("BONES_LIBRARY_OPS", "0") not in ("0", "", "false")


def _c(t):
    return t if t.is_contiguous() else t.contiguous()


def _fused_rows(ws):
    """If the tensors are adjacent row blocks of one storage return a single ``[sum rows, cols]`` view, else None."""
    w0 = ws[0]
    cols = w0.shape[1]
    off = w0.storage_offset()
    for w in ws:
        if (w.dtype != w0.dtype or w.shape[1] != cols or not w.is_contiguous() or w.storage_offset() != off
                or w.untyped_storage().data_ptr() != w0.untyped_storage().data_ptr()):
            return None
        off += w.numel()
    rows = sum(w.shape[0] for w in ws)
    return torch.empty(0, dtype=w0.dtype, device=w0.device).set_(w0.untyped_storage(), w0.storage_offset(), (rows, cols),
                                                                 (cols, 1))


# -- GEMM helpers (2-D, row-major tensors) -----------------------------------------------------------------------
def mm_nt(x, w, out=None, epi=L.EPI_BF16, r=None, alpha=1.0, beta=1.0, out_dtype=BF16):
    """``x [M,K] @ w[N,K]^T``"""
    m, k = x.shape
    n = w.shape[0]
    out = out if out is not None else torch.empty(m, n, dtype=out_dtype, device=x.device)
    L.gemm(x, w, out, m=m, n=n, k=k, lda=x.stride(0), ldb=w.stride(0), ldd=out.stride(0), epi=epi, r=r,
           ldr=r.stride(0) if r is not None else 0, alpha=alpha, beta=beta)
    COUNTS["gemm"] += 1
    return out


def mm_nn(x, w, out=None, epi=L.EPI_BF16, r=None, alpha=1.0, beta=1.0):
    """``x [M,N] @ w[N,K]`` (w row-major: the contraction index is w's row -> MN-major B operand)"""
    m, n = x.shape
    k = w.shape[1]
    out = out if out is not None else torch.empty(m, k, dtype=BF16, device=x.device)
    L.gemm(x, w, out, m=m, n=k, k=n, lda=x.stride(0), ldb=w.stride(0), ldd=out.stride(0), b_major=1, epi=epi, r=r,
           ldr=r.stride(0) if r is not None else 0, alpha=alpha, beta=beta)
    COUNTS["gemm"] += 1
    return out


def mm_nn_acc(x, w, out32):
    """``out32 [M,K] (fp32) += x[M,N] @ w[N,K]``: the fp32 accumulate form lets a long contraction over few output tiles be
    split across the SMs (split-K with vector atomics)"""
    m, n = x.shape
    k = w.shape[1]
    L.gemm(x, w, out32, m=m, n=k, k=n, lda=x.stride(0), ldb=w.stride(0), ldd=out32.stride(0), b_major=1, epi=L.EPI_ACC_F32)
    COUNTS["gemm"] += 1
    return out32


def mm_tn_acc(dy, x, grad, alpha=1.0, push_ptr=None):
    """``grad [N,K] (fp32) += alpha * dy[M,N]^T @ x[M,K]`` (both operands MN-major: contraction over rows).
    ``push_ptr``: device address of the same gradient buffer on the GPU that owns this matrix; the GEMM epilogue then
    adds its tiles there with vector atomics over NVLink, which is the reduce-scatter of the data-parallel gradient done
    tile by tile inside the weight-gradient GEMM."""
    m, n = dy.shape
    k = x.shape[1]
    L.gemm(dy, x, grad, m=n, n=k, k=m, lda=dy.stride(0), ldb=x.stride(0), ldd=grad.stride(0), a_major=1, b_major=1,
           epi=L.EPI_ACC_F32, alpha=alpha, d_ptr=push_ptr, atomic=push_ptr is not None)
    COUNTS["gemm"] += 1
    return grad


def mm_tn(dy, x, out):
    """``out [N,K] (bf16) = dy[M,N]^T @ x[M,K]`` in one piece: the accumulator is rounded once."""
    m, n = dy.shape
    k = x.shape[1]
    L.gemm(dy, x, out, m=n, n=k, k=m, lda=dy.stride(0), ldb=x.stride(0), ldd=out.stride(0), a_major=1, b_major=1)
    COUNTS["gemm"] += 1
    return out


def _wgrad_direct(n, k, m, sms=148):
    """Whether a weight gradient ``[n, k]`` of ``m`` rows that autograd gets back (no slab to accumulate into) is written as bf16 by the
    GEMM.  Accumulating in fp32 lets the GEMM share the contraction out over all ``sms`` SMs, from 32 K blocks of 64 rows on, but costs a
    zero fill, a read-modify-write with atomics and a cast.  us for a K block: 0.27 a wave of single CTAs, 0.31 a wave of pairs, 0.40 for
    each full set of pair tiles where they are shared out; the fp32 route's passes: 9 (5 for one narrow column of tiles) and 1.8 for each million
    weights.  Above 13 000 rows the direct form has gained at most 3 % and lost 8.  Direct / shared, us:
    5120 x 1280 of 1000 rows 17 / 39, 4096 46 / 55, 12288 126 / 131, 16384 179 / 165; 3840 x 1280 (75 tiles, two waves of 74 pairs) of 2048 27 / 40,
    6144 65 / 63, 8192 84 / 74, 12288 122 / 100; 2560 x 1280 (one wave) 8192 45 / 51, 12288 66 / 68; 1280 x 1280 of 2048 15 / 20, 4096 24 / 25,
    6144 34 / 30, 16384 77 / 51; 1024 x 1024 of 2048 16 / 17, 4096 25 / 20; 256 x 256 of 2048 13.6 / 14.1, 3072 18 / 15; 256 x 128 of 2048 13.3 / 11.4."""
    if not 0 < m <= 13312:
        return False
    blocks, tiles, pairs = -(-m // 64), -(-n // 256) * -(-k // 256), sms // 2
    if blocks < 32:
        return True
    waves = min(-(-(-(-n // 128) * -(-k // w)) // sms) for w in (128, 192, 256))          # as bones_gemm_bf16_auto chooses
    direct = 0.27 * waves if waves == 1 or min(n, k) < 256 else 0.31 * -(-tiles // pairs)
    return blocks * (direct - 0.40 * tiles / pairs) <= (9 if k > 128 else 5) + 1.8e-6 * n * k


@functools.lru_cache(maxsize=None)
def _sms(device):
    return torch.cuda.get_device_properties(device).multi_processor_count


def _wgrad(dy2, x2, ws):
    """Weight gradient for one or several row-adjacent weights.  Returns the tuple autograd expects."""
    grads = [getattr(w, "main_grad", None) for w in ws]
    if all(g is not None for g in grads):
        push = [getattr(w, "main_grad_push", None) for w in ws]       # owner-side addresses (fused reduce-scatter)
        fused = _fused_rows(grads) if len(grads) > 1 else grads[0]
        if all(p is not None for p in push):
            # one GEMM when the weights are adjacent in the owner's buffer too (same owner), else one per weight
            adjacent = all(push[j + 1] == push[j] + grads[j].numel() * 4 for j in range(len(ws) - 1))
            if fused is not None and adjacent:
                mm_tn_acc(dy2, x2, fused, push_ptr=push[0])
            else:
                o = 0
                for w, g, pp in zip(ws, grads, push):
                    mm_tn_acc(dy2[:, o:o + w.shape[0]], x2, g, push_ptr=pp)
                    o += w.shape[0]
        elif fused is not None:
            mm_tn_acc(dy2, x2, fused)
        else:
            o = 0
            for w, g in zip(ws, grads):
                mm_tn_acc(dy2[:, o:o + w.shape[0]], x2, g)
                o += w.shape[0]
        return tuple(None for _ in ws)
    if _wgrad_direct(dy2.shape[1], x2.shape[1], dy2.shape[0], _sms(x2.device)) and all(w.dtype == BF16 for w in ws):
        full = torch.empty(dy2.shape[1], x2.shape[1], dtype=BF16, device=x2.device)
        mm_tn(dy2, x2, full)
        if len(ws) == 1:
            return (full,)
        return tuple(g.clone() for g in full.split([w.shape[0] for w in ws]))
    full = torch.zeros(dy2.shape[1], x2.shape[1], dtype=torch.float32, device=x2.device)
    mm_tn_acc(dy2, x2, full)
    outs, o = [], 0
    for w in ws:
        outs.append(full[o:o + w.shape[0]].to(w.dtype))
        o += w.shape[0]
    return tuple(outs)


class _LinearFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, residual, *ws):
        shp = x.shape
        x2 = _c(x).view(-1, shp[-1])
        w = _fused_rows(ws) if len(ws) > 1 else ws[0]
        if w is None:
            w = torch.cat(ws, 0)
        r2 = _c(residual).view(-1, w.shape[0]) if residual is not None else None
        y = mm_nt(x2, w, epi=L.EPI_BF16_RES if r2 is not None else L.EPI_BF16, r=r2)
        ctx.save_for_backward(x2, w)
        ctx.ws, ctx.has_res, ctx.shp = ws, residual is not None, shp
        return y.view(*shp[:-1], w.shape[0])

    @staticmethod
    def backward(ctx, dy):
        x2, w = ctx.saved_tensors
        dy2 = _c(dy).view(-1, w.shape[0])
        dx = mm_nn(dy2, w).view(ctx.shp) if ctx.needs_input_grad[0] else None
        gws = _wgrad(dy2, x2, ctx.ws)
        return (dx, dy if ctx.has_res else None) + gws


def _mx_linear_ok(x, ws):
    return (x.dtype == BF16 and x.shape[-1] % 128 == 0 and all(w.shape[0] % 128 == 0 for w in ws)
            and not any(getattr(w, "main_grad_push", None) is not None for w in ws))


def linear(x, w, residual=None, precision="bf16"):
    if precision == "mxfp8" and _mx_linear_ok(x, (w,)):
        from . import mxfp8
        return mxfp8._MxLinearFn.apply(x, residual, w)
    return _LinearFn.apply(x, residual, w)


def linear_qkv(x, wq, wk, wv, precision="bf16"):
    if precision == "mxfp8" and _mx_linear_ok(x, (wq, wk, wv)):
        from . import mxfp8
        return mxfp8._MxLinearFn.apply(x, None, wq, wk, wv)
    return _LinearFn.apply(x, None, wq, wk, wv)


class _MlpFn(torch.autograd.Function):
    """c_fc GEMM with ReLU^2 epilogue, c_proj GEMM with residual epilogue.  Only ``h = relu(pre)^2`` is kept; the
    backward recovers ``relu(pre) = sqrt(h)`` inside the dX GEMM's epilogue (reference: ``relu2 bwd_from_h``,
    round1/source/train.py:537)."""

    @staticmethod
    def forward(ctx, x, w_fc, w_proj, residual):
        shp = x.shape
        x2 = _c(x).view(-1, shp[-1])
        r2 = _c(residual).view(-1, w_proj.shape[0]) if residual is not None else None
        m, c = x2.shape
        f, n = w_fc.shape[0], w_proj.shape[0]
        h, y = torch.empty(m, f, dtype=BF16, device=x.device), torch.empty(m, n, dtype=BF16, device=x.device)
        L.call("bones_mlp_bf16_fwd", x2.data_ptr(), w_fc.data_ptr(), w_proj.data_ptr(), r2.data_ptr() if r2 is not None else 0, h.data_ptr(), y.data_ptr(),
               m, c, f, n, x2.stride(0), w_fc.stride(0), w_proj.stride(0), r2.stride(0) if r2 is not None else 0, L.GEMM_MODE, L.raw_stream(),
               launches=2)
        COUNTS["gemm"] += 2
        ctx.save_for_backward(x2, h, w_fc, w_proj)
        ctx.has_res, ctx.shp = residual is not None, shp
        ctx.ws = (w_fc, w_proj)
        COUNTS["mlp"] += 1
        return y.view(shp[:-1] + (w_proj.shape[0],))

    @staticmethod
    def backward(ctx, dy):
        x2, h, w_fc, w_proj = ctx.saved_tensors
        dy2 = _c(dy).view(-1, w_proj.shape[0])
        m, c = x2.shape
        f, n = w_fc.shape[0], w_proj.shape[0]
        dpre, dx = torch.empty(m, f, dtype=BF16, device=dy.device), torch.empty(m, c, dtype=BF16, device=dy.device)
        direct = [_wgrad_direct(*s, m, _sms(x2.device)) and w.dtype == BF16 and getattr(w, "main_grad", None) is None for w, s in zip(ctx.ws, ((f, c), (n, f)))]
        g_fc = torch.empty(f, c, dtype=BF16, device=dy.device) if direct[0] else None
        g_proj = torch.empty(n, f, dtype=BF16, device=dy.device) if direct[1] else None
        L.call("bones_mlp_bf16_bwd", dy2.data_ptr(), x2.data_ptr(), h.data_ptr(), w_fc.data_ptr(), w_proj.data_ptr(), dpre.data_ptr(), dx.data_ptr(),
               g_fc.data_ptr() if direct[0] else 0, g_proj.data_ptr() if direct[1] else 0, m, c, f, n, dy2.stride(0), x2.stride(0), w_fc.stride(0),
               w_proj.stride(0), L.GEMM_MODE, L.raw_stream(), launches=2 + sum(direct))
        COUNTS["gemm"] += 2 + sum(direct)
        if not direct[1]:
            (g_proj,) = _wgrad(dy2, h, (ctx.ws[1],))
        if not direct[0]:
            (g_fc,) = _wgrad(dpre, x2, (ctx.ws[0],))
        return dx.view(ctx.shp), g_fc, g_proj, (dy if ctx.has_res else None)


def mlp(x, w_fc, w_proj, residual=None, precision="bf16"):
    if precision == "mxfp8":
        from . import mxfp8
        return mxfp8.mlp(x, w_fc, w_proj, residual)
    return _MlpFn.apply(x, w_fc, w_proj, residual)


# -- norms ---------------------------------------------------------------------------------------------------------
class _RmsNormFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x):
        x2 = _c(x).view(-1, x.shape[-1])
        y = torch.empty_like(x2)
        L.call("bones_rmsnorm_fwd", L.ptr(x2), L.ptr(y), _I(x2.shape[0]), _I(x2.shape[1]), L.stream())
        ctx.save_for_backward(x2)
        COUNTS["rmsnorm"] += 1
        return y.view(x.shape)

    @staticmethod
    def backward(ctx, dy):
        (x2,) = ctx.saved_tensors
        dy2 = _c(dy).view(x2.shape)
        dx = torch.empty_like(x2)
        L.call("bones_rmsnorm_bwd", L.ptr(x2), L.ptr(dy2), L.ptr(None), L.ptr(dx), _I(x2.shape[0]), _I(x2.shape[1]),
               L.stream())
        return dx.view(dy.shape)


def rms_norm(x):
    if x.dtype != BF16:
        from ..ref import functional as RF
        return RF.rms_norm(x)
    if _LIBRARY_OPS:
        from . import registry
        COUNTS["rmsnorm"] += 1
        return registry.rms_norm(x)
    return _RmsNormFn.apply(x)


class _NormSplitFn(torch.autograd.Function):
    """``x -> (x, rms_norm(x))`` for the ``x + f(norm(x))`` pattern: the backward adds the gradient of the pass-through
    copy inside the norm-backward kernel instead of leaving a separate accumulation to autograd."""

    @staticmethod
    def forward(ctx, x):
        x2 = _c(x).view(-1, x.shape[-1])
        y = torch.empty_like(x2)
        L.call("bones_rmsnorm_fwd", L.ptr(x2), L.ptr(y), _I(x2.shape[0]), _I(x2.shape[1]), L.stream())
        ctx.save_for_backward(x2)
        COUNTS["rmsnorm"] += 1
        return x.view(x.shape), y.view(x.shape)

    @staticmethod
    def backward(ctx, dx_pass, dy):
        (x2,) = ctx.saved_tensors
        if dy is None:
            return dx_pass
        dy2 = _c(dy).view(x2.shape)
        add = _c(dx_pass).view(x2.shape) if dx_pass is not None else None
        dx = torch.empty_like(x2)
        L.call("bones_rmsnorm_bwd", L.ptr(x2), L.ptr(dy2), L.ptr(add), L.ptr(dx), _I(x2.shape[0]), _I(x2.shape[1]), L.stream())
        return dx.view(dy.shape)


def norm_split(x):
    if x.dtype != BF16:
        from ..ref import functional as RF
        return x, RF.rms_norm(x)
    return _NormSplitFn.apply(x)


class X0Accum:
    """Shared by the blocks of one forward pass: their backward passes add the gradient of the common ``x0`` operand into
    one buffer inside the kernel, and the first block (the last to run backward) hands the sum to autograd."""

    def __init__(self):
        self.pending = 0
        self.buf = None


class _ResidMixNormFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, x0, a, b, acc=None):
        ctx.acc = acc
        if acc is not None:
            acc.pending += 1
        x2, x02 = _c(x).view(-1, x.shape[-1]), _c(x0).view(-1, x.shape[-1])
        xm, xn = torch.empty_like(x2), torch.empty_like(x2)
        af, bf = a.detach().float().reshape(1), b.detach().float().reshape(1)
        L.call("bones_resid_mix_norm_fwd", L.ptr(x2), L.ptr(x02), L.ptr(af), L.ptr(bf), L.ptr(xm), L.ptr(xn),
               _I(x2.shape[0]), _I(x2.shape[1]), L.stream())
        ctx.save_for_backward(x2, x02, xm, af, bf)
        ctx.shape = x.shape
        COUNTS["resid_mix_norm"] += 1
        return xm.view(x.shape), xn.view(x.shape)

    @staticmethod
    def backward(ctx, dxm, dxn):
        x2, x02, xm, af, bf = ctx.saved_tensors
        if dxm is None:
            dxm = torch.zeros_like(xm)
        if dxn is None:
            dxn = torch.zeros_like(xm)
        dxm2, dxn2 = _c(dxm).view(x2.shape), _c(dxn).view(x2.shape)
        acc = ctx.acc
        dx = torch.empty_like(x2)
        accumulate = acc is not None and acc.buf is not None
        dx0 = acc.buf if accumulate else torch.empty_like(x2)
        dab = torch.zeros(2, dtype=torch.float32, device=x2.device)
        L.call("bones_resid_mix_norm_bwd", L.ptr(x2), L.ptr(x02), L.ptr(xm), L.ptr(af), L.ptr(bf), L.ptr(dxm2),
               L.ptr(dxn2), L.ptr(dx), L.ptr(dx0), L.ptr(dab[0:1]), L.ptr(dab[1:2]), _I(x2.shape[0]), _I(x2.shape[1]),
               _I(int(accumulate)), L.stream())
        if acc is not None:
            acc.buf = dx0
            acc.pending -= 1
            if acc.pending > 0:
                return dx.view(ctx.shape), None, dab[0:1], dab[1:2], None
            acc.buf = None
        return dx.view(ctx.shape), dx0.view(ctx.shape), dab[0:1], dab[1:2], None


def resid_mix_norm(x, x0, a, b, acc=None):
    return _ResidMixNormFn.apply(x, x0, a, b, acc)


# -- embedding -------------------------------------------------------------------------------------------------------
class _EmbeddingFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, idx, weight):
        flat = _c(idx).view(-1)
        out = torch.empty(flat.numel(), weight.shape[1], dtype=weight.dtype, device=weight.device)
        L.call("bones_gather_rows", L.ptr(weight), L.ptr(flat), _I(int(flat.dtype == torch.int64)), L.ptr(out),
               _I(flat.numel()), _I(weight.shape[1]), _L(weight.shape[0]), L.stream())
        ctx.save_for_backward(flat)
        ctx.weight = weight
        COUNTS["embedding"] += 1
        return out.view(*idx.shape, weight.shape[1])

    @staticmethod
    def backward(ctx, dy):
        (flat,) = ctx.saved_tensors
        w = ctx.weight
        grad = getattr(w, "main_grad", None)
        ret = None
        if grad is None:
            grad = torch.zeros(w.shape, dtype=torch.float32, device=w.device)
            ret = grad
        dy2 = _c(dy).view(-1, w.shape[1])
        L.call("bones_scatter_add_rows", L.ptr(dy2), L.ptr(flat), _I(int(flat.dtype == torch.int64)), L.ptr(grad),
               _I(flat.numel()), _I(w.shape[1]), _L(w.shape[0]), L.stream())
        return None, (ret.to(w.dtype) if ret is not None else None)


def embedding(idx, weight, dtype):
    if weight.dtype != BF16:
        return F.embedding(idx, weight).to(dtype)
    return _EmbeddingFn.apply(idx, weight)


# -- attention -------------------------------------------------------------------------------------------------------
def attention(qkv, cos, sin, n_head, head_dim, scale, doc_start, window):
    """RoPE + QK-norm + causal (document-reset, optionally banded) attention on the tcgen05 flash-attention kernels
    (``csrc/attention.cu``, ``csrc/attention_bwd_split.cu``).  A shape the kernels do not cover raises: the SDPA route
    exists only as the explicit baseline (``BONES_KERNELS=ref``), never as a silent fallback (reference: a kernel
    route that does not apply on the device raises, round2/source/train.py:4882-4887)."""
    from . import attention_bwd as AB
    from . import attention_native as AN
    t = qkv.shape[1]
    pad = -t % AB.length_multiple(head_dim)
    if pad:
        # the single-kernel backward (`BONES_ATTN_BWD=fused`) works on whole 128-token tiles: the sequence is zero-padded at
        # the end, which causal masking keeps away from the real positions, and the padding rows are dropped again.  The
        # default kernels take any length (rows past the end are zeros of the tensor maps, and are not stored).
        qkv = F.pad(qkv, (0, 0, 0, pad))
        cos, sin = F.pad(cos, (0, 0, 0, pad)), F.pad(sin, (0, 0, 0, pad))
        if doc_start is not None:
            doc_start = F.pad(doc_start, (0, pad), value=t)
    why = AN.why_not(qkv, n_head, head_dim, window)
    if why:
        raise ValueError(f"native attention does not cover this call: {why}")
    COUNTS["attention"] += 1
    if _LIBRARY_OPS and head_dim == 128:             # the same kernels behind torch.library custom ops (ops/registry.py)
        from . import registry
        y = registry.attention(qkv, cos, sin, n_head, head_dim, scale, doc_start, window)
    else:
        y = AN.attention(qkv, cos, sin, n_head, head_dim, scale, doc_start, window)
    return y[:, :t] if pad else y


# -- loss head -------------------------------------------------------------------------------------------------------
LOSS_ROWS = max(128, int(os.environ.get("BONES_LOSS_ROWS", 4096)))       # rows per logits block


def _logits_stats_ok(x2, w, vocab) -> bool:
    """What the logits GEMM with row statistics covers: bf16, whole 32-column chunks, aligned operands."""
    return (x2.dtype == BF16 and w.dtype == BF16 and w.dim() == 2 and w.stride(1) == 1 and w.shape[0] % 32 == 0 and vocab % 8 == 0 and x2.shape[1] % 8 == 0
            and w.stride(0) % 8 == 0 and w.data_ptr() % 16 == 0 and x2.data_ptr() % 16 == 0 and LOSS_ROWS <= 65535)


def _logits_stats(x2, w, out, vocab, cap, part, targets, z_target):
    """Soft-capped logits into ``out`` (None: not stored) and their rows' partial sums of exponentials into ``part``."""
    L.call("bones_logits_stats", L.ptr(x2), L.ptr(w), L.ptr(out), _I(x2.shape[0]), _I(w.shape[0]), _I(x2.shape[1]), _L(x2.stride(0)), _L(w.stride(0)),
           _L(out.stride(0) if out is not None else 0), _F(cap), _I(vocab), L.ptr(part), L.ptr(targets), L.ptr(z_target), L.stream())
    COUNTS["gemm"] += 1


def _mm_tn_write(dy, x, grad):
    """``grad [N,K] (fp32) = dy[M,N]^T @ x[M,K]``: the first accumulation into a buffer that holds nothing yet"""
    m, n = dy.shape
    k = x.shape[1]
    L.gemm(dy, x, grad, m=n, n=k, k=m, lda=dy.stride(0), ldb=x.stride(0), ldd=grad.stride(0), a_major=1, b_major=1, epi=L.EPI_F32)
    COUNTS["gemm"] += 1


def _by_address(t) -> bool:
    """Whether a kernel can stand in for PyTorch operators on ``t`` inside a backward: it has memory of its own (the batched
    gradients of ``is_grads_batched`` do not) and no graph is being recorded through it (``create_graph``)."""
    if torch.is_grad_enabled() and t.requires_grad:
        return False
    try:
        t.data_ptr()
    except RuntimeError:
        return False
    return True


def _scale_cast(g32, scale, dtype):
    """``g32`` rounded to ``dtype``, times ``scale`` (a device scalar), rounded again."""
    if dtype != BF16 or g32.numel() % 8 or not _by_address(scale):
        return g32.to(dtype) * scale.to(dtype)
    out = torch.empty(g32.shape, dtype=dtype, device=g32.device)
    L.call("bones_scale_cast", L.ptr(g32), L.ptr(_c(scale.float())), L.ptr(out), _L(g32.numel()), L.stream())
    return out


class _LmHeadLossFn(torch.autograd.Function):
    """Chunked head: for each block of rows the logits GEMM, the softcap cross-entropy (which overwrites the logits
    with their gradient), the dX GEMM and the dW GEMM (accumulating into the head's gradient slab) run back to back, so
    only one ``[rows, V]`` block of logits ever exists and no logits are recomputed in backward.  The loss is the mean
    over valid targets divided by ``loss_div`` (reference: ``chunked_loss_mean`` round2/source/train.py:6364-6391 and
    ``loss_scaled`` :11712)."""

    @staticmethod
    def forward(ctx, x, w, targets, vocab, cap, loss_div, row_weights, want_grad, aux=None, label_smoothing=0.0):
        # aux: up to two (targets, absolute row weights) pairs that share the row's soft-max (multi-token prediction)
        shp = x.shape
        x2 = _c(x).view(-1, shp[-1])
        m = x2.shape[0]
        tg = _c(targets).view(-1).to(torch.int64)
        nll = torch.empty(m, dtype=torch.float32, device=x.device)
        n_valid = (tg >= 0).sum().float().reshape(1)
        # dX contracts over the whole vocabulary into few output tiles: accumulated in fp32 so the contraction can be split
        dx32 = torch.zeros(x2.shape, dtype=torch.float32, device=x.device) if want_grad else None
        rw = _c(row_weights).view(-1).float() if row_weights is not None else None
        vp = w.shape[0]
        grad_w = getattr(w, "main_grad", None)
        own_gw, fresh = None, False
        if want_grad and grad_w is None:
            # with so many output tiles the contraction is not split: the first block can write instead of accumulate
            fresh = m > 0 and -(-vp // 256) * -(-w.shape[1] // 256) >= WGRAD_WHOLE_TILES
            own_gw = grad_w = (torch.empty if fresh else torch.zeros)(w.shape, dtype=torch.float32, device=w.device)
        buf = torch.empty(min(LOSS_ROWS, m), vp, dtype=BF16, device=x.device)
        aux = [(_c(t).view(-1).to(torch.int64), _c(wk).view(-1).float()) for t, wk in (aux or [])][:2]
        nll_aux = torch.zeros(m, dtype=torch.float32, device=x.device) if aux else None

        def aux_ptrs(r0, r1):
            out = []
            for k in range(2):
                out += [L.ptr(aux[k][0][r0:r1]), L.ptr(aux[k][1][r0:r1])] if k < len(aux) else [L.ptr(None), L.ptr(None)]
            return out + [L.ptr(nll_aux[r0:r1] if aux else None)]

        # the logits GEMM leaves the rows' sums of exponentials, so the loss kernels pass over the logits once; label smoothing
        # needs their plain sum too and takes the two-pass kernel
        stats = _logits_stats_ok(x2, w, vocab) and label_smoothing == 0.0 and want_grad
        if stats:
            rows, dev = buf.shape[0], x.device
            part = torch.empty(-(-vp // 256) * 2, rows, dtype=torch.float32, device=dev)
            info = torch.empty(rows, 4, dtype=torch.float32, device=dev)
        for r0 in range(0, m, LOSS_ROWS):
            r1 = min(m, r0 + LOSS_ROWS)
            lg = buf[:r1 - r0]
            # the logits GEMM soft-caps in its epilogue (cap * tanh(. / cap)); the loss kernel then only exponentiates
            if stats:
                ap = aux_ptrs(r0, r1)
                _logits_stats(x2[r0:r1], w, lg, vocab, cap, part, None, None)
                L.call("bones_ce_finish", L.ptr(part), _I(part.shape[0]), _I(r1 - r0), L.ptr(lg), _L(vp), L.ptr(None), L.ptr(tg[r0:r1]), _I(vocab),
                       _F(cap), L.ptr(nll[r0:r1]), L.ptr(info), L.ptr(rw[r0:r1] if rw is not None else None), L.ptr(n_valid), _F(1.0 / loss_div),
                       *aux_ptrs(r0, r1), L.stream())
                L.call("bones_ce_grad", L.ptr(lg), _L(vp), L.ptr(info), L.ptr(tg[r0:r1]), ap[0], ap[2], _I(vocab), _F(cap), _I(r1 - r0), L.stream())
            else:
                mm_nt(x2[r0:r1], w, out=lg, epi=L.EPI_SOFTCAP, alpha=1.0 / cap, beta=cap)
                L.call("bones_softcap_ce", L.ptr(lg), _L(vp), L.ptr(tg[r0:r1]), _I(vocab), _F(cap), L.ptr(nll[r0:r1]),
                       L.ptr(lg if want_grad else None), L.ptr(rw[r0:r1] if rw is not None else None), L.ptr(n_valid),
                       _F(1.0 / loss_div), _I(r1 - r0), _I(1), *aux_ptrs(r0, r1), _F(label_smoothing), L.stream())
            if want_grad:
                mm_nn_acc(lg, w, dx32[r0:r1])
                if fresh and r0 == 0:
                    _mm_tn_write(lg, x2[r0:r1], grad_w)
                else:
                    mm_tn_acc(lg, x2[r0:r1], grad_w)
        COUNTS["lmhead_loss"] += 1
        ctx.dx, ctx.shp, ctx.own_gw, ctx.xdtype, ctx.wdtype = dx32, shp, own_gw, x2.dtype, w.dtype
        if rw is not None:
            loss = (nll * rw).sum()
        else:
            loss = nll.sum() / n_valid.clamp_min(1.0)[0] / loss_div
        if aux:
            loss = loss + nll_aux.sum()
        ctx.mark_non_differentiable(nll)
        return loss, nll

    @staticmethod
    def backward(ctx, dloss, _dnll):
        dx = _scale_cast(ctx.dx, dloss, ctx.xdtype).view(ctx.shp)
        gw = _scale_cast(ctx.own_gw, dloss, ctx.wdtype) if ctx.own_gw is not None else None
        return dx, gw, None, None, None, None, None, None, None, None


@torch.no_grad()
def _lmhead_nll(x, w, targets, vocab, cap):
    """Per-row negative log-likelihoods (0 where the target is masked); the logits never leave the GEMM."""
    x2 = _c(x).view(-1, x.shape[-1])
    m = x2.shape[0]
    tg = _c(targets).view(-1).to(torch.int64)
    nll, z = torch.empty(m, dtype=torch.float32, device=x.device), torch.empty(m, dtype=torch.float32, device=x.device)
    # the partial sums are 2 KB a row at 65536 columns: in blocks of rows, as the logits of a training step are
    part = torch.empty(-(-w.shape[0] // 256) * 2 * min(LOSS_ROWS, m), dtype=torch.float32, device=x.device)
    null = L.ptr(None)
    for r0 in range(0, m, LOSS_ROWS):
        r1 = min(m, r0 + LOSS_ROWS)
        _logits_stats(x2[r0:r1], w, None, vocab, cap, part, tg[r0:r1], z[r0:r1])
        L.call("bones_ce_finish", L.ptr(part), _I(-(-w.shape[0] // 256) * 2), _I(r1 - r0), null, _L(0), L.ptr(z[r0:r1]), L.ptr(tg[r0:r1]), _I(vocab),
               _F(cap), L.ptr(nll[r0:r1]), null, null, null, _F(1.0), null, null, null, null, null, L.stream())
    COUNTS["lmhead_loss"] += 1
    return nll


def lmhead_loss(x, w, targets, vocab, cap, reduction="mean", row_weights=None, loss_div=1.0, aux=None, label_smoothing=0.0):
    if reduction != "mean" and not aux and label_smoothing == 0.0 and 0 < x.numel() and _logits_stats_ok(_c(x).view(-1, x.shape[-1]), w, vocab):
        nll = _lmhead_nll(x, w, targets, vocab, cap)
        return nll.sum() if reduction == "sum" else nll.view(targets.shape)
    want_grad = torch.is_grad_enabled() and (x.requires_grad or w.requires_grad) and reduction == "mean"
    loss, nll = _LmHeadLossFn.apply(x, w, targets, vocab, cap, float(loss_div), row_weights, want_grad, aux,
                                    float(label_smoothing))
    if reduction == "mean":
        return loss
    if reduction == "sum":
        return nll.sum()
    return nll.view(targets.shape)


def lmhead_logits(x, w, vocab, cap):
    shp = x.shape
    x2 = _c(x).view(-1, shp[-1])
    lg = mm_nt(x2, w)
    out = torch.empty(x2.shape[0], vocab, dtype=torch.float32, device=x.device)
    L.call("bones_softcap_logits", L.ptr(lg), _L(w.shape[0]), L.ptr(out), _I(vocab), _F(cap), _L(x2.shape[0]), L.stream())
    return out.view(*shp[:-1], vocab)


# -- output-side hashed table ----------------------------------------------------------------------------------------
def os1_apply_signs(x, hsign, out_dtype=None):
    """``signs(hsign) * x`` for rows ``x [n, dim]`` (bf16 or fp32) and sign hashes ``hsign [n]`` int64."""
    x = _c(x)
    out_dtype = out_dtype or x.dtype
    kind = {(BF16, BF16): 0, (torch.float32, torch.float32): 1, (torch.float32, BF16): 2}[(x.dtype, out_dtype)]
    out = torch.empty(x.shape, dtype=out_dtype, device=x.device)
    L.call("bones_os1_signs", L.ptr(x), L.ptr(_c(hsign)), L.ptr(out), _L(x.shape[0]), _I(x.shape[1]), _I(kind), L.stream())
    return out


def os1_gate_dot(u, code, nxt, a0):
    """``sd[i] = u[i] . code[nxt[i]] / a0`` (0 where ``nxt[i] < 0``), fp32."""
    sd = torch.empty(u.shape[0], dtype=torch.float32, device=u.device)
    L.call("bones_os1_gate_dot", L.ptr(_c(u)), L.ptr(code), L.ptr(_c(nxt)), L.ptr(sd), _L(u.shape[0]), _I(u.shape[1]),
           _F(1.0 / a0), L.stream())
    return sd


def os1_row_step(table, rows, g, lr, eps, cap):
    """In place on ``table[rows]``: the normalised step and the row budget.  Returns the count of rows the budget scaled
    (a device int32 scalar)."""
    capped = torch.zeros(1, dtype=torch.int32, device=table.device)
    L.call("bones_os1_row_step", L.ptr(table), L.ptr(_c(rows)), L.ptr(_c(g)), _I(rows.numel()), _I(table.shape[1]), _F(lr),
           _F(eps), _F(cap * lr), L.ptr(capped), _I(int(table.dtype == torch.float32)), L.stream())
    return capped


class _LmHeadLossOs1Fn(torch.autograd.Function):
    """The chunked loss head with the output table's read-out: per block of rows the logits GEMM, the scores GEMM
    ``S = U C^T / a0``, one element-wise kernel that adds ``glin S + G k relu(S - thr)`` and soft-caps, the
    cross-entropy kernel (logits overwritten by their gradient), then dX, dW and ``dU = (glin / a0) dLogits C``
    (reference: the OS1-fused loss-head pair, round2/source/train.py:5881-5957 and :6461-6501)."""

    @staticmethod
    def forward(ctx, x, w, u, code, gate, targets, vocab, cap, loss_div, row_weights, want_grad, a0, glin, kthr, thr):
        shp = x.shape
        x2 = _c(x).view(-1, shp[-1])
        u2 = _c(u).view(-1, u.shape[-1])
        m = x2.shape[0]
        tg = _c(targets).view(-1).to(torch.int64)
        gt = _c(gate).view(-1).float()
        nll = torch.empty(m, dtype=torch.float32, device=x.device)
        n_valid = (tg >= 0).sum().float().reshape(1)
        dx32 = torch.zeros(x2.shape, dtype=torch.float32, device=x.device) if want_grad else None
        du32 = torch.zeros(u2.shape, dtype=torch.float32, device=x.device) if want_grad else None
        rw = _c(row_weights).view(-1).float() if row_weights is not None else None
        vp = w.shape[0]
        grad_w = getattr(w, "main_grad", None)
        own_gw = None
        if want_grad and grad_w is None:
            own_gw = grad_w = torch.zeros(w.shape, dtype=torch.float32, device=w.device)
        rows = min(LOSS_ROWS, m)
        buf = torch.empty(rows, vp, dtype=BF16, device=x.device)
        sbuf = torch.empty(rows, vp, dtype=BF16, device=x.device)
        null = L.ptr(None)
        for r0 in range(0, m, LOSS_ROWS):
            r1 = min(m, r0 + LOSS_ROWS)
            lg, sc = buf[:r1 - r0], sbuf[:r1 - r0]
            mm_nt(x2[r0:r1], w, out=lg)
            mm_nt(u2[r0:r1], code, out=sc, alpha=1.0 / a0)
            L.call("bones_os1_combine", L.ptr(lg), L.ptr(sc), L.ptr(gt[r0:r1]), _L(r1 - r0), _I(vp), _L(vp), _F(cap), _F(glin),
                   _F(kthr), _F(thr), _I(1), L.stream())
            L.call("bones_softcap_ce", L.ptr(lg), _L(vp), L.ptr(tg[r0:r1]), _I(vocab), _F(cap), L.ptr(nll[r0:r1]),
                   L.ptr(lg if want_grad else None), L.ptr(rw[r0:r1] if rw is not None else None), L.ptr(n_valid),
                   _F(1.0 / loss_div), _I(r1 - r0), _I(1), null, null, null, null, null, _F(0.0), L.stream())
            if want_grad:
                mm_nn_acc(lg, w, dx32[r0:r1])
                mm_tn_acc(lg, x2[r0:r1], grad_w)
                mm_nn_acc(lg, code, du32[r0:r1])
        COUNTS["lmhead_loss_os1"] += 1
        ctx.dx = dx32.to(x2.dtype) if want_grad else None
        ctx.du = (du32 * (glin / a0)) if want_grad else None
        ctx.shp, ctx.ushp, ctx.own_gw, ctx.wdtype, ctx.udtype = shp, u.shape, own_gw, w.dtype, u.dtype
        if rw is not None:
            loss = (nll * rw).sum()
        else:
            loss = nll.sum() / n_valid.clamp_min(1.0)[0] / loss_div
        ctx.mark_non_differentiable(nll)
        return loss, nll

    @staticmethod
    def backward(ctx, dloss, _dnll):
        dx = ctx.dx.view(ctx.shp) * dloss.to(ctx.dx.dtype)
        du = (ctx.du.view(ctx.ushp) * dloss.float()).to(ctx.udtype)
        gw = ctx.own_gw.to(ctx.wdtype) * dloss.to(ctx.wdtype) if ctx.own_gw is not None else None
        return (dx, gw, du) + (None,) * 12


def lmhead_loss_os1(x, w, targets, vocab, cap, u, code, gate, a0, glin, beta, thr, reduction="mean", row_weights=None,
                    loss_div=1.0):
    want_grad = torch.is_grad_enabled() and (x.requires_grad or w.requires_grad or u.requires_grad) and reduction == "mean"
    loss, nll = _LmHeadLossOs1Fn.apply(x, w, u, code, gate, targets, vocab, cap, float(loss_div), row_weights, want_grad,
                                       float(a0), float(glin), float(beta / (1.0 - thr)), float(thr))
    if reduction == "mean":
        return loss
    if reduction == "sum":
        return nll.sum()
    return nll.view(targets.shape)


def lmhead_logits_os1(x, w, vocab, cap, u, code, gate, a0, glin, beta, thr):
    shp = x.shape
    x2 = _c(x).view(-1, shp[-1])
    u2 = _c(u).view(-1, u.shape[-1])
    vp = w.shape[0]
    lg = mm_nt(x2, w)
    sc = mm_nt(u2, code, alpha=1.0 / a0)
    L.call("bones_os1_combine", L.ptr(lg), L.ptr(sc), L.ptr(_c(gate).view(-1).float()), _L(x2.shape[0]), _I(vp), _L(vp),
           _F(cap), _F(glin), _F(beta / (1.0 - thr)), _F(thr), _I(0), L.stream())
    out = torch.empty(x2.shape[0], vocab, dtype=torch.float32, device=x.device)
    L.call("bones_softcap_logits", L.ptr(lg), _L(vp), L.ptr(out), _I(vocab), _F(cap), _L(x2.shape[0]), L.stream())
    return out.view(*shp[:-1], vocab)


# -- MoE -------------------------------------------------------------------------------------------------------------
class _RouterFn(torch.autograd.Function):
    """Router logits ``h [T, C] @ R[E, C]^T`` in fp32 on the tcgen05 GEMM.  ``E`` (16) is far below a tensor-core tile, so
    the router is padded to 128 rows: the padding costs a few GFLOP, while the library route this replaces converted the
    whole activation to fp32 and ran SIMT fp32 GEMMs (a fifth of an MoE layer's non-GEMM time).  Inputs are the exact
    bf16 values and the accumulation is fp32, which is what ``F.linear(h.float(), R.float())`` computes (reference: the
    fp32 router, round2/source/train.py:11023)."""

    @staticmethod
    def forward(ctx, h, router):
        e, c = router.shape
        rp = torch.zeros(128, c, dtype=BF16, device=h.device)
        rp[:e].copy_(router.detach())
        out = mm_nt(h, rp, epi=L.EPI_F32, out_dtype=torch.float32)
        ctx.save_for_backward(h, rp)
        ctx.e, ctx.rdtype = e, router.dtype
        COUNTS["moe_router"] += 1
        return out[:, :e].contiguous()

    @staticmethod
    def backward(ctx, dl):
        h, rp = ctx.saved_tensors
        t, c = h.shape
        dlp = torch.zeros(t, 128, dtype=BF16, device=h.device)
        dlp[:, :ctx.e].copy_(dl)
        dh = mm_nn(dlp, rp)
        dr32 = torch.zeros(128, c, dtype=torch.float32, device=h.device)
        mm_tn_acc(dlp, h, dr32)
        return dh, dr32[:ctx.e].to(ctx.rdtype)


def router_logits(h, router):
    if h.dtype != BF16 or router.shape[0] > 128 or h.shape[1] % 8:
        return F.linear(h.float(), router.float())
    return _RouterFn.apply(_c(h), router)


class _MoeRouterFn(torch.autograd.Function):
    """The whole router: logits on the padded tensor-core GEMM (as in ``_RouterFn``), then one kernel for soft-max, top-k choice,
    gates and the statistics of the auxiliary loss; backward one kernel that writes the padded bf16 logit gradient both
    gradient GEMMs read (``csrc/router.cu``)."""

    @staticmethod
    def forward(ctx, h, router, topk, aux_w, z_w, want_aux):
        e, c = router.shape
        n, dev = h.shape[0], h.device
        rp = torch.zeros(128, c, dtype=BF16, device=dev)
        rp[:e].copy_(router.detach())
        logits = mm_nt(h, rp, epi=L.EPI_F32, out_dtype=torch.float32)
        idx = torch.empty(n, topk, dtype=torch.int64, device=dev)
        gates = torch.empty(n, topk, dtype=torch.float32, device=dev)
        aux = torch.empty((), dtype=torch.float32, device=dev) if want_aux else None
        stats = torch.empty(2 + e, dtype=torch.float32, device=dev) if want_aux else None
        part = torch.empty(-(-n // 128) * (2 * e + 1), dtype=torch.float32, device=dev) if want_aux else None
        L.call("bones_moe_route_fwd", L.ptr(logits), _L(128), _L(n), _I(e), _I(topk), L.ptr(idx), L.ptr(gates), L.ptr(part), _F(aux_w), _F(z_w),
               L.ptr(aux), L.ptr(stats), L.stream(), launches=2 if want_aux else 1)
        ctx.save_for_backward(h, rp, logits, idx, stats)
        ctx.meta, ctx.rdtype = (e, topk, aux_w, z_w), router.dtype
        ctx.set_materialize_grads(False)
        ctx.mark_non_differentiable(*([idx, stats] if want_aux else [idx]))
        COUNTS["moe_router"] += 1
        return idx, gates, aux, stats

    @staticmethod
    def backward(ctx, _didx, dgates, daux, _dstats):
        h, rp, logits, idx, stats = ctx.saved_tensors
        e, topk, aux_w, z_w = ctx.meta
        n, c = h.shape
        dlp = torch.empty(n, 128, dtype=BF16, device=h.device)
        dgates = _c(dgates.float()) if dgates is not None else None
        daux = _c(daux.float()) if daux is not None else None
        f = ctypes.c_void_p(stats.data_ptr() + 8) if stats is not None else L.ptr(None)
        L.call("bones_moe_route_bwd", L.ptr(logits), _L(128), _L(n), _I(e), _I(topk), L.ptr(idx), L.ptr(dgates), L.ptr(daux), f, _F(aux_w), _F(z_w),
               L.ptr(dlp), L.stream())
        dh = mm_nn(dlp, rp) if ctx.needs_input_grad[0] else None
        dr = None
        if ctx.needs_input_grad[1]:
            dr32 = torch.zeros(128, c, dtype=torch.float32, device=h.device)
            mm_tn_acc(dlp, h, dr32)
            dr = dr32[:e].to(ctx.rdtype)
        return dh, dr, None, None, None, None


def moe_router_ok(h, router, topk):
    """The fused router covers bf16 activations, up to 64 experts, one or two different choices and the GEMM's 16-byte rows."""
    return h.dtype == BF16 and router.shape[0] <= 64 and h.shape[1] % 8 == 0 and topk in (1, 2) and topk <= router.shape[0] and h.shape[0] > 0


def moe_router(h, router, topk, aux_w, z_w, want_aux):
    return _MoeRouterFn.apply(_c(h), router, topk, float(aux_w), float(z_w), want_aux)


def moe_slots(idx, b, t, n_exp, cap):
    """Native capacity slotting: ``idx [b*t, k]`` int64 -> ``(slot [b*t, k], tok [E*b*cap])``."""
    n, k = idx.shape
    idx = _c(idx)
    slot = torch.empty(n, k, dtype=torch.int64, device=idx.device)
    tok = torch.empty(n_exp * b * cap, dtype=torch.int64, device=idx.device)
    L.call("bones_moe_slots", L.ptr(idx), L.ptr(slot), L.ptr(tok), _I(b), _I(t), _I(k), _I(n_exp), _I(cap), L.stream())
    COUNTS["moe_slots"] += 1
    return slot, tok


class _DispatchFn(torch.autograd.Function):
    """Forward: slot gather.  Backward: every token sums the gradients of its (at most k) slots -- the combine kernel
    with unit gates -- so both directions are gathers (reference: ``MoeGatherRows``, round2/source/train.py:10637)."""

    @staticmethod
    def forward(ctx, h, tok, slot):
        out = torch.empty(tok.numel(), h.shape[1], dtype=h.dtype, device=h.device)
        L.call("bones_gather_rows", L.ptr(h), L.ptr(tok), _I(1), L.ptr(out), _I(tok.numel()), _I(h.shape[1]),
               _L(h.shape[0]), L.stream())
        ctx.save_for_backward(tok, slot if slot is not None else tok)
        ctx.n, ctx.has_slot = h.shape[0], slot is not None
        COUNTS["moe_dispatch"] += 1
        return out

    @staticmethod
    def backward(ctx, dxs):
        tok, slot = ctx.saved_tensors
        dxs = _c(dxs)
        if ctx.has_slot:
            dh = torch.empty(ctx.n, dxs.shape[1], dtype=dxs.dtype, device=dxs.device)
            L.call("bones_moe_combine", L.ptr(dxs), L.ptr(slot), L.ptr(None), L.ptr(None), L.ptr(dh), _I(ctx.n), _I(dxs.shape[1]),
                   _I(slot.shape[1]), _L(dxs.shape[0]), L.stream())
            return dh, None, None
        g = torch.zeros(ctx.n, dxs.shape[1], dtype=torch.float32, device=dxs.device)
        L.call("bones_scatter_add_rows", L.ptr(dxs), L.ptr(tok), _I(1), L.ptr(g), _I(tok.numel()), _I(dxs.shape[1]),
               _L(ctx.n), L.stream())
        return g.to(dxs.dtype), None, None


def moe_dispatch(h, tok, slot=None):
    return _DispatchFn.apply(_c(h), _c(tok), _c(slot) if slot is not None else None)


class _CombineFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, ys, slot, gates, residual, tok):
        n, k = slot.shape
        out = torch.empty(n, ys.shape[1], dtype=ys.dtype, device=ys.device)
        g32 = _c(gates.float())
        L.call("bones_moe_combine", L.ptr(ys), L.ptr(slot), L.ptr(g32), L.ptr(residual), L.ptr(out), _I(n), _I(ys.shape[1]), _I(k),
               _L(ys.shape[0]), L.stream())
        ctx.save_for_backward(ys, slot, g32, tok)
        ctx.has_res = residual is not None
        COUNTS["moe_combine"] += 1
        return out

    @staticmethod
    def backward(ctx, dout):
        if not (ctx.needs_input_grad[0] or ctx.needs_input_grad[2]):         # the residual's alone: an addition's
            return None, None, None, dout, None
        ys, slot, g32, tok = ctx.saved_tensors
        residual_grad = dout if ctx.has_res else None
        n_slots = ys.shape[0]
        s = torch.where((slot < 0) | (slot > n_slots), n_slots, slot) if tok is None or not _by_address(dout) else None
        if tok is None:              # the token in each slot, where the caller did not have it
            tok = torch.full((n_slots + 1,), slot.shape[0], dtype=torch.int64, device=ys.device)
            tok.scatter_(0, s.view(-1), torch.arange(slot.shape[0], device=ys.device).repeat_interleave(slot.shape[1]))
        if not _by_address(dout):    # what is wanted of it is not known here: perhaps only the residual's, an addition's
            yp = torch.cat([ys, ys.new_zeros(1, ys.shape[1])]).float()
            d = dout.float()
            dg = torch.stack([(yp.index_select(0, s[:, k]) * d).sum(-1) for k in range(s.shape[1])], -1) if s.shape[1] else None
            gate = torch.zeros(n_slots + 1, device=ys.device).scatter_(0, s.view(-1), g32.view(-1))[:n_slots, None]
            used = torch.zeros(n_slots + 1, dtype=torch.bool, device=ys.device).scatter_(0, s.view(-1), True)[:n_slots, None]
            rows = d.index_select(0, tok[:n_slots].clamp(0, slot.shape[0] - 1))
            return torch.where(used, gate * rows, 0.0).to(ys.dtype), None, dg, residual_grad, None
        dout = _c(dout)
        dys = torch.empty_like(ys)
        dg = torch.zeros_like(g32)
        L.call("bones_moe_combine_bwd", L.ptr(ys), L.ptr(slot), L.ptr(g32), L.ptr(tok), L.ptr(dout), L.ptr(dys), L.ptr(dg), _I(slot.shape[0]),
               _I(ys.shape[1]), _I(slot.shape[1]), _L(ys.shape[0]), L.stream())
        return dys, None, dg, residual_grad, None


def moe_combine(ys, slot, gates, residual=None, tok=None):
    if residual is not None and (residual.dtype != ys.dtype or residual.data_ptr() % 16):
        return _CombineFn.apply(_c(ys), _c(slot), gates, None, tok) + residual
    return _CombineFn.apply(_c(ys), _c(slot), gates, _c(residual) if residual is not None else None, tok)


# A weight gradient of the experts, or of the loss head, that autograd gets back (no slab to accumulate into, as the trainer has) is
# written whole by the GEMM once it has so many 256 x 256 tiles that accumulating would not split its contraction either (4 x 74 CTA
# pairs, the GEMM's own rule): experts in bf16, the same accumulator rounded once, without the fp32 zero fill, the read-modify-write
# and the cast; the head's first block of rows in fp32, without the zero fill.  For 16 experts of 2560 x 1280 a layer spent 400 us on
# them (4 plain GEMMs 731 -> 479 us, fills and casts 158 us less).
WGRAD_WHOLE_TILES = 296


class _ExpertsFn(torch.autograd.Function):
    """Local experts as one batched GEMM pair over ``[E_local, rows, d]`` (grouped by expert)."""

    @staticmethod
    def forward(ctx, xs, w_fc, w_proj):
        e, hdim, d = w_fc.shape
        x3 = _c(xs).view(e, -1, d)
        rows = x3.shape[1]
        h = torch.empty(e, rows, hdim, dtype=BF16, device=xs.device)
        L.gemm(x3, w_fc, h, m=rows, n=hdim, k=d, lda=d, ldb=d, ldd=hdim, epi=L.EPI_RELU2, batch=e, stride_a=rows * d,
               stride_b=hdim * d, stride_d=rows * hdim)
        y = torch.empty(e, rows, d, dtype=BF16, device=xs.device)
        L.gemm(h, w_proj, y, m=rows, n=d, k=hdim, lda=hdim, ldb=hdim, ldd=d, batch=e, stride_a=rows * hdim,
               stride_b=d * hdim, stride_d=rows * d)
        ctx.save_for_backward(x3, h, w_fc, w_proj)
        ctx.ws = (w_fc, w_proj)
        COUNTS["moe_experts"] += 1
        return y.view(xs.shape)

    @staticmethod
    def backward(ctx, dy):
        x3, h, w_fc, w_proj = ctx.saved_tensors
        e, hdim, d = w_fc.shape
        rows = x3.shape[1]
        dy3 = _c(dy).view(e, rows, d)
        dpre = torch.empty(e, rows, hdim, dtype=BF16, device=dy.device)
        L.gemm(dy3, w_proj, dpre, m=rows, n=hdim, k=d, lda=d, ldb=hdim, ldd=hdim, b_major=1, epi=L.EPI_MUL_2SQRT, r=h,
               ldr=hdim, batch=e, stride_a=rows * d, stride_b=d * hdim, stride_d=rows * hdim, stride_r=rows * hdim)
        dx = torch.empty(e, rows, d, dtype=BF16, device=dy.device)
        L.gemm(dpre, w_fc, dx, m=rows, n=d, k=hdim, lda=hdim, ldb=d, ldd=d, b_major=1, batch=e, stride_a=rows * hdim,
               stride_b=hdim * d, stride_d=rows * d)
        outs = []
        for w, a, b in ((ctx.ws[0], dpre, x3), (ctx.ws[1], dy3, h)):
            g = getattr(w, "main_grad", None)
            n_out, n_in = w.shape[1], w.shape[2]
            if g is None and w.dtype == BF16 and e * -(-n_out // 256) * -(-n_in // 256) >= WGRAD_WHOLE_TILES:
                ret = torch.empty(w.shape, dtype=BF16, device=w.device)
                L.gemm(a, b, ret, m=n_out, n=n_in, k=rows, lda=n_out, ldb=n_in, ldd=n_in, a_major=1, b_major=1, batch=e,
                       stride_a=rows * n_out, stride_b=rows * n_in, stride_d=n_out * n_in)
                outs.append(ret)
                continue
            ret = None
            if g is None:
                g = ret = torch.zeros(w.shape, dtype=torch.float32, device=w.device)
            L.gemm(a, b, g, m=n_out, n=n_in, k=rows, lda=n_out, ldb=n_in, ldd=n_in, a_major=1, b_major=1,
                   epi=L.EPI_ACC_F32, batch=e, stride_a=rows * n_out, stride_b=rows * n_in, stride_d=n_out * n_in)
            outs.append(ret.to(w.dtype) if ret is not None else None)
        COUNTS["gemm"] += 4
        return dx.view(dy.shape), outs[0], outs[1]


def moe_experts(xs, w_fc, w_proj, precision="bf16"):
    if precision == "mxfp8":
        from . import mxfp8
        if mxfp8.experts_apply(xs, w_fc, w_proj):
            return mxfp8._MxExpertsFn.apply(xs, w_fc, w_proj)
    return _ExpertsFn.apply(xs, w_fc, w_proj)


# -- tables ----------------------------------------------------------------------------------------------------------
def sparse_adam_rows(table, rows, g, m, v, step, lr, beta1, beta2, eps, decay):
    if table.dtype != BF16:
        raise RuntimeError("native sparse Adam expects a bf16 table")
    L.call("bones_sparse_adam", L.ptr(table), L.ptr(_c(rows)), L.ptr(_c(g)), L.ptr(m), L.ptr(v), _I(rows.numel()),
           _I(table.shape[1]), _F(lr), _F(beta1), _F(beta2), _F(eps), _F(decay), _I(step), L.stream())
    COUNTS["sparse_adam"] += 1
