"""Greedy decoding with a KV cache.

The reference scores teacher-forced full sequences only (round2/submission/inference.py:26-27); autoregressive decoding
is an added capability.  The cache stores, per layer, keys *after* RoPE and QK-norm and raw values, so a decode step
rotates only the new token (RoPE at its absolute position) and attends over the cached prefix restricted to the current
document and the layer's window.
"""
from __future__ import annotations

import ctypes

import torch
import torch.nn.functional as F

from .. import ops
from ..models.moe import MoeMLP
from ..ref import functional as RF

_I = ctypes.c_int


def L_check():
    from ..ops import _lib as L
    L.check_error_word()


class KVCache:
    def __init__(self, model, batch: int, max_len: int):
        cfg = model.config
        dev, dt = model.lm_head.weight.device, model.lm_head.weight.dtype
        shape = (cfg.n_layer, batch, max_len, cfg.n_head, cfg.head_dim)
        self.k = torch.zeros(shape, dtype=dt, device=dev)
        self.v = torch.zeros(shape, dtype=dt, device=dev)
        self.doc_start = torch.zeros(batch, dtype=torch.int32, device=dev)
        self.len = 0
        self.tokens = None          # token history [batch, max_len], kept when the model has hashed tables


def _attend(q, k, v, scale, lo):
    """q ``[B,H,1,D]``, k/v ``[B,L,H,D]``; keys at positions < ``lo[b]`` are masked."""
    b, l = k.shape[0], k.shape[1]
    s = torch.einsum("bhqd,blhd->bhql", q.float(), k.float()) * scale
    pos = torch.arange(l, device=k.device)[None, None, None, :]
    s = s.masked_fill(pos < lo[:, None, None, None], float("-inf"))
    return torch.einsum("bhql,blhd->bqhd", torch.softmax(s, -1), v.float())


@torch.no_grad()
def _forward_cached(model, idx, cache: KVCache):
    """Run ``idx [B, t]`` (the whole prompt at prefill, one token afterwards), appending to the cache.  Returns the
    logits of the last position ``[B, V]``."""
    cfg = model.config
    b, t = idx.shape
    p0 = cache.len
    dev = idx.device
    pos = torch.arange(p0, p0 + t, device=dev)
    # document starts: most recent BOS at or before each new position
    if cfg.doc_mask:
        marks = torch.where(idx == cfg.bos_id, pos[None, :].expand(b, t).to(torch.int32),
                            torch.zeros(b, t, dtype=torch.int32, device=dev))
        ds = torch.maximum(torch.cummax(marks, 1).values, cache.doc_start[:, None])
        cache.doc_start = ds[:, -1].clone()
    else:
        ds = torch.zeros(b, t, dtype=torch.int32, device=dev)
    cos, sin = model.cos[p0:p0 + t], model.sin[p0:p0 + t]
    x = F.embedding(idx, model.transformer.wte.weight)
    if model.tables is not None:
        # rows keyed by the last `order` tokens: the cache keeps the token history for contexts that start before this call
        if cache.tokens is None:
            cache.tokens = torch.zeros(b, cache.k.shape[2], dtype=torch.int64, device=dev)
        cache.tokens[:, p0:p0 + t] = idx
        hist, tb = cache.tokens[:, :p0 + t], model.tables
        ids = torch.stack([RF.ngram_rows(hist, o, tb.rows, tb.seed + j, _doc_start_full(hist, cfg) if cfg.doc_mask else None)[:, p0:]
                           for j, o in enumerate(tb.orders)])
        x = tb.add_lookup(x, idx, None, model.table_lambda, rows=ids)
    x = RF.rms_norm(x)
    x0 = x
    skips = []
    n_layer, n_skip = cfg.n_layer, model.n_skip
    for i, blk in enumerate(model.transformer.h):
        if n_skip and i >= n_layer - n_skip:
            x = x + model.skip_lambda[i - (n_layer - n_skip)].to(x.dtype) * skips.pop()
        x = RF.resid_mix(x, x0, blk.resid_lambda, blk.x0_lambda)
        xn = RF.rms_norm(x)
        at = blk.attn
        q = F.linear(xn, at.c_q.weight).view(b, t, at.n_head, at.head_dim)
        k = F.linear(xn, at.c_k.weight).view(b, t, at.n_head, at.head_dim)
        v = F.linear(xn, at.c_v.weight).view(b, t, at.n_head, at.head_dim)
        if model.value_embeds is not None and str(i) in model.value_embeds:
            ve = F.embedding(idx, model.value_embeds[str(i)].weight).view(b, t, at.n_head, at.head_dim)
            v = v + blk.ve_lambda.to(v.dtype) * ve.to(v.dtype)
        q = RF.rms_norm(_rope_at(q, cos, sin))
        k = RF.rms_norm(_rope_at(k, cos, sin))
        cache.k[i, :, p0:p0 + t] = k
        cache.v[i, :, p0:p0 + t] = v
        ys = []
        for j in range(t):                                   # prefill is short in decode benchmarks; one row at a time
            cur = p0 + j
            lo = ds[:, j].to(torch.int64)
            if at.window:
                lo = torch.maximum(lo, torch.full_like(lo, max(0, (cur // 128 - (at.window // 128 - 1)) * 128)))
            ys.append(_attend(q[:, j:j + 1].transpose(1, 2), cache.k[i, :, :cur + 1], cache.v[i, :, :cur + 1],
                              at.scale, lo))
        y = torch.cat(ys, 1).reshape(b, t, -1).to(x.dtype)
        x = x + F.linear(y, at.c_proj.weight)
        xn = RF.rms_norm(x)
        if isinstance(blk.mlp, MoeMLP):
            x = blk.mlp(xn, residual=x)
        else:
            x = x + RF.mlp(xn, blk.mlp.c_fc.weight, blk.mlp.c_proj.weight)
        if n_skip and i < n_skip:
            skips.append(x)
    cache.len = p0 + t
    x = RF.rms_norm(x[:, -1])
    return RF.softcap_logits(F.linear(x, model.lm_head.weight)[..., :cfg.vocab_size], cfg.softcap)


def _doc_start_full(hist, cfg):
    return RF.doc_start_positions(hist, cfg.bos_id)


def _rope_at(x, cos, sin):
    d = x.shape[-1] // 2
    x1, x2 = x[..., :d].float(), x[..., d:].float()
    c, s = cos[None, :, None, :].float(), sin[None, :, None, :].float()
    return torch.cat([x1 * c + x2 * s, -x1 * s + x2 * c], -1).to(x.dtype)


def _token_rows(out, b, device) -> bool:
    """Whether ``out`` is what the fused step's last kernel reads forced tokens from and writes generated ones to by address:
    ``b`` rows of int64 on the model's device, each contiguous, any distance apart that keeps them disjoint."""
    return (out.dim() == 2 and out.shape[0] == b and out.dtype == torch.int64 and out.device == device and out.stride(1) == 1
            and (b == 1 or out.stride(0) >= out.shape[1]))


def projection_splits(b, n, k, residual, sms):
    """CTAs of a cluster that share the contraction of each 128-column tile of a decode projection (``n`` columns, ``k`` long).

    Doubled while a CTA keeps a K block of 64, up to what the batch makes worth while and what the ``sms`` SMs take in one go.
    A CTA finishes at least four sequences: up to 16 of them 4 CTAs (8 pad the sequences to 32), up to 32 8 CTAs.  Above, the exchange
    of the partial sums (32 KB a CTA) costs as much as the loads: 2 CTAs, except that the residual epilogue (out, c_proj: few columns,
    and per sequence a residual, x0 and sums of squares to handle) is shorter the fewer sequences a CTA finishes: 16, and 8 above
    64 sequences, where an SM holds one CTA.  Room: two CTAs of up to 64 sequences fit an SM, but clusters leave gaps: 1.6 CTAs an
    SM, 1.25 where clusters of 8 meet 17 to 32 sequences, one above 64 sequences and 0.8 of clusters of four or more (16 tiles
    by 8 CTAs: 524 us where 4 take 480).

    Six layers, us a step, all layers on this kernel, this rule against 2 CTAs for every projection of more than ten tiles and at most 160
    CTAs (``use_rows`` takes 1280 and 1408 wide up to 64 sequences to the other kernel, where they are faster still): 1280 wide the
    same (batch 64 242, batch 24 186, batch 8 171); 1408 wide 256 for 342 at batch 64, 336 for 399 at 128; 2048 wide 349 for 441, 437 for 515,
    246 for 253 at batch 8; 256 wide 145 for 148 and 204 for 212; 512 to 1152 wide the same.
    """
    tiles, kb = n // 128, k // 64
    most = 4 if b <= 16 else 8 if b <= 32 else 2 if not residual else 16 if b <= 64 else 8
    splits = 1
    while splits < most and splits * 2 <= kb:
        room = 1.6 if b <= 16 or 32 < b <= 64 else 1.25 if b <= 32 else 1.0 if splits == 1 else 0.8
        if tiles * splits * 2 > room * sms:
            break
        splits *= 2
    return splits


# What a projection brings to L2 ahead of the next one at most: a layer's largest weights with room to spare (13 MB at width 1280); of
# the head's 168 MB only as much as is read first.
AHEAD_LIMIT = 16 << 20


def rows_plan(b, n, k, sms):
    """``(columns of a tile, CTAs that share its contraction)`` of a projection on ``csrc/decode_rows.cu``, or None where it does not apply:
    more than 64 sequences (its MMA has 64 rows), too few or too many columns for one wave.

    A CTA fills an SM's shared memory, so a plan is one wave: at most ``sms`` CTAs, 0.9 of them in clusters of four or more, which leave
    gaps.  The contraction is shared until a CTA's part is 1536 at most (a chain of 96 MMAs, 2 us) and tiles of 32 columns or more
    occupy half of the SMs.  Within that, wide tiles (all CTAs read the same rows of X from L2: fewer of them, less traffic), but narrow
    ones in clusters of four or more, where a CTA's weights and its exchange count for more.  20 layers, 1280 wide, us a step, all else equal:
    qkv at batch 64 / 40 / 16 / 4 in tiles of 64 637 / 607 / 549 / 528, 48 644 / 607 / 545 / 520, 32 650 / 605 / 560 / 530, 64 by two CTAs
    654 / 633 / 568 / 523; out 32 by two 636 / 605 / 544 / 520, 16 by one 643 / 593 / 556 / 550; c_fc 64 634 / 597 / 534 / 518, 32 655 / 614 /
    569 / 543; c_proj 40 by four 634 / 594 / 534 / 517, 64 by four 660 / 597 / 536 / 517, 32 by two 661 / 621 / 560 / 548.
    """
    if b > 64 or k % 128:
        return None
    for s in (1, 2, 4, 8):
        if s > k // 128 or (k > 1536 * s and s < 8):
            continue
        fit = [nt for nt in (64, 48, 40, 32) if n % nt == 0 and sms // 2 <= n // nt * s <= (sms if s < 4 else int(0.9 * sms))]
        if fit:
            return (fit[0] if s < 4 else fit[-1]), s
    # few columns: the most CTAs with parts of 256 or more (256 wide: 115 us a step of six layers for 145 at batch 64, 103 for 106 at 8)
    few = [(n // nt * s, -s, nt) for nt in (16, 32, 64) for s in (1, 2, 4, 8)
           if n % nt == 0 and (s == 1 or k >= 256 * s) and k <= 1536 * s and n // nt * s < sms // 2]
    return (max(few)[2], -max(few)[1]) if few else None


def use_rows(b, c, a, hidden, sms):
    """Whether the layers' projections run on ``csrc/decode_rows.cu``: all four or none, since two of its CTAs, or one and one of the other
    kernel's, do not share an SM (2048 wide, ``out`` alone on it: 10 to 15 % slower).  Between 256 and 896 wide, models with few sequences
    stay on the other kernel, whose clusters split their contractions further.  Six layers, us a step here / there: 128 wide at batch 1 / 8 /
    16 88 / 93, 92 / 98, 94 / 100; 256 98 / 98, 103 / 106, 105 / 108; 384 113 / 107, 116 / 116, 118 / 118, at 20 121 / 128; 512 121 / 115, 125 / 121,
    127 / 126, at 20 132 / 132; 640 125 / 124, 129 / 131, 131 / 135; 768 134 / 133, 138 / 141, 137 / 141; 896 138 / 144, 138 / 149, 142 / 153."""
    if 256 < c < 896 and b <= 16:
        return False
    return all(rows_plan(b, n, k, sms) is not None for n, k in ((3 * a, c), (c, a), (hidden, c), (c, hidden)))


def head_on_rows(b, n, k):
    """Whether the head ``[n, k]`` of a step whose layers run on ``csrc/decode_rows.cu`` runs there too, its tiles walked by one CTA an SM.

    Above 32 sequences the other kernel pads to 64 and holds one CTA an SM; up to 16 it is the faster everywhere.  Between, what counts is
    the head's bytes.  A tile of a short contraction costs more here than there.  us a step of four layers here / there: 1280 x 65536 at
    batch 12 142.0 / 141.6, 20 143.8 / 142.5, 28 145.8 / 144.7, 33 148 / 158, 40 149 / 156, 64 157 / 160; 1024 x 32768 at 20 115.5 / 114.5, 33
    117.6 / 118.9, 64 125 / 127; 1536 x 65536 at 18 164.7 / 165.8, 28 169 / 170.5, 33 166 / 176; 1024 x 131072 at 18 158 / 162, 28 161 / 168, 64 169 /
    190.  Of six layers: 256 x 65536 at 20 129 / 122, 64 133.5 / 130, 256 x 8192 at 64 the same; 768 x 32768 at 40 160.5 / 158."""
    return (b > 32 and (k >= 1024 or n <= 16384)) or (b > 16 and n * k >= 100_000_000)


class NativeDecoder:
    """One decode step as a CUDA graph over the native kernels: embedding, fused norms, tcgen05 GEMMs, the two decode
    kernels (``csrc/decode.cu``: RoPE + QK-norm + cache append, cached attention), soft-capped logits, arg-max.  The
    position, the per-sequence document starts, the current tokens and the output buffer live on the device and are
    advanced inside the graph, so generating ``n`` tokens is ``n`` graph replays with no host synchronisation.
    Eligible: bf16 models on CUDA whose blocks all have attention with head_dim 128.  MoE blocks run their routed experts
    inside the graph (router, slotting, grouped expert GEMMs, combine: all device-side, a decode step uses one slot per
    sequence and expert); hashed input tables are looked up from row ids hashed on the device from the token history."""

    @staticmethod
    def eligible(model) -> bool:
        cfg = model.config
        w = model.lm_head.weight
        tables_ok = model.tables is None or model.tables.dtype == torch.bfloat16
        return (w.is_cuda and w.dtype == torch.bfloat16 and cfg.head_dim == 128 and tables_ok and getattr(model, "os1", None) is None
                and not ops.reference_path() and all(blk.attn is not None for blk in model.transformer.h))

    def __init__(self, model, cache: KVCache, first_tokens: torch.Tensor, out: torch.Tensor, prompt_len: int = 0):
        # positions below ``prompt_len`` are teacher-forced from ``out`` (stepwise prefill through the same graph)
        self.model, self.cache, self.out = model, cache, out
        dev = first_tokens.device
        self.prompt_len = torch.tensor([prompt_len], dtype=torch.int32, device=dev)
        self.tok = first_tokens.clone().to(torch.int64)
        self.pos = torch.tensor([cache.len], dtype=torch.int32, device=dev)
        self.graph = None
        cfg = model.config
        b, a = self.tok.shape[0], cfg.n_head * cfg.head_dim
        self.qbuf = torch.empty(b, a, dtype=torch.bfloat16, device=dev)
        self.y = torch.empty(b, a, dtype=torch.bfloat16, device=dev)
        # With few rows a projection has too few output tiles to pull its weights at memory speed, so its contraction
        # runs as a batch of products over K chunks of 256, each into its own fp32 slice, which the finishing kernel
        # adds in a fixed order (no atomics: a step is reproducible bit for bit).
        self.split = b <= 128 and cfg.n_embd % 256 == 0 and a % 256 == 0
        self.dense = [not isinstance(blk.mlp, MoeMLP) for blk in model.transformer.h]
        self.fused = self._fused_ok()
        if self.fused:
            c, f32, bf = cfg.n_embd, torch.float32, torch.bfloat16
            self.wqkv = [torch.cat([blk.attn.c_q.weight, blk.attn.c_k.weight, blk.attn.c_v.weight]) for blk in model.transformer.h]
            self.x0, self.xa, self.xb = (torch.empty(b, c, dtype=bf, device=dev) for _ in range(3))
            self.qkv = torch.empty(b, 3 * a, dtype=bf, device=dev)
            self.h = torch.empty(b, cfg.mlp_ratio * c, dtype=bf, device=dev)
            self.ssq_a, self.ssq_b = (torch.empty(c // 16, b, dtype=f32, device=dev) for _ in range(2))
            self.sms = torch.cuda.get_device_properties(dev).multi_processor_count
            self.rows = use_rows(b, c, a, cfg.mlp_ratio * c, self.sms)
            self.ticket = torch.zeros(1, dtype=torch.int32, device=dev)
            self.last_logits = torch.empty(b, model.lm_head.weight.shape[0], dtype=bf, device=dev)
        elif self.split:
            self.wqkv = [torch.cat([blk.attn.c_q.weight, blk.attn.c_k.weight, blk.attn.c_v.weight]).contiguous()
                         for blk in model.transformer.h]
            ws = self.wqkv + [blk.attn.c_proj.weight for blk in model.transformer.h]
            ws += [w for blk, dense in zip(model.transformer.h, self.dense) if dense for w in (blk.mlp.c_fc.weight, blk.mlp.c_proj.weight)]
            self.split = all(w.shape[1] % 256 == 0 for w in ws)
            self.part = torch.empty(max(b * w.shape[0] * (w.shape[1] // 256) for w in ws), dtype=torch.float32, device=dev)

    def _fused_ok(self) -> bool:
        """Whether the step runs on the kernels of ``csrc/decode_gemm.cu``: a plain dense decoder with at most 128 sequences.
        Any other ``out`` goes through the indexed reads and writes of the general step, which take or refuse it."""
        model, cfg = self.model, self.model.config
        ws = [w for blk, dense in zip(model.transformer.h, self.dense) if dense
              for w in (blk.attn.c_q.weight, blk.attn.c_k.weight, blk.attn.c_v.weight, blk.attn.c_proj.weight, blk.mlp.c_fc.weight, blk.mlp.c_proj.weight)]
        ws += [model.lm_head.weight, model.transformer.wte.weight]
        scalars = [v for blk in model.transformer.h for v in (blk.resid_lambda, blk.x0_lambda)]
        return (self.tok.shape[0] <= 128 and all(self.dense) and model.tables is None and model.value_embeds is None and not model.n_skip
                and len(model.transformer.h) > 0 and cfg.n_embd % 128 == 0 and _token_rows(self.out, self.tok.shape[0], self.tok.device)
                and all(w.dtype == torch.bfloat16 and w.is_contiguous() and w.data_ptr() % 16 == 0 and w.shape[0] % 128 == 0 and w.shape[1] % 64 == 0 for w in ws)
                and all(v.dtype == torch.float32 for v in scalars) and model.cos.dtype == torch.float32 and model.sin.dtype == torch.float32)

    def _proj(self, x, w, out, epi, ssq=None, n_ssq=0, res=None, mix=None, ssq_out=None, nxt=None):
        """One projection of the fused step, ``nxt`` the weights that it reads next; returns how many partial sums of squares a sequence has in ``ssq_out``."""
        from ..ops import _lib as L
        b, (n, k) = x.shape[0], w.shape
        x0, ma, mb = (self.x0, mix[0], mix[1]) if mix is not None else (None, None, None)
        head = epi == 3
        plan = None if not self.rows else rows_plan(b, n, k, self.sms) if not head else (64, 1) if head_on_rows(b, n, k) else None
        cap = ctypes.c_float(self.model.config.softcap)
        if plan is not None:
            nt, splits = plan
            L.call("bones_decode_rows", L.ptr(x), L.ptr(w), L.ptr(out), _I(b), _I(n), _I(k), _I(nt), _I(splits), _I(self.sms if head else 0), _I(epi), L.ptr(ssq), _I(n_ssq), L.ptr(res),
                   L.ptr(x0), L.ptr(ma), L.ptr(mb), L.ptr(ssq_out), cap, L.ptr(nxt),
                   ctypes.c_longlong(0 if nxt is None else min(2 * nxt.numel(), AHEAD_LIMIT)), _I(1), L.stream())
            return n // nt
        splits = projection_splits(b, n, k, res is not None, self.sms)
        L.call("bones_decode_gemm", L.ptr(x), L.ptr(w), L.ptr(out), _I(b), _I(n), _I(k), _I(splits), _I(epi), L.ptr(ssq), _I(n_ssq), L.ptr(res),
               L.ptr(x0), L.ptr(ma), L.ptr(mb), L.ptr(ssq_out), cap, _I(1), L.stream())
        return n // 128

    def _step_fused(self):
        """Five kernels a layer (qkv, attention, out, c_fc, c_proj), one before the first and two after the last; the norms,
        the residual mix, ReLU^2 and the soft-cap are in the projections' epilogues."""
        from ..ops import _lib as L
        model, cache, cfg = self.model, self.cache, self.model.config
        tok, pos, b, c = self.tok, self.pos, self.tok.shape[0], cfg.n_embd
        tmax = cache.k.shape[2]
        ds = cache.doc_start if cfg.doc_mask else None
        hs = model.transformer.h
        w = model.transformer.wte.weight
        L.call("bones_decode_begin", L.ptr(tok), L.ptr(pos), L.ptr(ds), ctypes.c_longlong(cfg.bos_id), L.ptr(w), ctypes.c_longlong(w.shape[0]), _I(c),
               L.ptr(hs[0].resid_lambda), L.ptr(hs[0].x0_lambda), L.ptr(self.x0), L.ptr(self.xa), L.ptr(self.ssq_a), _I(b), L.stream())
        n_ssq = 1
        for i, blk in enumerate(hs):
            at = blk.attn
            self._proj(self.xa, self.wqkv[i], self.qkv, 0, ssq=self.ssq_a, n_ssq=n_ssq, nxt=at.c_proj.weight)
            L.call("bones_decode_attn_step", L.ptr(self.qkv), L.ptr(model.cos), L.ptr(model.sin), L.ptr(cache.k[i]), L.ptr(cache.v[i]), L.ptr(pos), L.ptr(ds),
                   L.ptr(self.y), _I(b), _I(at.n_head), _I(tmax), ctypes.c_float(at.scale), _I(at.window // 128), L.stream())
            n_ssq = self._proj(self.y, at.c_proj.weight, self.xb, 2, res=self.xa, ssq_out=self.ssq_b, nxt=blk.mlp.c_fc.weight)
            self._proj(self.xb, blk.mlp.c_fc.weight, self.h, 1, ssq=self.ssq_b, n_ssq=n_ssq, nxt=blk.mlp.c_proj.weight)
            nxt = hs[i + 1] if i + 1 < len(hs) else None
            mix = (nxt.resid_lambda, nxt.x0_lambda) if nxt is not None else None
            n_ssq = self._proj(self.h, blk.mlp.c_proj.weight, self.xa, 2, res=self.xb, mix=mix, ssq_out=self.ssq_a,
                               nxt=self.wqkv[i + 1] if nxt is not None else model.lm_head.weight)
        self._proj(self.xa, model.lm_head.weight, self.last_logits, 3, ssq=self.ssq_a, n_ssq=n_ssq)
        L.call("bones_decode_end", L.ptr(self.last_logits), ctypes.c_longlong(self.last_logits.shape[1]), _I(cfg.vocab_size), L.ptr(pos),
               L.ptr(self.prompt_len), L.ptr(self.out), ctypes.c_longlong(self.out.stride(0)), _I(self.out.shape[1]), L.ptr(tok), L.ptr(self.ticket), _I(b),
               L.stream())

    def _lin(self, x, w, mode=0, residual=None):
        """``x [b, k] @ w[n, k]^T`` as ``k / 256`` batched partial products into fp32 slices, then their ordered sum as
        bf16 (mode 0), through ReLU^2 (2) or ``+ residual`` (1)."""
        from ..ops import _lib as L
        b, k = x.shape
        n = w.shape[0]
        splits = k // 256
        part = self.part[:splits * b * n]
        L.gemm(x, w, part, m=b, n=n, k=256, lda=x.stride(0), ldb=w.stride(0), ldd=n, epi=L.EPI_F32, force_bn=128, pair=False,
               batch=splits, stride_a=256, stride_b=256, stride_d=b * n)
        out = torch.empty(b, n, dtype=torch.bfloat16, device=x.device)
        L.call("bones_acc_finish", L.ptr(part), ctypes.c_int(splits), ctypes.c_longlong(b * n), L.ptr(residual), L.ptr(out),
               ctypes.c_longlong(b * n), ctypes.c_int(mode), L.stream())
        return out

    def _step(self):
        from ..ops import _lib as L
        from ..ops import cuda as C
        if self.fused:
            return self._step_fused()
        model, cache, cfg = self.model, self.cache, self.model.config
        tok, pos = self.tok, self.pos
        b, tmax = tok.shape[0], cache.k.shape[2]
        if cfg.doc_mask:
            cache.doc_start.copy_(torch.where(tok == cfg.bos_id, pos.expand(b), cache.doc_start))
        x = ops.embedding(tok, model.transformer.wte.weight, torch.bfloat16)
        if model.tables is not None:
            tb = model.tables
            ds = cache.doc_start if cfg.doc_mask else None
            for j, o in enumerate(tb.orders):
                rows = RF.ngram_rows_at(self.out, pos, o, tb.rows, tb.seed + j, ds)
                x = x + model.table_lambda[j].to(x.dtype) * tb.gather(j, rows)
        x = ops.rms_norm(x)
        x0 = x
        skips = []
        n_layer, n_skip = cfg.n_layer, model.n_skip
        for i, blk in enumerate(model.transformer.h):
            if n_skip and i >= n_layer - n_skip:
                x = x + model.skip_lambda[i - (n_layer - n_skip)].to(x.dtype) * skips.pop()
            x, xn = ops.resid_mix_norm(x, x0, blk.resid_lambda, blk.x0_lambda)
            at = blk.attn
            qkv = self._lin(xn, self.wqkv[i]) if self.split else ops.linear_qkv(xn, at.c_q.weight, at.c_k.weight, at.c_v.weight)
            ve = lam = None
            if model.value_embeds is not None and str(i) in model.value_embeds:
                ve = ops.embedding(tok, model.value_embeds[str(i)].weight, torch.bfloat16)
                lam = blk.ve_lambda.detach().float()
            L.call("bones_decode_qkv", L.ptr(qkv), L.ptr(model.cos), L.ptr(model.sin), L.ptr(ve), L.ptr(lam), L.ptr(self.qbuf),
                   L.ptr(cache.k[i]), L.ptr(cache.v[i]), L.ptr(pos), C._I(b), C._I(at.n_head), C._I(tmax), L.stream())
            L.call("bones_decode_attn", L.ptr(self.qbuf), L.ptr(cache.k[i]), L.ptr(cache.v[i]), L.ptr(pos),
                   L.ptr(cache.doc_start if cfg.doc_mask else None), L.ptr(self.y), C._I(b), C._I(at.n_head), C._I(tmax),
                   C._F(at.scale), C._I(at.window // 128), L.stream())
            if self.split:
                x = self._lin(self.y, at.c_proj.weight, 1, x)
                x, xn = ops.norm_split(x)
                if self.dense[i]:
                    x = self._lin(self._lin(xn, blk.mlp.c_fc.weight, 2), blk.mlp.c_proj.weight, 1, x)
                else:
                    x = blk.mlp(xn.view(b, 1, -1), residual=x.view(b, 1, -1)).view(b, -1)
            else:
                x = ops.linear(self.y, at.c_proj.weight, residual=x)
                x, xn = ops.norm_split(x)
                x = blk.mlp(xn.view(b, 1, -1), residual=x.view(b, 1, -1)).view(b, -1) if not self.dense[i] else blk.mlp(xn, residual=x)
            if n_skip and i < n_skip:
                skips.append(x)
        xn = ops.rms_norm(x)
        logits = C.mm_nt(xn, model.lm_head.weight, epi=L.EPI_SOFTCAP, alpha=1.0 / cfg.softcap, beta=cfg.softcap)
        self.last_logits = logits                                          # [B, padded vocab] bf16, soft-capped
        nxt = logits[:, :cfg.vocab_size].float().argmax(-1)
        pos.add_(1)
        at = pos.to(torch.int64)
        forced = self.out.index_select(1, at)[:, 0]
        nxt = torch.where((pos < self.prompt_len).expand_as(nxt), forced, nxt)
        self.out.index_copy_(1, at, nxt[:, None])                         # token at position pos (after the increment)
        tok.copy_(nxt)

    @torch.no_grad()
    def run(self, n_steps: int):
        """``n_steps`` decode steps; the first one runs eagerly (it also warms every kernel up), the rest replay the graph."""
        if n_steps <= 0:
            return
        self._step()
        if n_steps == 1:
            return
        if self.graph is None:
            torch.cuda.synchronize()
            self.graph = torch.cuda.CUDAGraph()
            side = torch.cuda.Stream()
            side.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(side):
                with torch.cuda.graph(self.graph, stream=side):
                    self._step()
            torch.cuda.current_stream().wait_stream(side)       # capturing does not execute the step
        for _ in range(n_steps - 1):
            self.graph.replay()


@torch.no_grad()
def greedy_decode(model, prompts: torch.Tensor, n_new: int) -> torch.Tensor:
    """``prompts [B, P]`` -> ``[B, P + n_new]`` by arg-max decoding."""
    b, p = prompts.shape
    if p + n_new > model.config.sequence_len:
        raise ValueError("prompt + new tokens exceed the model's sequence length")
    if getattr(model, "os1", None) is not None or any(blk.attn is None for blk in model.transformer.h):
        return greedy_decode_full(model, prompts, n_new)          # output table and attention-free blocks: cache-free route
    cache = KVCache(model, b, p + n_new)
    if NativeDecoder.eligible(model) and n_new >= 1:
        out = torch.zeros(b, p + n_new, dtype=torch.int64, device=prompts.device)
        out[:, :p] = prompts
        if p <= 512:
            # short prompts are pre-filled token by token through the same graph (teacher-forced), then decoded
            dec = NativeDecoder(model, cache, prompts[:, 0], out, prompt_len=p)
            dec.run(p + n_new - 1)
        else:
            # long prompts: prefill on the cached PyTorch route, then one graph replay per generated token
            logits = _forward_cached(model, prompts, cache)
            first = logits.argmax(-1)
            out[:, p] = first
            if n_new > 1:
                dec = NativeDecoder(model, cache, first, out)
                dec.run(n_new - 1)
        L_check()
        return out
    out = [prompts]
    logits = _forward_cached(model, prompts, cache)
    for _ in range(n_new):
        nxt = logits.argmax(-1, keepdim=True)
        out.append(nxt)
        if cache.len >= p + n_new:
            break
        logits = _forward_cached(model, nxt, cache)
    return torch.cat(out, 1)[:, :p + n_new]


@torch.no_grad()
def greedy_decode_full(model, prompts: torch.Tensor, n_new: int) -> torch.Tensor:
    """Cache-free decoding (re-runs the full forward per token); the oracle for the cached path and the route used
    when hashed tables are attached."""
    seq = prompts
    for _ in range(n_new):
        logits = model(seq)[:, -1]
        seq = torch.cat([seq, logits.argmax(-1, keepdim=True)], 1)
    return seq
