"""The work a user of ``them_bones_b200`` has it do, as measurable cases.

Every case is one call (or one forward and backward) through a public entry point: the operators of ``ops``, the MoE
block of ``models.moe``, the Newton-Schulz iteration of the Muon optimizer and the CUDA-graph decoder.  The sizes are
those of the dense and MoE benchmark models (20 layers, width 1280, 10 heads of 128, hidden 5120, 16 experts of 2560,
vocabulary 65536, sequences of 2048 in documents of 128 to 2048 tokens), of the tiny model (width 256, 4 heads of 64,
vocabulary 8192) and of scoring, where sequences have any length.

``listed`` gives the fixed cases, ``draw`` further ones of the same ranges, ``prepare`` the state a program holds before
the call, ``run`` the call, ``work`` the bytes and operations it cannot do without, ``tolerance`` how far two correct
implementations may be apart and ``exact`` the results in 64 bits from plain torch.
"""
from __future__ import annotations

import math
import random

import torch
import torch.nn.functional as F

BF16 = torch.bfloat16


# -- the cases ---------------------------------------------------------------------------------------------------------
def listed():
    return [
        # one attention layer of a training micro-step of the dense model: packed documents, forward and backward
        dict(name="attention_train", kind="attention", b=16, t=2048, heads=10, head_dim=128, window=0, docs=True, backward=True),
        # a banded layer of the sliding-window recipe on shorter windows
        dict(name="attention_window", kind="attention", b=4, t=1024, heads=10, head_dim=128, window=256, docs=True, backward=True),
        # the tiny model's attention: latency
        dict(name="attention_tiny", kind="attention", b=4, t=256, heads=4, head_dim=64, window=0, docs=True, backward=True),
        # scoring a batch of requests of a ragged length
        dict(name="attention_score", kind="attention", b=8, t=1777, heads=10, head_dim=128, window=0, docs=True, backward=False),
        # the MLP of a training micro-step, block-scaled
        dict(name="mlp_mxfp8_train", kind="mlp", rows=32768, width=1280, hidden=5120, precision="mxfp8", backward=True),
        # the same MLP in bf16 on a small ragged batch
        dict(name="mlp_bf16_small", kind="mlp", rows=1000, width=1280, hidden=5120, precision="bf16", backward=True),
        # a block's residual mix and its two norms
        dict(name="norm_train", kind="norm", rows=65536, width=1280, backward=True),
        # the loss head of a training micro-step
        dict(name="head_train", kind="head", rows=16384, width=1280, vocab=65536, backward=True),
        # per-token log-likelihoods of a request: what scoring asks of the head
        dict(name="head_score", kind="head", rows=777, width=1280, vocab=65536, backward=False),
        # an MoE block of a training micro-step, all experts on one GPU
        dict(name="moe_train", kind="moe", b=8, t=2048, width=1280, hidden=2560, experts=16, topk=2, precision="mxfp8"),
        # the optimizer's orthogonalisation of one rank's share of the MLP matrices
        dict(name="newton_schulz", kind="newton_schulz", n=5, r=5120, c=1280),
        # serving: a batch of sequences through the cached decode step, token by token (prompts, then the next-token logits)
        dict(name="decode", kind="decode", layers=20, width=1280, heads=10, vocab=65536, batch=64, steps=128),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["attention", "attention", "mlp", "mlp", "norm", "head", "head", "moe", "newton_schulz", "decode"])
    if kind == "attention":
        hd = rng.choice([128, 128, 128, 64])
        heads, t = (rng.choice([2, 4, 10]), _log_int(rng, 100, 2048)) if hd == 128 else (4, _log_int(rng, 60, 512))
        if rng.random() < 0.5:
            t = -(-t // 128) * 128
        b = _log_int(rng, 1, max(1, min(16, 32768 // t)))
        return dict(kind=kind, b=b, t=t, heads=heads, head_dim=hd, window=rng.choice([0, 0, 0, 256, 512]), docs=rng.random() < 0.75,
                    backward=rng.random() < 0.6)
    if kind == "mlp":
        width, hidden = rng.choice([(1280, 5120), (1280, 5120), (256, 1024), (1280, 2560)])
        return dict(kind=kind, rows=_log_int(rng, 64, 32768), width=width, hidden=hidden, precision=rng.choice(["bf16", "mxfp8"]),
                    backward=rng.random() < 0.7)
    if kind == "norm":
        return dict(kind=kind, rows=_log_int(rng, 64, 65536), width=rng.choice([1280, 1280, 256]), backward=rng.random() < 0.7)
    if kind == "head":
        width, vocab = rng.choice([(1280, 65536), (1280, 65536), (256, 8192)])
        return dict(kind=kind, rows=_log_int(rng, 64, 16384), width=width, vocab=vocab, backward=rng.random() < 0.6)
    if kind == "moe":
        t = rng.choice([512, 1024, 2048])
        return dict(kind=kind, b=_log_int(rng, 1, 8), t=t, width=1280, hidden=2560, experts=rng.choice([8, 16]), topk=rng.choice([1, 2]),
                    precision=rng.choice(["bf16", "mxfp8"]))
    if kind == "newton_schulz":
        r, c = rng.choice([(1280, 1280), (5120, 1280), (1280, 5120), (1024, 256)])
        return dict(kind=kind, n=_log_int(rng, 1, 10 if max(r, c) <= 1280 else 5), r=r, c=c)
    return dict(kind=kind, layers=rng.choice([4, 12, 20]), width=1280, heads=10, vocab=65536, batch=_log_int(rng, 1, 64),
                steps=_log_int(rng, 16, 128))


# -- inputs ------------------------------------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _normal(g, *shape, std=1.0, dtype=BF16):
    return (torch.randn(*shape, generator=g, device="cuda", dtype=torch.float32) * std).to(dtype)


def _doc_starts(b, t, seed):
    """``[b, t]``: for each position the first position of its document; documents of 128 to 2048 tokens packed back to
    back into windows, so that a window usually begins inside one."""
    rng = random.Random(seed)
    rows = []
    for _ in range(b):
        row, begin, end = [], 0, rng.randint(1, rng.randint(128, 2048))
        while len(row) < t:
            row += [begin] * (min(end, t) - begin)
            begin, end = end, end + rng.randint(128, 2048)
        rows.append(row)
    return torch.tensor(rows, dtype=torch.int32)


def _rotary(t, d, base=100000.0):
    """Rotary tables rounded to bf16, kept in fp32 (as the models hold them)."""
    inv = 1.0 / (base ** (torch.arange(0, d, 2, dtype=torch.float32, device="cuda") / d))
    a = torch.outer(torch.arange(t, dtype=torch.float32, device="cuda"), inv)
    return a.cos().to(BF16).float(), a.sin().to(BF16).float()


def _zipf(g, vocab, *shape):
    """Token ids, Zipf(1.1) over ``1 .. vocab - 1`` (0 is the document mark)."""
    cdf = torch.arange(1, vocab, dtype=torch.float64).pow(-1.1).cumsum(0)          # on the CPU: the same sums every time
    u = torch.rand(shape, generator=g, device="cuda", dtype=torch.float64)
    return torch.searchsorted((cdf / cdf[-1]).cuda(), u).clamp_max(vocab - 2) + 1


def _attention_inputs(case, seed):
    g = _gen(seed)
    b, t, h, d = case["b"], case["t"], case["heads"], case["head_dim"]
    qkv = _normal(g, b, t, 3 * h * d)
    cos, sin = _rotary(t, d)
    ds = _doc_starts(b, t, seed).cuda() if case["docs"] else None
    return dict(qkv=qkv, cos=cos, sin=sin, ds=ds, dy=_normal(g, b, t, h * d) if case["backward"] else None)


def _mlp_inputs(case, seed):
    g = _gen(seed)
    m, c, f = case["rows"], case["width"], case["hidden"]
    s = math.sqrt(3.0 / c)
    return dict(x=_normal(g, m, c), w_fc=_normal(g, f, c, std=0.7 * s), w_proj=_normal(g, c, f, std=0.3 * s), residual=_normal(g, m, c),
                dy=_normal(g, m, c) if case["backward"] else None)


def _norm_inputs(case, seed):
    g = _gen(seed)
    m, c = case["rows"], case["width"]
    d = dict(x=_normal(g, m, c, std=2.0), x0=_normal(g, m, c), a=torch.full((1,), 0.9, device="cuda"), b=torch.full((1,), 0.2, device="cuda"))
    if case["backward"]:
        # correlated with the operands, so that the gains' gradients are not the small remainder of large sums
        dx2 = (_normal(g, m, c).float() + 0.3 * d["x"].float() + 0.3 * d["x0"].float()).to(BF16)
        d.update(dn1=_normal(g, m, c), dx2=dx2, dn2=_normal(g, m, c))
    return d


def _head_inputs(case, seed):
    g = _gen(seed)
    m, c, v = case["rows"], case["width"], case["vocab"]
    targets = _zipf(g, v, m)
    targets[torch.rand(m, generator=g, device="cuda") < 0.01] = -1            # masked targets: document starts
    return dict(x=_normal(g, m, c), w=_normal(g, v, c, std=2.0 / math.sqrt(c)), targets=targets)


def _moe_inputs(case, seed):
    g = _gen(seed)
    b, t, c, f, e = case["b"], case["t"], case["width"], case["hidden"], case["experts"]
    s = math.sqrt(3.0 / c)
    return dict(x=_normal(g, b, t, c), residual=_normal(g, b, t, c), router=_normal(g, e, c, std=s), w_fc=_normal(g, e, f, c, std=0.7 * s),
                w_proj=_normal(g, e, c, f, std=0.3 * s), dy=_normal(g, b, t, c))


def _moe_capacity(case):
    return max(1, int(round(1.25 * case["t"] * case["topk"] / case["experts"])))


def _newton_schulz_inputs(case, seed):
    g = _gen(seed)
    x = torch.randn(case["n"], case["r"], case["c"], generator=g, device="cuda")
    # a gradient's spectrum: a few strong directions over noise
    u, v = (torch.randn(case["n"], k, 8, generator=g, device="cuda") for k in (case["r"], case["c"]))
    x = x + 4.0 * u @ v.mT
    return dict(x=(x / x.norm(dim=(1, 2), keepdim=True)).to(BF16).contiguous())


def _decode_inputs(case, seed):
    g = _gen(seed)
    c, v = case["width"], case["vocab"]
    s = math.sqrt(1.0 / c)
    layers = []
    for _ in range(case["layers"]):
        w = {k: _normal(g, c, c, std=s) for k in ("q", "k", "v")}
        w.update(o=_normal(g, c, c, std=0.3 * s), fc=_normal(g, 4 * c, c, std=0.4 * s), proj=_normal(g, c, 4 * c, std=0.3 * s))
        layers.append(w)
    tokens = _zipf(g, v, case["batch"], case["steps"])
    tokens[:, 0] = 0
    tokens[torch.rand(tokens.shape, generator=g, device="cuda") < 1.0 / 256] = 0        # a new document begins
    return dict(layers=layers, wte=_normal(g, v, c, std=0.8), head=_normal(g, v, c, std=2.0 * s), tokens=tokens)


_INPUTS = dict(attention=_attention_inputs, mlp=_mlp_inputs, norm=_norm_inputs, head=_head_inputs, moe=_moe_inputs,
               newton_schulz=_newton_schulz_inputs, decode=_decode_inputs)


def prepare(case, seed):
    from them_bones_b200.ops import mxfp8
    st = _INPUTS[case["kind"]](case, seed)
    mxfp8.weights_updated()                        # new weights: their quantised copies are made anew
    for name in ("qkv", "x", "x0", "a", "b", "w", "w_fc", "w_proj", "residual"):
        if name in st and case.get("backward") and st[name].is_floating_point():
            st[name].requires_grad_(True)
    if case["kind"] == "moe":
        st["block"] = _moe_block(case, st)
        st["x"].requires_grad_(True)
    if case["kind"] == "decode":
        st = _decode_state(case, st)
    st["case"] = case
    return st


def _moe_block(case, st):
    from them_bones_b200.config import GPTConfig
    from them_bones_b200.models.moe import MoeMLP
    cfg = GPTConfig(sequence_len=case["t"], vocab_size=65536, n_layer=20, n_head=10, n_embd=case["width"], mlp_precision=case["precision"],
                    moe_layers=(2,), moe_experts=case["experts"], moe_topk=case["topk"], moe_capacity=_moe_capacity(case),
                    moe_hidden=case["hidden"])
    with torch.device("cuda"):
        block = MoeMLP(cfg, 2)
    for name in ("router", "w_fc", "w_proj"):
        p = getattr(block, name)
        p.data = st.pop(name)
    return block


def _decode_state(case, st):
    from them_bones_b200.config import GPTConfig
    from them_bones_b200.models.gpt import GPT
    cfg = GPTConfig(sequence_len=2048, vocab_size=case["vocab"], n_layer=case["layers"], n_head=case["heads"], n_embd=case["width"], doc_mask=True)
    with torch.device("cuda"):
        model = GPT(cfg)
    model.transformer.wte.weight.data, model.lm_head.weight.data = st["wte"], st["head"]
    for blk, w in zip(model.transformer.h, st["layers"]):
        at = blk.attn
        for lin, key in ((at.c_q, "q"), (at.c_k, "k"), (at.c_v, "v"), (at.c_proj, "o"), (blk.mlp.c_fc, "fc"), (blk.mlp.c_proj, "proj")):
            lin.weight.data = w[key]
        blk.resid_lambda.data.fill_(1.0)
        blk.x0_lambda.data.fill_(0.05)
    model.cast_compute(BF16)
    return dict(model=model.eval(), tokens=st["tokens"])


# -- the calls ---------------------------------------------------------------------------------------------------------
def run(st):
    return _RUN[st["case"]["kind"]](st, st["case"])


def _run_attention(st, case):
    from them_bones_b200 import ops
    d = case["head_dim"]
    with torch.set_grad_enabled(case["backward"]):
        y = ops.attention(st["qkv"], st["cos"], st["sin"], case["heads"], d, 1.0 / math.sqrt(d), st["ds"], case["window"])
        if not case["backward"]:
            return y
        return [y] + list(torch.autograd.grad(y, [st["qkv"]], st["dy"]))


def _run_mlp(st, case):
    from them_bones_b200 import ops
    with torch.set_grad_enabled(case["backward"]):
        y = ops.mlp(st["x"], st["w_fc"], st["w_proj"], residual=st["residual"], precision=case["precision"])
        if not case["backward"]:
            return y
        return [y] + list(torch.autograd.grad(y, [st["x"], st["w_fc"], st["w_proj"]], st["dy"]))


def _run_norm(st, case):
    from them_bones_b200 import ops
    with torch.set_grad_enabled(case["backward"]):
        xm, n1 = ops.resid_mix_norm(st["x"], st["x0"], st["a"], st["b"])
        x2, n2 = ops.norm_split(xm)
        if not case["backward"]:
            return [n1, x2, n2]
        return [n1, x2, n2] + list(torch.autograd.grad([n1, x2, n2], [st["x"], st["x0"], st["a"], st["b"]],
                                                       [st["dn1"], st["dx2"], st["dn2"]]))


def _run_head(st, case):
    from them_bones_b200 import ops
    if not case["backward"]:
        with torch.no_grad():
            return ops.lmhead_loss(st["x"], st["w"], st["targets"], case["vocab"], 15.0, reduction="none")
    loss = ops.lmhead_loss(st["x"], st["w"], st["targets"], case["vocab"], 15.0)
    return [loss] + list(torch.autograd.grad(loss, [st["x"], st["w"]]))


def _run_moe(st, case):
    block, aux = st["block"], []
    y = block(st["x"], residual=st["residual"], moe_aux=aux)
    grads = torch.autograd.grad([y, aux[0][0]], [st["x"], block.router, block.w_fc, block.w_proj], [st["dy"], torch.ones_like(aux[0][0])])
    return [y, aux[0][0]] + list(grads)


def _run_newton_schulz(st, case):
    from them_bones_b200.ops.muon_native import newton_schulz
    return newton_schulz(st["x"])


def _run_decode(st, case):
    from them_bones_b200.utils.decode import KVCache, NativeDecoder
    tokens = st["tokens"]
    b, p = tokens.shape
    with torch.no_grad():
        out = torch.zeros(b, p + 1, dtype=torch.int64, device=tokens.device)
        out[:, :p] = tokens
        dec = NativeDecoder(st["model"], KVCache(st["model"], b, p + 1), tokens[:, 0], out, prompt_len=p)
        dec.run(p)
    return dec.last_logits


_RUN = dict(attention=_run_attention, mlp=_run_mlp, norm=_run_norm, head=_run_head, moe=_run_moe, newton_schulz=_run_newton_schulz,
            decode=_run_decode)


# -- what a pass cannot do without -------------------------------------------------------------------------------------
def _attended_pairs(case):
    b, t, w = case["b"], case["t"], case["window"]
    q = torch.arange(t)
    lo = torch.clamp((q // 128 - (w // 128 - 1)) * 128, min=0) if w else torch.zeros_like(q)
    lo = torch.maximum(lo, _doc_starts(b, t, 1).long()) if case["docs"] else lo.expand(b, t)
    return int((q - lo + 1).sum())


def work(case):
    k = case["kind"]
    if k == "attention":
        a, n = case["heads"] * case["head_dim"], case["b"] * case["t"]
        return dict(flops=(14 if case["backward"] else 4) * _attended_pairs(case) * a, bytes=2 * n * a * (8 if case["backward"] else 4))
    if k == "mlp":
        m, c, f = case["rows"], case["width"], case["hidden"]
        return dict(flops=(12 if case["backward"] else 4) * m * c * f, bytes=2 * ((5 if case["backward"] else 3) * m * c + (4 if case["backward"] else 2) * c * f))
    if k == "norm":
        return dict(flops=0, bytes=2 * case["rows"] * case["width"] * (10 if case["backward"] else 5))
    if k == "head":
        m, c, v = case["rows"], case["width"], case["vocab"]
        return dict(flops=(6 if case["backward"] else 2) * m * c * v, bytes=2 * (m * c + v * c) * (2 if case["backward"] else 1) + 12 * m)
    if k == "moe":
        n, c, f, e = case["b"] * case["t"], case["width"], case["hidden"], case["experts"]
        return dict(flops=12 * n * case["topk"] * c * f, bytes=2 * (5 * n * c + 4 * e * c * f))
    if k == "newton_schulz":
        n, r, c = case["n"], case["r"], case["c"]
        s, l = min(r, c), max(r, c)
        # the two symmetric products need half of their entries
        return dict(flops=5 * n * (2 * s * s * l + s * s * l + s * s * s), bytes=4 * n * r * c)
    c, v, b, t = case["width"], case["vocab"], case["batch"], case["steps"]
    weights = case["layers"] * 12 * c * c + v * c
    cache = 2 * case["layers"] * b * c * min(t, 256)
    return dict(flops=2 * t * b * weights, bytes=2 * t * (weights + cache // 2))


# -- how far apart two correct implementations may be --------------------------------------------------------------------
def tolerance(case):
    k = case["kind"]
    if k == "attention":
        return dict(rel=1.5e-2)
    if k == "mlp":
        return dict(rel=2.5e-2 if case["precision"] == "mxfp8" else 1e-2)
    if k == "norm":
        return dict(rel=1e-2)
    if k == "head":
        return dict(rel=1e-2)
    if k == "moe":
        return dict(rel=4e-2 if case["precision"] == "mxfp8" else 2e-2)
    if k == "newton_schulz":
        return dict(rel=6e-2)
    return dict(rel=6e-2)


# -- the results in 64 bits ----------------------------------------------------------------------------------------------
def _norm64(x):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + 2.0 ** -23)


def _rope64(x, cos, sin):
    d = x.shape[-1] // 2
    x1, x2, c, s = x[..., :d], x[..., d:], cos.double()[:, None, :], sin.double()[:, None, :]
    return torch.cat([x1 * c + x2 * s, x2 * c - x1 * s], -1)


def _attend64(q, k, v, cos, sin, scale, ds, window):
    """``q, k, v [t, h, d]`` of one sequence, before rotation."""
    t = q.shape[0]
    q, k = _norm64(_rope64(q, cos, sin)), _norm64(_rope64(k, cos, sin))
    at = torch.arange(t, device=q.device)
    mask = at[None, :] <= at[:, None]
    if window:
        mask = mask & (at[:, None] // 128 - at[None, :] // 128 < window // 128)
    if ds is not None:
        mask = mask & (at[None, :] >= ds[:, None])
    s = torch.einsum("qhd,khd->hqk", q, k) * scale
    p = torch.softmax(s.masked_fill(~mask, float("-inf")), -1)
    return torch.einsum("hqk,khd->qhd", p, v)


def _exact_attention(case, st):
    b, t, h, d = case["b"], case["t"], case["heads"], case["head_dim"]
    ys, dqkvs = [], []
    for j in range(b):
        x = st["qkv"][j].double().requires_grad_(case["backward"])
        q, k, v = x.view(t, 3, h, d).unbind(1)
        y = _attend64(q, k, v, st["cos"], st["sin"], 1.0 / math.sqrt(d), st["ds"][j] if st["ds"] is not None else None,
                      case["window"]).reshape(t, h * d)
        ys.append(y.detach())
        if case["backward"]:
            dqkvs.append(torch.autograd.grad(y, x, st["dy"][j].double())[0])
    return [torch.stack(ys), torch.stack(dqkvs)] if case["backward"] else torch.stack(ys)


def _exact_mlp(case, st):
    x, w1, w2, r = (st[k].double() for k in ("x", "w_fc", "w_proj", "residual"))
    a = F.relu(x @ w1.T)
    h = a.square()
    y = h @ w2.T + r
    if not case["backward"]:
        return y
    dy = st["dy"].double()
    dpre = (dy @ w2) * (2.0 * a)
    return [y, dpre @ w1, dpre.T @ x, dy.T @ h]


def _exact_norm(case, st):
    need = case["backward"]
    x, x0, a, b = (st[k].detach().double().requires_grad_(need) for k in ("x", "x0", "a", "b"))
    xm = a * x + b * x0
    n1 = _norm64(xm)
    outs = [n1, xm, n1]
    if not need:
        return outs
    grads = torch.autograd.grad([n1, xm, n1], [x, x0, a, b], [st["dn1"].double(), st["dx2"].double(), st["dn2"].double()])
    return [o.detach() for o in outs] + list(grads)


def _exact_head(case, st):
    m, v = case["rows"], case["vocab"]
    w, tg, cap = st["w"].detach().double(), st["targets"], 15.0
    nll, dx = torch.zeros(m, dtype=torch.float64, device="cuda"), []
    dw = torch.zeros_like(w)
    n_valid = (tg >= 0).sum()
    for r0 in range(0, m, 4096):
        x, t = st["x"][r0:r0 + 4096].detach().double(), tg[r0:r0 + 4096]
        th = torch.tanh(x @ w.T / cap)
        lse = torch.logsumexp(cap * th, -1)
        ok = t >= 0
        nll[r0:r0 + 4096] = torch.where(ok, lse - (cap * th).gather(1, t.clamp_min(0)[:, None])[:, 0], 0.0)
        if case["backward"]:
            g = torch.exp(cap * th - lse[:, None])
            g.scatter_add_(1, t.clamp_min(0)[:, None], torch.full((t.shape[0], 1), -1.0, dtype=torch.float64, device="cuda"))
            g *= (1.0 - th.square()) * ok[:, None] / n_valid
            dx.append(g @ w)
            dw += g.T @ x
    return [nll.sum() / n_valid, torch.cat(dx), dw] if case["backward"] else nll


def _exact_moe(case, st):
    b, t, c, e, k = case["b"], case["t"], case["width"], case["experts"], case["topk"]
    x = st["x"].detach().double().requires_grad_(True)
    router, w1, w2 = (st[n].detach().double().requires_grad_(True) for n in ("router", "w_fc", "w_proj"))
    h = x.view(b * t, c)
    logits = h @ router.T
    p = torch.softmax(logits, -1)
    top, idx = p.topk(k, dim=-1)
    gates = top / top.sum(-1, keepdim=True) if k == 2 else top
    cap = _moe_capacity(case)
    out = torch.zeros_like(h)
    chosen = F.one_hot(idx, e).sum(1)
    place = (chosen.view(b, t, e).cumsum(1).view(b * t, e) - chosen).gather(1, idx)       # earlier choices of the same expert
    for j in range(e):
        tok, which = ((idx == j) & (place < cap)).nonzero(as_tuple=True)
        a = F.relu(h[tok] @ w1[j].T)
        out = out.index_add(0, tok, gates[tok, which][:, None] * (a.square() @ w2[j].T))
    y = out.view(b, t, c) + st["residual"].double()
    aux = 0.01 * e * ((chosen.double().mean(0) / k) * p.mean(0)).sum()
    grads = torch.autograd.grad([y, aux], [x, router, w1, w2], [st["dy"].double(), torch.ones_like(aux)])
    return [y.detach(), aux.detach()] + list(grads)


# Polar-Express coefficients of the quintic iteration, as the optimizer applies them
_POLAR = [(8.156554524902461, -22.48329292557795, 15.878769915207462), (4.042929935166739, -2.808917465908714, 0.5000178451051316),
          (3.8916678022926607, -2.772484153217685, 0.5060648178503393), (3.285753657755655, -2.3681294933425376, 0.46449024233003106),
          (2.3465413258596377, -1.7097828382687081, 0.42323551169305323)]


def _exact_newton_schulz(case, st):
    x = st["x"].double()
    for a, b, c in _POLAR:
        if case["r"] > case["c"]:
            g = x.mT @ x
            x = a * x + x @ (b * g + c * (g @ g))
        else:
            g = x @ x.mT
            x = a * x + (b * g + c * (g @ g)) @ x
    return x


def _exact_decode(case, st):
    b, t = st["tokens"].shape
    h, d = case["heads"], case["width"] // case["heads"]
    cos, sin = _rotary(t, d)
    marks = torch.where(st["tokens"] == 0, torch.arange(t, device="cuda"), 0)
    ds = torch.cummax(marks, 1).values
    x = _norm64(st["wte"].double()[st["tokens"]])
    x0 = x
    for w in st["layers"]:
        x = x + 0.05 * x0
        n = _norm64(x)
        q, k, v = ((n @ w[key].double().T).view(b, t, h, d) for key in ("q", "k", "v"))
        y = torch.stack([_attend64(q[j], k[j], v[j], cos, sin, 1.0 / math.sqrt(d), ds[j], 0) for j in range(b)])
        x = x + y.reshape(b, t, -1) @ w["o"].double().T
        x = x + F.relu(_norm64(x) @ w["fc"].double().T).square() @ w["proj"].double().T
    return 15.0 * torch.tanh(_norm64(x[:, -1]) @ st["head"].double().T / 15.0)


_EXACT = dict(attention=_exact_attention, mlp=_exact_mlp, norm=_exact_norm, head=_exact_head, moe=_exact_moe,
              newton_schulz=_exact_newton_schulz, decode=_exact_decode)


def exact(case, seed):
    return _EXACT[case["kind"]](case, _INPUTS[case["kind"]](case, seed))
