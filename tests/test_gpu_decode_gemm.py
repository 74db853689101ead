"""The decode step's projections against 64-bit sums, and the fused step against the PyTorch cache route."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu
I = ctypes.c_int


@pytest.mark.parametrize("b,n,k,splits,epi", [(1, 128, 64, 1, 0), (16, 384, 1280, 4, 0), (17, 128, 576, 2, 1), (33, 256, 1280, 4, 2), (64, 1280, 5120, 8, 2),
                                              (65, 256, 128, 2, 1), (128, 640, 1280, 8, 3), (64, 1024, 1280, 1, 3), (5, 256, 512, 4, 2), (32, 256, 640, 8, 0), (64, 256, 1280, 16, 2),
                                              (37, 128, 1088, 16, 1), (3, 128, 1024, 16, 2), (9, 256, 640, 8, 0), (128, 128, 1024, 16, 2)])
def test_projection_epilogues(b, n, k, splits, epi):
    from them_bones_b200.ops import _lib as L
    g = torch.Generator(device="cuda").manual_seed(b + n)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()  # noqa: E731
    x, w, res, x0 = rnd(b, k), rnd(n, k) * 0.05, rnd(b, n), rnd(b, n)
    out = torch.full((b, n), float("nan"), device="cuda", dtype=torch.bfloat16)
    ssq_in = torch.rand(3, b, generator=g, device="cuda") * k
    ssq_out = torch.full((n // 128, b), float("nan"), device="cuda")
    ma, mb = torch.tensor([0.9], device="cuda"), torch.tensor([0.3], device="cuda")
    scaled = epi != 2
    L.call("bones_decode_gemm", L.ptr(x), L.ptr(w), L.ptr(out), I(b), I(n), I(k), I(splits), I(epi), L.ptr(ssq_in if scaled else None), I(3), L.ptr(res),
           L.ptr(x0 if epi == 2 else None), L.ptr(ma), L.ptr(mb), L.ptr(ssq_out if epi == 2 else None), ctypes.c_float(15.0), I(0), L.stream())
    torch.cuda.synchronize()
    L.check_error_word()
    acc = x.double() @ w.double().T
    if scaled:
        acc = acc * torch.rsqrt(ssq_in.double().sum(0) / k + 2.0 ** -23)[:, None]
    want = {0: acc, 1: acc.clamp_min(0).square(), 2: 0.9 * (acc + res.double()) + 0.3 * x0.double(), 3: 15 * torch.tanh(acc / 15)}[epi]
    # one bf16 rounding (two for the residual), the square doubles the accumulator's error
    assert float((out.double() - want).norm() / want.norm()) < 5e-3
    if epi == 2:
        assert torch.allclose(ssq_out.sum(0), out.float().square().sum(1), rtol=1e-5)


@pytest.mark.parametrize("b,steps,window", [(1, 20, 0), (3, 140, 128), (64, 5, 0), (100, 3, 0)])
def test_fused_step_matches_the_pytorch_route(b, steps, window):
    from them_bones_b200.config import GPTConfig
    from them_bones_b200.models.gpt import GPT
    from them_bones_b200.utils import decode as D
    torch.manual_seed(b)
    cfg = GPTConfig(sequence_len=256, vocab_size=1024, n_layer=3, n_head=2, n_embd=256, head_dim=128, doc_mask=True, attn_window=window, attn_long=(2,))
    with torch.device("cuda"):
        model = GPT(cfg)
    model.init_weights()
    for p in model.parameters():
        if p.dim() == 2:
            torch.nn.init.normal_(p, std=0.05)
    model.cast_compute(torch.bfloat16).eval()
    toks = torch.randint(1, 1000, (b, steps), device="cuda")
    toks[:, 0] = 0
    toks[0, steps // 2] = 0
    out = torch.zeros(b, steps + 1, dtype=torch.int64, device="cuda")
    out[:, :steps] = toks
    with torch.no_grad():
        cache = D.KVCache(model, b, steps + 1)
        dec = D.NativeDecoder(model, cache, toks[:, 0], out, prompt_len=steps)
        assert dec.fused
        dec.run(steps)
        ref = D._forward_cached(model, toks, D.KVCache(model, b, steps + 1))
    D.L_check()
    got = dec.last_logits.float()
    assert float((got - ref).norm() / ref.norm()) < 3e-2
    assert torch.equal(out[:, :steps], toks) and torch.equal(out[:, steps], got.argmax(-1))
    assert int(dec.pos) == steps and int(dec.ticket) == 0
