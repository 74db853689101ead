"""The decode step's projections with the sequences as MMA rows, against 64-bit sums."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu
I = ctypes.c_int


@pytest.mark.parametrize("b,n,k,nt,splits,ctas,epi", [
    (1, 16, 128, 16, 1, 0, 0), (64, 3840, 1280, 32, 1, 0, 0), (17, 240, 640, 24, 1, 3, 1), (8, 64, 256, 64, 1, 0, 2), (64, 1280, 1280, 16, 1, 0, 2),
    (33, 640, 384, 40, 1, 5, 2), (64, 1280, 5120, 40, 4, 0, 2), (9, 96, 1152, 48, 2, 0, 2), (50, 128, 1024, 64, 8, 0, 1), (64, 128, 640, 64, 2, 0, 2),
    (40, 48, 896, 16, 4, 0, 0), (64, 8192, 1280, 64, 1, 37, 3), (5, 1024, 256, 32, 1, 2, 3), (64, 32, 128, 32, 1, 0, 1)])
def test_projection_epilogues(b, n, k, nt, splits, ctas, epi):
    from them_bones_b200.ops import _lib as L
    g = torch.Generator(device="cuda").manual_seed(b + n)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()  # noqa: E731
    x, w, res, x0 = rnd(b, k), rnd(n, k) * 0.05, rnd(b, n), rnd(b, n)
    out = torch.full((b, n), float("nan"), device="cuda", dtype=torch.bfloat16)
    ssq_in = torch.rand(7, b, generator=g, device="cuda") * k
    ssq_out = torch.full((n // nt, b), float("nan"), device="cuda")
    ma, mb = torch.tensor([0.9], device="cuda"), torch.tensor([0.3], device="cuda")
    scaled = epi != 2
    L.call("bones_decode_rows", L.ptr(x), L.ptr(w), L.ptr(out), I(b), I(n), I(k), I(nt), I(splits), I(ctas), I(epi), L.ptr(ssq_in if scaled else None), I(7),
           L.ptr(res), L.ptr(x0 if epi == 2 else None), L.ptr(ma), L.ptr(mb), L.ptr(ssq_out if epi == 2 else None), ctypes.c_float(15.0), L.ptr(w), ctypes.c_longlong(2 * w.numel()), I(0), L.stream())
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


@pytest.mark.parametrize("b,n_embd,steps", [(17, 1024, 5), (64, 1024, 70), (3, 1024, 200), (64, 256, 5), (33, 1152, 3)])
def test_step_matches_the_pytorch_route(b, n_embd, steps):
    """The whole step on these kernels, and the attention's rounds of 32 and 64 keys across documents."""
    from them_bones_b200.config import GPTConfig
    from them_bones_b200.models.gpt import GPT
    from them_bones_b200.utils import decode as D
    torch.manual_seed(b)
    cfg = GPTConfig(sequence_len=256, vocab_size=1024, n_layer=2, n_head=n_embd // 128, n_embd=n_embd, head_dim=128, doc_mask=True)
    with torch.device("cuda"):
        model = GPT(cfg)
    model.init_weights()
    for p in model.parameters():
        if p.dim() == 2:
            torch.nn.init.normal_(p, std=0.03)
    model.cast_compute(torch.bfloat16).eval()
    toks = torch.randint(1, 1000, (b, steps), device="cuda")
    toks[:, 0] = 0
    toks[::3, steps // 3] = 0
    toks[0, steps - 1] = 0
    out = torch.cat([toks, torch.zeros(b, 1, dtype=torch.int64, device="cuda")], 1)
    with torch.no_grad():
        dec = D.NativeDecoder(model, D.KVCache(model, b, steps + 1), toks[:, 0], out, prompt_len=steps)
        dec.run(steps)
        ref = D._forward_cached(model, toks, D.KVCache(model, b, steps + 1))
    D.L_check()
    assert dec.fused and dec.rows == D.use_rows(b, n_embd, n_embd, 4 * n_embd, dec.sms)
    got = dec.last_logits.float()
    # bf16 activations through two layers, rounded at other places by the two routes
    assert float((got - ref).norm() / ref.norm()) < 3e-2
