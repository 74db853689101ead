"""The loss head on logits statistics from the GEMM: losses and gradients against 64 bits, over row and vocabulary remainders."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _exact(x, w, tg, vocab, cap, weights, aux):
    x, w = x.detach().double().requires_grad_(True), w.detach().double().requires_grad_(True)
    z = cap * torch.tanh(x @ w[:vocab].T / cap)
    lse = torch.logsumexp(z, -1)
    nll = torch.where(tg >= 0, lse - z.gather(1, tg.clamp_min(0)[:, None])[:, 0], 0.0)
    loss = (nll * weights).sum()
    for t, a in aux:
        loss = loss + (torch.where(t >= 0, lse - z.gather(1, t.clamp_min(0)[:, None])[:, 0], 0.0) * a.double()).sum()
    return nll.detach(), loss.detach(), torch.autograd.grad(loss, [x, w])


@pytest.mark.parametrize("m,c,vocab,padded,n_aux,weighted", [(1, 64, 264, 288, 0, False), (31, 128, 1000, 1024, 2, False), (257, 256, 8192, 8192, 0, True),
                                                             (4100, 64, 8200, 8256, 1, False), (300, 1280, 65536, 65536, 0, False), (33, 64, 96, 96, 2, True)])
def test_loss_and_gradients(m, c, vocab, padded, n_aux, weighted):
    from them_bones_b200 import ops
    from them_bones_b200.ops import _lib as L
    g = torch.Generator(device="cuda").manual_seed(m + vocab)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    x = rnd(m, c).bfloat16().requires_grad_(True)
    w = (rnd(padded, c) * 2 / c ** 0.5).bfloat16().requires_grad_(True)
    draw = lambda: torch.where(torch.rand(m, generator=g, device="cuda") < 0.1, -1, torch.randint(0, vocab, (m,), generator=g, device="cuda"))  # noqa: E731
    tg = draw()
    tg[0] = vocab - 1
    weights = torch.rand(m, generator=g, device="cuda") if weighted else None
    aux = [(draw(), torch.rand(m, generator=g, device="cuda") / m) for _ in range(n_aux)]
    loss = ops.lmhead_loss(x, w, tg, vocab, 15.0, row_weights=weights, loss_div=2.0, aux=aux)
    dx, dw = torch.autograd.grad(loss, [x, w], torch.tensor(3.0, device="cuda"))
    nll = ops.lmhead_loss(x, w, tg, vocab, 15.0, reduction="none")
    total = ops.lmhead_loss(x, w, tg, vocab, 15.0, reduction="sum")
    torch.cuda.synchronize()
    L.check_error_word()
    ew = weights.double() if weighted else torch.full((m,), 0.5 / max(1, int((tg >= 0).sum())), device="cuda", dtype=torch.float64)
    enll, eloss, (edx, edw) = _exact(x, w, tg, vocab, 15.0, ew, aux)
    rel = lambda a, b: float((a.double() - b).norm() / b.norm().clamp_min(1e-30))  # noqa: E731
    # logits are bf16 (2^-9 of up to 15); the gradients add the rounding of the logits' gradient and their own
    assert rel(nll, enll) < 4e-3 and rel(loss, eloss) < 4e-3 and rel(total, enll.sum()) < 4e-3
    assert bool((nll[tg < 0] == 0).all()) and not nll.requires_grad
    assert rel(dx, 3 * edx) < 1e-2, rel(dx, 3 * edx)
    assert rel(dw[:vocab], 3 * edw[:vocab]) < 1e-2 and bool((dw[vocab:] == 0).all())


def test_all_targets_masked_gives_zero():
    from them_bones_b200 import ops
    x = torch.randn(40, 64, device="cuda").bfloat16().requires_grad_(True)
    w = torch.randn(512, 64, device="cuda").bfloat16().requires_grad_(True)
    loss = ops.lmhead_loss(x, w, torch.full((40,), -1, device="cuda"), 512, 15.0)
    dx, dw = torch.autograd.grad(loss, [x, w])
    assert float(loss) == 0.0 and not dx.any() and not dw.any()
