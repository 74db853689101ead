"""The loss head's row weights of either sign, against 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,c,vocab,padded,n_aux", [(33, 64, 264, 288, 0), (40, 64, 1000, 1024, 2), (130, 128, 8192, 8192, 1), (20, 64, 65544, 65568, 1)])
def test_negative_row_weights(m, c, vocab, padded, n_aux):
    """Weights are absolute and may be negative (an advantage, a penalty): the loss and its gradient are linear in them."""
    from them_bones_b200 import ops
    from them_bones_b200.ops import _lib as L
    g = torch.Generator(device="cuda").manual_seed(m + vocab)
    x = torch.randn(m, c, generator=g, device="cuda").bfloat16().requires_grad_(True)
    w = (torch.randn(padded, c, generator=g, device="cuda") * 2 / c ** 0.5).bfloat16().requires_grad_(True)
    targets = [torch.randint(0, vocab, (m,), generator=g, device="cuda") for _ in range(1 + n_aux)]
    targets[0][::7] = -1
    weights = [torch.randn(m, generator=g, device="cuda") for _ in targets]
    weights[0][3] = 0
    if n_aux:
        targets[1][5], weights[0][5], weights[1][5] = (targets[0][5] + 1) % vocab, 1.0, -1.0       # the probability terms cancel
        for wk in weights[2:]:
            wk[5] = 0
    loss = ops.lmhead_loss(x, w, targets[0], vocab, 15.0, row_weights=weights[0], aux=list(zip(targets[1:], weights[1:])))
    dx, dw = torch.autograd.grad(loss, [x, w])
    torch.cuda.synchronize()
    L.check_error_word()
    x64, w64 = x.detach().double().requires_grad_(True), w.detach().double().requires_grad_(True)
    z = 15 * torch.tanh(x64 @ w64[:vocab].T / 15)
    lse = torch.logsumexp(z, -1)
    want = 0
    for t, a in zip(targets, weights):
        want = want + (torch.where(t >= 0, lse - z.gather(1, t.clamp_min(0)[:, None])[:, 0], 0.0) * a.double()).sum()
    ex, ew = torch.autograd.grad(want, [x64, w64])
    rel = lambda a, b: float((a.double() - b).norm() / b.norm())  # noqa: E731
    # logits are bf16 (2^-9), the logits' gradient and the results are rounded once more each; the loss is a sum of both signs
    scale = sum(float((lse.detach().abs() * a.abs()).sum()) for a in weights)
    assert abs(float(loss) - float(want)) < 4e-3 * scale
    assert rel(dx, ex) < 1e-2, rel(dx, ex)
    assert rel(dw[:vocab], ew[:vocab]) < 1e-2 and not dw[vocab:].any()
