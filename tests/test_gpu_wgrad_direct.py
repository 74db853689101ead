"""Weight gradients that the GEMM writes as bf16, and the bf16 MLP's one call each way, against 64-bit sums."""
import pytest
import torch

pytestmark = pytest.mark.gpu
# a bf16 result of fp32 sums: half a unit of the last of 8 bits, 2^-9 = 0.002 at most; the MLP's gradients see h and dpre rounded too
ROUNDED, CHAIN = 2.5e-3, 8e-3


def _rel(a, b):
    return float((a.double() - b).norm() / b.norm().clamp_min(1e-30))


@pytest.mark.parametrize("m,n,k", [(1, 8, 8), (40, 24, 264), (1000, 256, 1024), (2048, 256, 256), (2049, 256, 256), (4100, 1280, 1280), (4104, 1280, 1280), (333, 1288, 520)])
def test_weight_gradient(m, n, k):
    from them_bones_b200.ops import cuda as C
    g = torch.Generator(device="cuda").manual_seed(m + n)
    dy, x = (torch.randn(m, c, generator=g, device="cuda").bfloat16() for c in (n, k))
    w = torch.empty(n, k, device="cuda", dtype=torch.bfloat16)
    want = dy.double().T @ x.double()
    (got,) = C._wgrad(dy, x, (w,))
    assert got.dtype == torch.bfloat16 and got.shape == w.shape and _rel(got, want) < ROUNDED
    if n % 3 == 0:
        parts = C._wgrad(dy, x, tuple(w.split(n // 3)))
        assert torch.equal(torch.cat(parts), got) and len({p.untyped_storage().data_ptr() for p in parts}) == 3


def test_an_empty_batch_has_a_zero_gradient():
    from them_bones_b200.ops import cuda as C
    w = torch.empty(64, 32, device="cuda", dtype=torch.bfloat16)
    (got,) = C._wgrad(torch.empty(0, 64, device="cuda", dtype=torch.bfloat16), torch.empty(0, 32, device="cuda", dtype=torch.bfloat16), (w,))
    assert torch.equal(got, torch.zeros_like(got))


@pytest.mark.parametrize("m,c,f,n,residual,slab", [(1, 64, 128, 64, True, False), (130, 256, 1024, 256, False, False), (777, 256, 512, 320, True, True),
                                                   (2500, 128, 256, 128, True, False)])
def test_mlp(m, c, f, n, residual, slab):
    from them_bones_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(m)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()  # noqa: E731
    x, w1, w2 = rnd(m, c).requires_grad_(), (rnd(f, c) / c ** 0.5).requires_grad_(), (rnd(n, f) / f ** 0.5).requires_grad_()
    r, dy = rnd(m, n) if residual else None, rnd(m, n)
    if slab:                                      # one weight accumulates into the optimizer's slab, the other's gradient comes back
        w1.main_grad = torch.ones(f, c, device="cuda")
    y = ops.mlp(x, w1, w2, residual=r)
    gx, g1, g2 = torch.autograd.grad(y, [x, w1, w2], dy, allow_unused=True)
    X, W1, W2, DY = (t.detach().double() for t in (x, w1, w2, dy))
    a = (X @ W1.T).clamp_min(0)
    want = a.square() @ W2.T + (r.double() if residual else 0)
    dpre = (DY @ W2) * 2 * a
    if slab:
        assert g1 is None
        g1 = w1.main_grad - 1
    assert _rel(y.detach(), want) < CHAIN and _rel(gx, dpre @ W1) < CHAIN and _rel(g1, dpre.T @ X) < CHAIN and _rel(g2, DY.T @ a.square()) < CHAIN
