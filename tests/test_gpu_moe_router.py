"""The fused MoE router against the PyTorch statement, and the stacked quantiser against one call per matrix."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,e,k,aux_w,z_w", [(1, 2, 2, 0.01, 0.0), (127, 16, 2, 0.01, 1e-3), (128, 64, 1, 0.01, 0.0), (1001, 16, 2, 0.02, 0.0),
                                             (4096, 5, 1, 0.0, 1e-3)])
def test_router_matches_statement(n, e, k, aux_w, z_w):
    from them_bones_b200 import ops
    from them_bones_b200.ref import functional as RF
    torch.manual_seed(n + e)
    h = torch.randn(n, 256, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    router = (0.1 * torch.randn(e, 256, device="cuda")).bfloat16().requires_grad_(True)
    dg = torch.randn(n, k, device="cuda")
    idx, gates, aux, stats = ops.moe_router(h, router, k, aux_w, z_w)
    dh, dr = torch.autograd.grad([gates, aux], [h, router], [dg, torch.tensor(3.0, device="cuda")])
    h64, r64 = h.detach().double().requires_grad_(True), router.detach().double().requires_grad_(True)
    logits = h64 @ r64.T
    top = logits.topk(min(e, k + 1), dim=1).values.detach()
    clear = ((top[:, :-1] - top[:, 1:]).min(1).values > 1e-4) if e > 1 else torch.ones(n, dtype=torch.bool, device="cuda")
    p = torch.softmax(logits, -1)
    assert torch.equal(idx[clear], p.topk(k, dim=-1).indices[clear])
    v = p.gather(1, idx)
    g64 = v / v.sum(1, keepdim=True) if k == 2 else v
    f = torch.nn.functional.one_hot(idx, e).sum(1).double().mean(0) / k
    lb, z = e * (f * p.mean(0)).sum(), torch.logsumexp(logits, -1).square().mean()
    a64 = aux_w * lb + z_w * z
    dh64, dr64 = torch.autograd.grad([g64, a64], [h64, r64], [dg.double(), torch.tensor(3.0, device="cuda", dtype=torch.float64)])
    rel = lambda a, b: float((a.double() - b).norm() / b.norm().clamp_min(1e-30))  # noqa: E731
    # fp32 soft-max and sums: a few 2^-23 per value; the gradients pass through one bf16 rounding each (2^-9)
    assert rel(gates, g64) < 1e-5 and rel(aux, a64) < 1e-5
    assert rel(stats, torch.cat([torch.stack([lb, z]), f])) < 1e-5
    assert rel(dh, dh64) < 8e-3 and rel(dr, dr64) < 8e-3
    again = ops.moe_router(h, router, k, aux_w, z_w)
    assert torch.equal(again[3], stats) and torch.equal(again[2], aux)
    with torch.no_grad():
        i2, g2, a2, s2 = ops.moe_router(h, router, k, aux_w, z_w, want_aux=False)
    assert a2 is None and s2 is None and torch.equal(i2, idx) and torch.equal(g2, gates)
    if n > 1:                                  # rows without a number choose what argmax on them chooses
        bad = h.detach().clone()
        bad[0] = float("nan")
        ib = ops.moe_router(bad, router, k, aux_w, z_w)[0]
        ref = RF.moe_route(torch.full((1, e), float("nan"), device="cuda"), k)[1]
        assert torch.equal(ib[:1], ref) and torch.equal(ib[1:], idx[1:])


@pytest.mark.parametrize("e,r,c,group_r,group_c", [(2, 128, 128, 128, 256), (3, 160, 256, 224, 128), (5, 2560, 1280, 128, 256)])
def test_stacked_quantiser_equals_one_call_per_matrix(e, r, c, group_r, group_c):
    from them_bones_b200.ops import mxfp8 as MX
    torch.manual_seed(e)
    x = torch.randn(e, r, c, device="cuda", dtype=torch.bfloat16) * torch.logspace(-2, 2, e, device="cuda").bfloat16()[:, None, None]
    stacked = MX.quant2(x, col=True, group_r=group_r, group_c=group_c)
    for j in range(e):
        for got, want in zip(stacked, MX.quant2(x[j], col=True, group_r=group_r, group_c=group_c)):
            assert torch.equal(got[j], want)
