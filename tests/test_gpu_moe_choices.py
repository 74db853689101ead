"""Which router calls the fused kernels cover, and that the others keep their answers."""
import pytest
import torch


@pytest.mark.parametrize("n,c,e,k,dtype,ok", [(4, 64, 1, 1, "bfloat16", True), (4, 64, 1, 2, "bfloat16", False), (4, 64, 2, 2, "bfloat16", True),
                                              (4, 64, 4, 3, "bfloat16", False), (4, 64, 65, 2, "bfloat16", False), (0, 64, 4, 2, "bfloat16", False),
                                              (4, 60, 4, 2, "bfloat16", False), (4, 64, 4, 2, "float32", False)])
def test_what_the_fused_router_covers(n, c, e, k, dtype, ok):
    from them_bones_b200.ops import cuda as C
    assert C.moe_router_ok(torch.zeros(n, c, dtype=getattr(torch, dtype)), torch.zeros(e, c), k) == ok


@pytest.mark.gpu
def test_two_choices_among_one_expert():
    """More choices than experts: both go to the only one, with equal gates."""
    from them_bones_b200 import ops
    from them_bones_b200.ref import functional as RF
    torch.manual_seed(0)
    h = torch.randn(9, 64, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    router = torch.randn(1, 64, device="cuda", requires_grad=True)
    idx, gates, aux, stats = ops.moe_router(h, router, 2, 0.01, 1e-3)
    (gates.sum() + aux).backward()
    want = RF.moe_route(torch.zeros(9, 1, device="cuda"), 2)
    assert torch.equal(idx, want[1]) and torch.equal(gates.detach(), want[2]) and torch.isfinite(h.grad).all() and stats.shape == (3,)
