"""The MoE combine and its gradient by slot, against the PyTorch statement: dropped assignments, empty slots, residual."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k,e,cap,c,with_res,with_tok", [(1, 1, 2, 1, 8, False, True), (65, 2, 4, 20, 264, True, True), (300, 2, 16, 30, 1280, True, False),
                                                           (128, 3, 5, 128, 512, False, True)])
def test_combine_matches_statement(n, k, e, cap, c, with_res, with_tok):
    from them_bones_b200 import ops
    from them_bones_b200.ref import functional as RF
    g = torch.Generator(device="cuda").manual_seed(n)
    idx = torch.rand(n, e, generator=g, device="cuda").topk(k, dim=1).indices
    slot, tok = RF.moe_slots(idx, 1, n, e, cap)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()  # noqa: E731
    ys, res, dout = rnd(e * cap, c), rnd(n, c), rnd(n, c)
    gates = torch.rand(n, k, generator=g, device="cuda")
    ys.requires_grad_(True), gates.requires_grad_(True), res.requires_grad_(True)
    out = ops.moe_combine(ys, slot, gates, res if with_res else None, tok if with_tok else None)
    ins = [ys, gates] + ([res] if with_res else [])
    got = torch.autograd.grad(out, ins, dout)
    y64, g64 = ys.detach().double().requires_grad_(True), gates.detach().double().requires_grad_(True)
    yp = torch.cat([y64, y64.new_zeros(1, c)])
    want = (g64[..., None] * yp[slot]).sum(1)
    dy, dg = torch.autograd.grad(want, [y64, g64], dout.double())
    want = want.detach() + (res.detach().double() if with_res else 0)
    rel = lambda a, b: float((a.double() - b).norm() / b.norm().clamp_min(1e-30))  # noqa: E731
    assert rel(out, want) < 6e-3               # one or two bf16 roundings
    assert rel(got[0], dy) < 4e-3 and rel(got[1], dg) < 1e-5
    assert bool((got[0][tok == n] == 0).all()) and bool((got[1][slot == e * cap] == 0).all())
    if with_res:
        assert torch.equal(got[2], dout)


@pytest.mark.parametrize("n,k,c", [(1, 0, 8), (37, 3, 264), (64, 8, 128), (50, 9, 264), (5, 13, 1280), (3, 40, 64)])
def test_any_number_of_choices(n, k, c):
    """Up to eight choices a token keeps its slots in registers; any other number goes through the general form."""
    from them_bones_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(n + k)
    slots = n * k + 5
    perm = torch.randperm(slots, generator=g, device="cuda")[: n * k].view(n, k)
    slot = torch.where(torch.rand(n, k, generator=g, device="cuda") < 0.2, slots, perm)
    ys, dout = (torch.randn(m, c, generator=g, device="cuda").bfloat16() for m in (slots, n))
    gates = torch.rand(n, k, generator=g, device="cuda")
    ys.requires_grad_(True), gates.requires_grad_(True)
    out = ops.moe_combine(ys, slot, gates)
    dy, dg = torch.autograd.grad(out, [ys, gates], dout)
    yp = torch.cat([ys.detach().double(), torch.zeros(1, c, device="cuda", dtype=torch.float64)])
    want = (gates.detach().double()[..., None] * yp[slot]).sum(1)
    rel = lambda a, b: float((a.double() - b).norm() / b.norm().clamp_min(1e-30))  # noqa: E731
    assert rel(out.detach(), want) < 4e-3                      # one bf16 rounding
    wdg = (yp[slot] * dout.double()[:, None]).sum(-1)
    wdy = torch.zeros(slots + 1, c, device="cuda", dtype=torch.float64)
    wdy.index_add_(0, slot.reshape(-1), (gates.detach().double()[..., None] * dout.double()[:, None]).reshape(-1, c))
    assert rel(dg, wdg) < 1e-5 and rel(dy, wdy[:slots]) < 4e-3


def test_gradients_that_have_no_address():
    """Batched gradients, and gradients that are recorded (``create_graph``): the residual's is the incoming one, as an addition's,
    and the others are those of the kernel."""
    from them_bones_b200 import ops
    from them_bones_b200.ref import functional as RF
    slot, tok = RF.moe_slots(torch.rand(12, 4, device="cuda").topk(2, dim=1).indices, 1, 12, 4, 3)
    ys, res, dout = (torch.randn(n, 64, device="cuda").bfloat16() for n in (12, 12, 12))
    ys.requires_grad_(True), res.requires_grad_(True)
    gates = torch.rand(12, 2, device="cuda", requires_grad=True)
    out = ops.moe_combine(ys, slot, gates, res, tok)
    (g,) = torch.autograd.grad(out, res, torch.stack([dout, 2 * dout]), is_grads_batched=True, retain_graph=True)
    assert torch.equal(g, torch.stack([dout, 2 * dout]))
    plain = torch.autograd.grad(out, [ys, gates, res], dout, retain_graph=True)
    batched = torch.autograd.grad(out, [ys, gates, res], torch.stack([dout, -dout]), is_grads_batched=True, retain_graph=True)
    recorded = torch.autograd.grad(out, [ys, gates, res], dout.clone().requires_grad_(True), create_graph=True, retain_graph=True)
    rel = lambda a, b: float((a.float() - b.float()).norm() / b.float().norm())  # noqa: E731
    for p, b, r in zip(plain, batched, recorded):
        assert rel(b[0], p) < 2 ** -8 and rel(b[1], -p) < 2 ** -8 and rel(r.detach(), p) < 2 ** -8 and r.requires_grad       # one bf16 rounding each
    with torch.no_grad():
        fixed = ys.detach()
    (g,) = torch.autograd.grad(ops.moe_combine(fixed, slot, gates.detach(), res, tok), res, dout)
    assert torch.equal(g, dout)
