"""Backward of the loss head under the forms of autograd that hand it something other than a plain scalar."""
import pytest
import torch


class _Spy(torch.autograd.Function):
    """Its backward asks what the loss head's asks of the incoming gradient."""
    seen = []

    @staticmethod
    def forward(ctx, x):
        return x.sum()

    @staticmethod
    def backward(ctx, d):
        from them_bones_b200.ops.cuda import _by_address
        _Spy.seen.append(_by_address(d))
        return d.expand(3)


def test_which_gradients_a_kernel_may_take_by_address():
    x, s = torch.randn(3, requires_grad=True), torch.tensor(2.0, requires_grad=True)
    _Spy.seen.clear()
    torch.autograd.grad(_Spy.apply(x), x)
    torch.autograd.grad(_Spy.apply(x), x, create_graph=True)
    torch.autograd.grad(_Spy.apply(x) * s, x, create_graph=True)
    torch.autograd.grad(_Spy.apply(x), x, torch.arange(4.0), is_grads_batched=True)
    assert _Spy.seen == [True, True, False, False]


@pytest.mark.gpu
def test_batched_and_recorded_gradients():
    from them_bones_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(1)
    x = torch.randn(40, 64, generator=g, device="cuda").bfloat16().requires_grad_(True)
    w = (torch.randn(512, 64, generator=g, device="cuda") * 0.2).bfloat16().requires_grad_(True)
    tg = torch.randint(0, 512, (40,), generator=g, device="cuda")
    plain = torch.autograd.grad(ops.lmhead_loss(x, w, tg, 512, 15.0), [x, w])
    scales = torch.tensor([1.0, 0.0, -2.0], device="cuda")
    for a, b in zip(torch.autograd.grad(ops.lmhead_loss(x, w, tg, 512, 15.0), [x, w], scales, is_grads_batched=True), plain):
        assert torch.equal(a, torch.stack([b, torch.zeros_like(b), -2 * b]))       # powers of two: exact in bf16
    s = torch.tensor(2.0, device="cuda", requires_grad=True)
    dx, dw = torch.autograd.grad(ops.lmhead_loss(x, w, tg, 512, 15.0) * s, [x, w], create_graph=True)
    assert torch.equal(dx, 2 * plain[0]) and torch.equal(dw, 2 * plain[1])
    (ds,) = torch.autograd.grad(dx.float().sum() + dw.float().sum(), s)            # the gradients are linear in the factor
    want = plain[0].double().sum() + plain[1].double().sum()
    size = plain[0].double().abs().sum() + plain[1].double().abs().sum()
    assert abs(float(ds) - float(want)) < 2 ** -7 * float(size)                    # a bf16 sum of up to 32768 terms
