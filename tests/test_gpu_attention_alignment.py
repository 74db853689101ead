"""Attention on tensors that begin anywhere in their storage: what the kernels need aligned is copied, whatever the length."""
import math

import pytest
import torch


def _shifted(x, by):
    """The same values in a storage whose first element is ``by`` elements before."""
    out = torch.empty(x.numel() + by, dtype=x.dtype, device=x.device)[by:].view(x.shape)
    return out.copy_(x)


def test_aligned_copies_only_what_needs_it():
    from them_bones_b200.ops.attention_native import _aligned
    x = torch.randn(40)
    assert _aligned(x) is x and _aligned(x[4:]).data_ptr() == x.data_ptr() + 16
    for y in (x[1:], x[::2], x.view(4, 10).T):
        z = _aligned(y)
        assert z.data_ptr() % 16 == 0 and z.is_contiguous() and torch.equal(z, y)


def _run(fn, qkv, cos, sin, h, d, ds, window, g):
    x = qkv.detach().requires_grad_(True)
    y = fn(x, cos, sin, h, d, 1.0 / math.sqrt(d), ds, window)
    y.backward(g)
    return y.detach(), x.grad


@pytest.mark.gpu
@pytest.mark.parametrize("b,t,h,d,window", [(2, 128, 3, 64, 0), (2, 333, 2, 128, 128), (1, 256, 1, 64, 128), (2, 256, 2, 128, 0), (2, 200, 2, 64, 0), (1, 77, 2, 128, 0)])
def test_shifted_tensors_give_the_same_bits(b, t, h, d, window):
    from them_bones_b200 import ops
    from them_bones_b200.ops import _lib as L
    from them_bones_b200.ref import functional as RF
    torch.manual_seed(t + d)
    qkv = torch.randn(b, t, 3 * h * d, device="cuda", dtype=torch.bfloat16)
    g = torch.randn(b, t, h * d, device="cuda", dtype=torch.bfloat16)
    cos, sin = (v.bfloat16().float() for v in RF.rotary_tables(t, d, 10000.0, device="cuda"))
    ds = RF.doc_start_positions(torch.randint(0, 60, (b, t), device="cuda"), 0).int()
    want = _run(ops.attention, qkv, cos, sin, h, d, ds, window, g)
    from them_bones_b200.ops import registry as R
    for fn in [ops.attention] + ([R.attention] if d == 128 else []):         # the custom ops cover 128-wide heads
        got = _run(fn, _shifted(qkv, 1), _shifted(cos, 1), _shifted(sin, 3), h, d, _shifted(ds, 1), window, _shifted(g, 3))
        torch.cuda.synchronize()
        L.check_error_word()
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])


@pytest.mark.gpu
def test_entry_points_refuse_what_they_cannot_load():
    """The C entries check the addresses their 16-byte accesses need before anything is launched."""
    from ctypes import c_int, c_longlong

    from them_bones_b200.ops import _lib as L
    t, h, d = 128, 1, 64
    qkv = torch.zeros(t * 3 * h * d + 1, device="cuda", dtype=torch.bfloat16)
    qk, tab = torch.zeros(t, 2 * h * d, device="cuda", dtype=torch.bfloat16), torch.zeros(t * d // 2 + 1, device="cuda")
    for x, c in ((qkv[1:], tab), (qkv, tab[1:])):
        with pytest.raises(RuntimeError, match="-3"):
            L.call("bones_rope_qknorm_fwd", L.ptr(x), L.ptr(c), L.ptr(tab), L.ptr(qk), L.ptr(None), c_longlong(t), c_int(t), c_int(h), c_int(d), L.stream())
    torch.cuda.synchronize()
    assert not qk.any()
