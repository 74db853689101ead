"""Attention at lengths around the 128-token tile, both head widths, against the fp32 statement; sequences of a batch do not
reach into one another."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return float((a.float() - b.float()).norm() / b.float().norm().clamp_min(1e-12))


@pytest.mark.parametrize("b,t,h,d,window", [(3, 1, 2, 128, 0), (2, 127, 1, 64, 0), (2, 128, 4, 64, 0), (3, 129, 2, 128, 256), (2, 300, 3, 64, 128),
                                            (2, 1023, 2, 128, 0), (1, 2047, 1, 64, 512)])
def test_ragged_lengths_and_head_widths(b, t, h, d, window):
    from them_bones_b200 import ops
    from them_bones_b200.ops import _lib as L
    from them_bones_b200.ref import functional as RF
    torch.manual_seed(t + d)
    packed = torch.randn(b * t * 3 * h * d + 8, device="cuda", dtype=torch.bfloat16)
    qkv = packed[8 if t % 128 == 0 else 1:][:b * t * 3 * h * d].view(b, t, 3 * h * d)     # ragged: not 16-byte aligned either
    idx = torch.randint(0, 60, (b, t), device="cuda")
    ds = RF.doc_start_positions(idx, 0)
    cos, sin = (v.bfloat16().float() for v in RF.rotary_tables(t, d, 10000.0, device="cuda"))
    g = torch.randn(b, t, h * d, device="cuda", dtype=torch.bfloat16)
    x = qkv.detach().requires_grad_(True)
    y = ops.attention(x, cos, sin, h, d, 1.0 / math.sqrt(d), ds, window)
    y.backward(g)
    xr = qkv.float().requires_grad_(True)
    yr = RF.attention(xr, cos, sin, h, d, 1.0 / math.sqrt(d), ds, window)
    yr.backward(g.float())
    torch.cuda.synchronize()
    L.check_error_word()
    # bf16 probabilities, outputs and gradients: 2^-9 per rounding, a few of them in a row
    assert _rel(y, yr) < 8e-3, _rel(y, yr)
    if t > 1:
        assert _rel(x.grad, xr.grad) < 1e-2, _rel(x.grad, xr.grad)
    if b > 1:
        bad = qkv.clone()
        bad[1] = float("nan")
        with torch.no_grad():
            y2 = ops.attention(bad, cos, sin, h, d, 1.0 / math.sqrt(d), ds, window)
        assert torch.equal(y2[0], y[0]) and (b < 3 or torch.equal(y2[2], y[2]))
