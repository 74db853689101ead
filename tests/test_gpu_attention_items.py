"""The persistent forward over many work items a CTA: items of one tile, of two, of one to nine in documents, both head widths; and
the same bits in every call, whichever CTA takes which item."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("b,t,h,d,window,docs", [(220, 100, 4, 128, 0, False), (64, 640, 3, 64, 128, True), (40, 520, 4, 128, 256, False), (24, 1100, 8, 128, 0, True),
                                                 (37, 256, 4, 64, 0, True), (1, 128, 1, 128, 0, False)])
def test_many_items(b, t, h, d, window, docs):
    from them_bones_b200 import ops
    from them_bones_b200.ops import _lib as L
    from them_bones_b200.ref import functional as RF
    torch.manual_seed(b)
    qkv = torch.randn(b, t, 3 * h * d, device="cuda", dtype=torch.bfloat16)
    ds = RF.doc_start_positions(torch.randint(0, 300, (b, t), device="cuda"), 0) if docs else None
    cos, sin = (v.bfloat16().float() for v in RF.rotary_tables(t, d, 10000.0, device="cuda"))
    run = lambda: ops.attention(qkv, cos, sin, h, d, 1.0 / math.sqrt(d), ds, window)  # noqa: E731
    with torch.no_grad():
        y = run()
        for _ in range(5):
            assert torch.equal(run(), y)
        for j in {0, b // 2, b - 1}:              # a sequence at a time: the fp32 scores of a batch would be tens of GB
            want = RF.attention(qkv[j:j + 1].float(), cos, sin, h, d, 1.0 / math.sqrt(d), ds[j:j + 1] if docs else None, window)
            # q, k and the probabilities rounded to bf16 (2^-9 each), a sum of bf16 values rounded once more
            assert float((y[j:j + 1].float() - want).norm() / want.norm()) < 1.5e-2
    L.check_error_word()
