"""A CTA's first item is its own number, the others are drawn: calls with fewer items than SMs, as many, a few more, and first items
whose keys begin behind the first tile."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _check(b, t, h, d, ds, window):
    from them_bones_b200 import ops
    from them_bones_b200.ops import _lib as L
    from them_bones_b200.ref import functional as RF
    g = torch.Generator(device="cuda").manual_seed(b + t)
    qkv = torch.randn(b, t, 3 * h * d, generator=g, device="cuda").bfloat16()
    cos, sin = (v.bfloat16().float() for v in RF.rotary_tables(t, d, 10000.0, device="cuda"))
    with torch.no_grad():
        y = ops.attention(qkv, cos, sin, h, d, 1.0 / math.sqrt(d), ds, window)
        assert torch.equal(ops.attention(qkv, cos, sin, h, d, 1.0 / math.sqrt(d), ds, window), y)
        want = RF.attention(qkv.float(), cos, sin, h, d, 1.0 / math.sqrt(d), ds, window)
    # q, k and the probabilities rounded to bf16 (2^-9 each), a sum of bf16 values rounded once more; row by row, so that no item is lost among others
    rel = (y.float() - want).view(b * t, -1).norm(dim=1) / want.view(b * t, -1).norm(dim=1)
    assert float(rel.max()) < 3e-2 and float((y.float() - want).norm() / want.norm()) < 1.5e-2
    L.check_error_word()


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("more", [None, -1, 0, 1, 2])
def test_items_against_sms(more, d):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    _check(1 if more is None else sms + more, 90, 1, d, None, 0)


@pytest.mark.parametrize("b,h,d", [(1, 1, 64), (2, 3, 128), (40, 2, 64)])
@pytest.mark.parametrize("window", [0, 256])
def test_first_items_that_begin_behind_the_first_tile(b, h, d, window):
    from them_bones_b200.ref import functional as RF
    t = 700
    ids = torch.ones(b, t, dtype=torch.int64, device="cuda")
    ids[:, 300] = 0
    ids[::2, 513] = 0
    _check(b, t, h, d, RF.doc_start_positions(ids, 0), window)
