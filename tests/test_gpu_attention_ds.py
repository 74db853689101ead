"""dQ from the stored dS against dQ from a second pass over S and dP: the same bf16 dS enters the same products, tile by tile."""
import math

import pytest
import torch

CASES = [(1, 1, 1, 128, 0, False), (2, 128, 3, 64, 0, False), (1, 129, 2, 128, 0, True), (2, 700, 2, 64, 256, True), (1, 1664, 2, 128, 512, False),
         (3, 2048, 5, 128, 0, True), (2, 5000, 3, 64, 0, True), (1, 4999, 2, 128, 128, False)]


@pytest.mark.parametrize("t,window", [(1, 0), (128, 0), (129, 128), (1000, 256), (4096, 512), (640, 4096)])
def test_number_of_tile_pairs(t, window):
    from them_bones_b200.ops.attention_bwd import ds_tiles
    n, w = -(-t // 128), window // 128
    assert ds_tiles(t, window) == sum(1 for q in range(n) for k in range(q + 1) if w == 0 or q - k < w)


def test_scratch_is_optional(monkeypatch):
    from them_bones_b200.ops import attention_bwd as AB
    assert AB._ds_scratch(4096, "cpu").numel() == 4096 and AB._ds_scratch(AB.DS_LIMIT + 1, "cpu") is None

    def none_left(*args, **kwargs):
        raise torch.OutOfMemoryError("no memory")

    monkeypatch.setattr(torch, "empty", none_left)
    assert AB._ds_scratch(4096, "cpu") is None


@pytest.mark.gpu
@pytest.mark.parametrize("b,t,h,d,window,docs", CASES)
def test_both_routes_agree(monkeypatch, b, t, h, d, window, docs):
    from them_bones_b200 import ops
    from them_bones_b200.ops import _lib as L
    from them_bones_b200.ops import attention_bwd as AB
    from them_bones_b200.ref import functional as RF
    torch.manual_seed(t + d + window)
    qkv = torch.randn(b, t, 3 * h * d, device="cuda", dtype=torch.bfloat16)
    ds = RF.doc_start_positions(torch.randint(0, 600, (b, t), device="cuda"), 0) if docs else None
    cos, sin = (v.bfloat16().float() for v in RF.rotary_tables(t, d, 10000.0, device="cuda"))
    g = torch.randn(b, t, h * d, device="cuda", dtype=torch.bfloat16)

    def grad(limit):
        monkeypatch.setattr(AB, "DS_LIMIT", limit)
        x = qkv.detach().requires_grad_(True)
        ops.attention(x, cos, sin, h, d, 1.0 / math.sqrt(d), ds, window).backward(g)
        return x.grad

    junk = torch.full((b * h * AB.ds_tiles(t, window) * 8192,), float("nan"), device="cuda")   # what the scratch is cut from
    del junk
    stored, again = grad(1 << 40), grad(0)
    torch.cuda.synchronize()
    L.check_error_word()
    assert torch.isfinite(stored).all()
    a = h * d
    assert torch.equal(stored[..., a:], again[..., a:])            # dK, dV come from the same kernel
    # dQ: two fp32 sums of the same products; were S or dP to differ in a last bit, bf16 roundings of dS would (2^-9 each, in few
    # elements), and those of dQ.  (They do not: test_gpu_attention_scratch.py.)
    err = (stored[..., :a].float() - again[..., :a].float()).norm() / again[..., :a].float().norm().clamp_min(1e-12)
    assert t == 1 or float(err) < 2 ** -8, float(err)
