"""The attention backward's scratch: asked for only where it fits, and the gradients do not depend on whether it was had."""
import math
import types

import pytest
import torch


def _fake_memory(monkeypatch, total, reserved, allocated, capturing=False):
    asked = []
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: capturing)
    monkeypatch.setattr(torch.cuda, "get_device_properties", lambda device=None: types.SimpleNamespace(total_memory=total))
    monkeypatch.setattr(torch.cuda, "memory_stats",
                        lambda device=None: asked.append("cache") or {"reserved_bytes.all.current": reserved, "allocated_bytes.all.current": allocated})
    return asked


@pytest.mark.parametrize("mb,total,reserved,allocated,capturing,fits,asks", [
    (255, 0, 0, 0, False, True, 0),                                                   # small: tried at once
    (256, 2304, 0, 0, False, True, 1), (256, 2303, 0, 0, False, False, 1),            # the device's room, less what others may hold
    (512, 1000, 900, 388, False, True, 1), (512, 1000, 900, 389, False, False, 1),    # the allocator's cache
    (512, 3000, 1000, 800, False, False, 1),                                          # both together would mean giving the cache back
    (512, 0, 0, 0, True, True, 0), (4097, 90000, 0, 0, False, False, 0)])
def test_large_scratch_is_asked_for_only_where_it_fits(monkeypatch, mb, total, reserved, allocated, capturing, fits, asks):
    from them_bones_b200.ops import attention_bwd as AB
    tried = []
    asked = _fake_memory(monkeypatch, total << 20, reserved << 20, allocated << 20, capturing)
    monkeypatch.setattr(torch, "empty", lambda n, dtype, device: tried.append(n) or "scratch")
    assert (AB._ds_scratch(mb << 20, "cuda") == "scratch") == fits and (tried == [mb << 20]) == fits and len(asked) == asks


@pytest.mark.gpu
@pytest.mark.parametrize("b,t,h,d,window,docs", [(1, 1, 1, 128, 0, False), (2, 128, 3, 64, 0, False), (1, 129, 2, 128, 0, True), (2, 700, 2, 64, 256, True),
                                                 (1, 1664, 2, 128, 512, False), (3, 2048, 5, 128, 0, True), (2, 5000, 3, 64, 0, True),
                                                 (1, 4999, 2, 128, 128, False)])
def test_same_bits_with_and_without(monkeypatch, b, t, h, d, window, docs):
    from them_bones_b200 import ops
    from them_bones_b200.ops import _lib as L
    from them_bones_b200.ops import attention_bwd as AB
    from them_bones_b200.ref import functional as RF
    torch.manual_seed(t + d + window)
    qkv = torch.randn(b, t, 3 * h * d, device="cuda", dtype=torch.bfloat16)
    ds = RF.doc_start_positions(torch.randint(0, 600, (b, t), device="cuda"), 0) if docs else None
    cos, sin = (v.bfloat16().float() for v in RF.rotary_tables(t, d, 10000.0, device="cuda"))
    g = torch.randn(b, t, h * d, device="cuda", dtype=torch.bfloat16)

    def grad(route):
        ops.COUNTS[route] = 0
        x = qkv.detach().requires_grad_(True)
        ops.attention(x, cos, sin, h, d, 1.0 / math.sqrt(d), ds, window).backward(g)
        assert ops.COUNTS[route] == 1
        return x.grad

    stored = grad("attention_dq_stored")
    monkeypatch.setattr(AB, "DS_ASK", 0)
    monkeypatch.setattr(AB, "_fits", lambda nbytes, device: False)
    again = grad("attention_dq_again")
    torch.cuda.synchronize()
    L.check_error_word()
    # the same bf16 dS (S, P and dP of one pair of tiles are the same sums in either orientation) and the same sums over key tiles
    assert torch.equal(stored, again)
