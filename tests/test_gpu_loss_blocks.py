"""Scoring in blocks of rows: the same likelihoods whatever the block, and scratch that does not grow with the rows."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_blocks_give_the_same_likelihoods_and_bound_the_scratch(monkeypatch):
    from them_bones_b200 import ops
    from them_bones_b200.ops import _lib as L
    from them_bones_b200.ops import cuda as C
    g = torch.Generator(device="cuda").manual_seed(2)
    m, c, v = 2000, 64, 8192
    x, w = torch.randn(m, c, generator=g, device="cuda").bfloat16(), (torch.randn(v, c, generator=g, device="cuda") * 0.25).bfloat16()
    tg = torch.randint(-1, v, (m,), generator=g, device="cuda")
    whole, peaks = None, []
    for rows in (4096, 1999, 512, 128):
        monkeypatch.setattr(C, "LOSS_ROWS", rows)
        torch.cuda.synchronize()
        torch.cuda.reset_peak_memory_stats()
        before = torch.cuda.memory_allocated()
        nll = ops.lmhead_loss(x, w, tg, v, 15.0, reduction="none")
        peaks.append(torch.cuda.max_memory_allocated() - before)
        L.check_error_word()
        whole = nll if whole is None else whole
        assert torch.equal(nll, whole)
    part = 2 * (v // 256) * 4                       # bytes of partial sums a row
    assert peaks[0] > m * part and peaks[3] < peaks[0] - (m - 128) * part + 65536
