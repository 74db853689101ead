"""The decode step on the buffers a program hands it: token rows inside a larger tensor, of another layout or type."""
import pytest
import torch


def _model(n_embd=256, n_layer=2, mlp_ratio=4, **kw):
    from them_bones_b200.config import GPTConfig
    from them_bones_b200.models.gpt import GPT
    torch.manual_seed(3)
    cfg = GPTConfig(sequence_len=256, vocab_size=1024, n_layer=n_layer, n_head=n_embd // 128, n_embd=n_embd, head_dim=128, doc_mask=True, mlp_ratio=mlp_ratio, **kw)
    with torch.device("cuda"):
        model = GPT(cfg)
    model.init_weights()
    for p in model.parameters():
        if p.dim() == 2:
            torch.nn.init.normal_(p, std=0.05)
    return model.cast_compute(torch.bfloat16).eval()


def test_token_rows_that_the_last_kernel_addresses():
    from them_bones_b200.utils.decode import _token_rows
    cpu, big = torch.device("cpu"), torch.zeros(4, 9, dtype=torch.int64)
    assert _token_rows(big, 4, cpu) and _token_rows(big[:, :5], 4, cpu) and _token_rows(big[:, 3:], 4, cpu) and _token_rows(big[::2], 2, cpu)
    assert _token_rows(big[0, :5][None], 1, cpu)
    assert not _token_rows(big.T, 9, cpu) and not _token_rows(big[:, ::2], 4, cpu) and not _token_rows(big[:1].expand(4, 9), 4, cpu)
    assert not _token_rows(big.int(), 4, cpu) and not _token_rows(big, 3, cpu) and not _token_rows(big[0], 4, cpu)
    assert not _token_rows(big, 4, torch.device("meta"))


@pytest.mark.gpu
@pytest.mark.parametrize("layout", ["columns", "rows", "transposed", "steps"])
def test_tokens_in_a_view_of_a_larger_tensor(layout):
    from them_bones_b200.utils import decode as D
    model, b, p, n = _model(), 5, 7, 12
    prompts = torch.randint(1, 1000, (b, p), device="cuda")
    prompts[:, 0] = 0
    want = D.greedy_decode(model, prompts, n - p)
    big = torch.full({"columns": (b, n + 9), "rows": (2 * b, n), "transposed": (n, b), "steps": (b, 2 * n)}[layout], -7, dtype=torch.int64, device="cuda")
    view = {"columns": lambda: big[:, :n], "rows": lambda: big[::2], "transposed": lambda: big.T, "steps": lambda: big[:, ::2]}[layout]()
    view[:, :p] = prompts
    view[:, p:] = 0
    with torch.no_grad():
        dec = D.NativeDecoder(model, D.KVCache(model, b, n), prompts[:, 0], view, prompt_len=p)
        dec.run(n - 1)
    D.L_check()
    assert dec.fused == (layout in ("columns", "rows"))
    if dec.fused:
        assert torch.equal(view, want)             # the other route rounds elsewhere: equal tokens are not promised
    assert torch.equal(view[:, :p], prompts) and bool((view[:, p:] < 1024).all()) and int((big != -7).sum()) == int((view != -7).sum())


@pytest.mark.gpu
def test_token_rows_of_another_type_are_refused():
    from them_bones_b200.utils import decode as D
    model = _model()
    out = torch.zeros(3, 6, dtype=torch.int32, device="cuda")
    dec = D.NativeDecoder(model, D.KVCache(model, 3, 6), torch.zeros(3, dtype=torch.int64, device="cuda"), out)
    assert not dec.fused
    with pytest.raises((RuntimeError, IndexError)):
        dec.run(1)
