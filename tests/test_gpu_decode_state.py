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


@pytest.mark.gpu
@pytest.mark.parametrize("b,window", [(64, 0), (7, 128)])
def test_documents_that_begin_at_many_steps(b, window):
    """Every step some sequences begin a document: their attention sees nothing before it, from that very step on."""
    from them_bones_b200.utils import decode as D
    model, steps = _model(n_layer=3, attn_window=window, attn_long=(2,)), 150
    toks = torch.randint(1, 1000, (b, steps), device="cuda")
    toks[torch.rand(b, steps, device="cuda") < 0.2] = 0
    toks[:, 0] = 0
    toks[: b // 2, steps - 1] = 0
    out = torch.cat([toks, torch.zeros(b, 1, dtype=torch.int64, device="cuda")], 1)
    with torch.no_grad():
        cache = D.KVCache(model, b, steps + 1)
        dec = D.NativeDecoder(model, cache, toks[:, 0], out, prompt_len=steps)
        assert dec.fused
        dec.run(steps)
        got = dec.last_logits.float()
        # a document that begins with the last token: the same logits as that token alone
        alone = D._forward_cached(model, toks[: b // 2, -1:], _at(D.KVCache(model, b // 2, steps + 1), steps - 1))
        ref = D._forward_cached(model, toks, D.KVCache(model, b, steps + 1))
    D.L_check()
    last = torch.where(toks == 0, torch.arange(steps, device="cuda"), 0).amax(1).int()
    assert torch.equal(cache.doc_start, last)
    rel = ((got - ref).norm(dim=1) / ref.norm(dim=1))
    assert float(rel.max()) < 6e-2, rel            # bf16 activations of three layers, row by row
    rel = ((got[: b // 2] - alone).norm(dim=1) / alone.norm(dim=1))
    assert float(rel.max()) < 6e-2, rel


def _at(cache, pos):
    cache.len = pos
    return cache


@pytest.mark.gpu
def test_unknown_token_ids_have_zero_rows():
    """An id outside the embedding gives that sequence a zero row at that step, as in the embedding gather, not what an earlier
    step or another sequence left."""
    from them_bones_b200.utils import decode as D
    model, b, p = _model(), 6, 5
    for blk in model.transformer.h:
        blk.resid_lambda.data.fill_(0.9)
        blk.x0_lambda.data.fill_(0.3)
    toks = torch.randint(1, 1000, (b, p), device="cuda")
    toks[:, 0] = 0
    rows = model.transformer.wte.weight.shape[0]
    model.transformer.wte.weight.data[777] = 0
    toks[toks == 777] = 5

    def logits(ids):
        out = torch.cat([ids, torch.zeros(b, 1, dtype=torch.int64, device="cuda")], 1)
        with torch.no_grad():
            dec = D.NativeDecoder(model, D.KVCache(model, b, p + 1), ids[:, 0], out, prompt_len=p)
            assert dec.fused
            dec.run(p)
        return dec.last_logits.clone()

    zero, unknown = toks.clone(), toks.clone()
    zero[1, 2] = zero[4, p - 1] = zero[3, 1] = 777
    unknown[1, 2], unknown[4, p - 1], unknown[3, 1] = rows, -1, rows + 12345
    got, want = logits(unknown), logits(zero)
    D.L_check()
    assert torch.equal(got, want)


@pytest.mark.parametrize("sms", [64, 132, 148, 160])
@pytest.mark.parametrize("width", [128, 256, 512, 1024, 1280, 1408, 1536, 1664, 2048, 4096])
def test_projection_splits_follow_the_device(width, sms):
    """Powers of two that leave every CTA a K block and fit the device; a projection with few tiles is shared until the CTAs cover
    a good part of it, at any width."""
    from them_bones_b200.utils.decode import projection_splits
    for b in (1, 16, 17, 32, 33, 64, 65, 128):
        for n, k, res in ((3 * width, width, False), (width, width, True), (4 * width, width, False), (width, 4 * width, True), (65536, width, False)):
            s = projection_splits(b, n, k, res, sms)
            tiles, most = n // 128, 4 if b <= 16 else 8 if b <= 32 or b > 64 else 16
            assert s in (1, 2, 4, 8, 16) and s <= most and s <= k // 64
            assert s == 1 or tiles * s <= 1.6 * sms and (b <= 64 or tiles * s <= sms)
            if res and s < most and 2 * s <= k // 64:
                assert tiles * s > 0.4 * sms, (b, n, k, s)


@pytest.mark.gpu
@pytest.mark.parametrize("width,b", [(384, 40), (1408, 64), (1408, 100), (1536, 24), (2048, 8), (2048, 70)])
def test_step_at_other_widths(width, b):
    from them_bones_b200.utils import decode as D
    model, steps = _model(n_embd=width), 6
    toks = torch.randint(1, 1000, (b, steps), device="cuda")
    toks[:, 0] = 0
    out = torch.cat([toks, torch.zeros(b, 1, dtype=torch.int64, device="cuda")], 1)
    with torch.no_grad():
        dec = D.NativeDecoder(model, D.KVCache(model, b, steps + 1), toks[:, 0], out, prompt_len=steps)
        assert dec.fused
        dec.run(steps)
        ref = D._forward_cached(model, toks, D.KVCache(model, b, steps + 1))
    D.L_check()
    got = dec.last_logits.float()
    assert float((got - ref).norm() / ref.norm()) < 3e-2          # bf16 activations of two layers
