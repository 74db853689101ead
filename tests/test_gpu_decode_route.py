"""Decode steps on both sides of the lines between the two projection kernels, against the PyTorch route."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("b,n_embd,vocab", [(1, 128, 1024), (16, 256, 1024), (3, 384, 1024), (9, 896, 1024), (20, 1024, 2048), (32, 1024, 131072), (33, 1024, 2048),
                                            (40, 256, 32768), (40, 256, 16384)])
def test_step(b, n_embd, vocab):
    from them_bones_b200.config import GPTConfig
    from them_bones_b200.models.gpt import GPT
    from them_bones_b200.utils import decode as D
    torch.manual_seed(b)
    steps = 6
    cfg = GPTConfig(sequence_len=256, vocab_size=vocab, n_layer=2, n_head=n_embd // 128, n_embd=n_embd, head_dim=128, doc_mask=True)
    with torch.device("cuda"):
        model = GPT(cfg)
    model.init_weights()
    for p in model.parameters():
        if p.dim() == 2:
            torch.nn.init.normal_(p, std=0.03)
    model.cast_compute(torch.bfloat16).eval()
    toks = torch.randint(1, 1000, (b, steps), device="cuda")
    toks[:, 0] = 0
    out = torch.cat([toks, torch.zeros(b, 1, dtype=torch.int64, device="cuda")], 1)
    with torch.no_grad():
        dec = D.NativeDecoder(model, D.KVCache(model, b, steps + 1), toks[:, 0], out, prompt_len=steps)
        dec.run(steps)
        ref = D._forward_cached(model, toks, D.KVCache(model, b, steps + 1))
    D.L_check()
    assert dec.fused and dec.rows == D.use_rows(b, n_embd, n_embd, 4 * n_embd, dec.sms)
    got = dec.last_logits.float()[:, :vocab]
    # bf16 activations through two layers, rounded at other places by the two routes
    assert float((got - ref).norm() / ref.norm()) < 3e-2
