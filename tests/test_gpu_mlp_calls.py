"""The bf16 MLP's native calls on an empty batch, and with each way of running a product."""
import os
import subprocess
import sys

import pytest
import torch

pytestmark = pytest.mark.gpu


def test_empty_batch():
    from them_bones_b200 import ops
    x = torch.empty(3, 0, 64, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    w1, w2 = (torch.randn(*s, device="cuda").bfloat16().requires_grad_() for s in ((128, 64), (64, 128)))
    y = ops.mlp(x, w1, w2, residual=torch.empty_like(x))
    gx, g1, g2 = torch.autograd.grad(y, [x, w1, w2], torch.empty_like(y))
    assert y.shape == x.shape and gx.shape == x.shape and torch.equal(g1, torch.zeros_like(w1)) and torch.equal(g2, torch.zeros_like(w2))


_CODE = """
import torch
from them_bones_b200 import ops
g = torch.Generator(device="cuda").manual_seed(1)
for m in (40, 700):
    x, w1, w2, r, dy = (torch.randn(*s, generator=g, device="cuda").bfloat16() for s in ((m, 256), (512, 256), (256, 512), (m, 256), (m, 256)))
    w1, w2 = w1 / 16, w2 / 24
    ins = [t.requires_grad_() for t in (x, w1, w2)]
    y = ops.mlp(x, w1, w2, residual=r)
    got = [y.detach()] + list(torch.autograd.grad(y, ins, dy))
    X, W1, W2, DY = (t.detach().double() for t in (x, w1, w2, dy))
    a = (X @ W1.T).clamp_min(0)
    dpre = (DY @ W2) * 2 * a
    want = [a.square() @ W2.T + r.double(), dpre @ W1, dpre.T @ X, DY.T @ a.square()]
    # h and dpre are rounded to bf16 between the products
    assert all(float((u.double() - v).norm() / v.norm()) < 8e-3 for u, v in zip(got, want))
torch.cuda.synchronize()
from them_bones_b200.ops import _lib
_lib.check_error_word()
"""


@pytest.mark.parametrize("mode", ["0", "1", "auto"])
def test_each_way_of_running_a_product(mode):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", _CODE], cwd=root, env={**os.environ, "BONES_GEMM_PAIR": mode}, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
