"""Native calls from a thread that has made no CUDA call yet, as autograd's device thread may be: the library finds its context."""
import os
import subprocess
import sys
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu


def _in_new_thread(f):
    box = []

    def body():
        try:
            box.append(f())
        except BaseException as e:  # noqa: BLE001
            box.append(e)
    t = threading.Thread(target=body)
    t.start()
    t.join()
    if isinstance(box[0], BaseException):
        raise box[0]
    return box[0]


@pytest.mark.parametrize("m,n,k,pair", [(40, 64, 128, False), (512, 512, 128, True)])
def test_first_call_of_a_thread(m, n, k, pair):
    from them_bones_b200.ops import _lib as L
    a, b = (torch.randn(r, k, device="cuda").bfloat16() for r in (m, n))
    d, ref = torch.empty(2, m, n, device="cuda", dtype=torch.bfloat16)
    L.gemm(a, b, ref, m=m, n=n, k=k, lda=k, ldb=k, ldd=n, pair=pair)
    torch.cuda.synchronize()
    _in_new_thread(lambda: L.gemm(a, b, d, m=m, n=n, k=k, lda=k, ldb=k, ldd=n, pair=pair))
    torch.cuda.synchronize()
    assert torch.equal(d, ref)


def test_backward_in_a_process_whose_first_backward_is_a_product():
    """In a process of its own: autograd's thread lives on, and an earlier test may have given it a context."""
    code = """
import torch
from them_bones_b200 import ops
x, w = torch.randn(40, 64, device="cuda").bfloat16().requires_grad_(), torch.randn(128, 64, device="cuda").bfloat16().requires_grad_()
y = ops.linear(x, w)
dy = torch.ones_like(y)
room = [torch.empty(1 << 16, device="cuda") for _ in range(40)]
del room
dx, dw = torch.autograd.grad(y, [x, w], dy)
assert float((dx.float() - dy.float() @ w.float()).norm() / dx.float().norm()) < 5e-3
assert float((dw.float() - dy.float().T @ x.float()).norm() / dw.float().norm()) < 5e-3
"""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", code], cwd=root, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
