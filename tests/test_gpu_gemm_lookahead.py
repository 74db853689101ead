"""Single-CTA products on both sides of the contraction from which the issuing warp looks at the next stage ahead."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [96, 128, 160, 192, 224, 256])
@pytest.mark.parametrize("k", [8, 64, 72, 448, 1016, 1024, 1032, 1600])
def test_product(n, k):
    """Every tile width (and so ring depth), one tile a CTA and several, the last K block full and ragged."""
    from them_bones_b200.ops import _lib as L
    g = torch.Generator(device="cuda").manual_seed(n + k)
    for m in (40, 128 * 300):
        a, b = (torch.randn(r, k, generator=g, device="cuda").bfloat16() for r in (m, n))
        d = torch.full((m, n), float("nan"), device="cuda", dtype=torch.bfloat16)
        L.gemm(a, b, d, m=m, n=n, k=k, lda=k, ldb=k, ldd=n, pair=False, force_bn=n)
        want = a.float().double() @ b.double().T
        # fp32 sums rounded once: half a unit of 8 bits
        assert float((d.double() - want).norm() / want.norm()) < 2.5e-3
    L.check_error_word()
