"""The single-CTA GEMM's tile widths and the choice between them, on shapes whose last tiles are ragged."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k,b_major,bn", [(1, 264, 72, 0, 96), (129, 1000, 264, 0, 96), (200, 488, 128, 0, 160), (127, 456, 1280, 0, 224), (300, 392, 200, 1, 192),
                                              (64, 200, 64, 1, 192), (255, 1280, 640, 1, 0), (300, 1288, 1288, 0, 0), (700, 3840, 256, 0, 0)])
@pytest.mark.parametrize("epi", [0, 1, 2])
def test_tile_widths(m, n, k, b_major, bn, epi):
    from them_bones_b200.ops import _lib as L
    g = torch.Generator(device="cuda").manual_seed(m + n)
    a = torch.randn(m, k, generator=g, device="cuda").bfloat16()
    b = (0.1 * torch.randn((k, n) if b_major else (n, k), generator=g, device="cuda")).bfloat16()
    r = torch.randn(m, n, generator=g, device="cuda").bfloat16()
    d = torch.full((m, n), float("nan"), device="cuda", dtype=torch.bfloat16)
    L.gemm(a, b, d, m=m, n=n, k=k, lda=k, ldb=b.stride(0), ldd=n, b_major=b_major, epi=epi, r=r if epi == 1 else None, ldr=n if epi == 1 else 0,
           force_bn=bn, pair=False if bn else None)
    torch.cuda.synchronize()
    L.check_error_word()
    want = a.double() @ (b.double() if b_major else b.double().T)
    want = want + r.double() if epi == 1 else want.clamp_min(0).square() if epi == 2 else want
    assert float((d.double() - want).norm() / want.norm()) < 4e-3          # one bf16 rounding is 2^-9
