"""The Newton-Schulz iteration against 64 bits over tile remainders (one kernel, except for two matrices of 400 x 272: batched launches)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,r,c,steps", [(1, 16, 16, 5), (3, 144, 400, 5), (2, 400, 272, 3), (4, 400, 272, 4), (7, 64, 1024, 1), (4, 256, 256, 5), (6, 1280, 640, 2),
                                         (5, 384, 1280, 5), (40, 128, 128, 5)])
def test_matches_64_bits_and_repeats(n, r, c, steps):
    from them_bones_b200.ops import _lib as L
    from them_bones_b200.ops.muon_native import newton_schulz
    from them_bones_b200.ref.functional import POLAR_EXPRESS_COEFFS
    g = torch.Generator(device="cuda").manual_seed(n * r + c)
    x = torch.randn(n, r, c, generator=g, device="cuda")
    x = (x / x.norm(dim=(1, 2), keepdim=True)).bfloat16().contiguous()
    keep = x.clone()
    y = newton_schulz(x, steps)
    torch.cuda.synchronize()
    L.check_error_word()
    z = x.double()
    for a, b, k in POLAR_EXPRESS_COEFFS[:steps]:
        m = z.mT @ z if r > c else z @ z.mT
        p = b * m + k * (m @ m)
        z = a * z + (z @ p if r > c else p @ z)
    assert torch.equal(x, keep)
    # three bf16 roundings an iteration, amplified by its gain of up to 8 on small singular values
    assert float((y.double() - z).norm() / z.norm()) < 4e-2
    for _ in range(20):                        # the order of CTAs changes, the sums do not
        assert torch.equal(newton_schulz(x, steps), y)
