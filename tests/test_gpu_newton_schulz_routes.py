"""The one-kernel Newton-Schulz iteration against the batched launches it stands in for, and which stacks go where."""
import pytest
import torch


@pytest.mark.parametrize("k,r,c,steps,aligned,one", [(5, 5120, 1280, 5, True, True), (4, 400, 272, 4, True, True), (3, 1280, 1280, 5, True, False),
                                                     (2, 400, 272, 3, True, False), (1, 16, 16, 5, True, True), (3, 144, 400, 5, True, True), (1, 256, 4096, 8, True, True),
                                                     (4, 1280, 1280, 9, True, False), (4, 1280, 1280, 0, True, False), (4, 1280, 1288, 5, True, False),
                                                     (0, 128, 128, 5, True, False), (6, 1280, 640, 2, False, False)])
def test_which_stacks_run_in_one_kernel(k, r, c, steps, aligned, one):
    from them_bones_b200.ops.muon_native import in_one_kernel
    assert in_one_kernel(k, r, c, steps, aligned) == one


# also one to three matrices of several tiles, which the dispatch leaves to the launches: the shortest distances in the list
@pytest.mark.gpu
@pytest.mark.parametrize("n,r,c,steps", [(1, 640, 512, 5), (2, 400, 272, 3), (2, 512, 1024, 5), (3, 400, 1024, 4), (3, 1280, 640, 5), (4, 400, 272, 4), (1, 16, 16, 5),
                                         (3, 144, 400, 5), (7, 64, 1024, 1), (6, 1280, 640, 2), (5, 384, 1280, 5), (40, 128, 128, 5), (5, 1280, 1280, 5)])
def test_one_kernel_against_the_launches(n, r, c, steps):
    from them_bones_b200 import ops
    from them_bones_b200.ops import _lib as L
    from them_bones_b200.ops import muon_native as M
    g = torch.Generator(device="cuda").manual_seed(n * r + c)
    x = torch.randn(n, r, c, generator=g, device="cuda")
    x = (x / x.norm(dim=(1, 2), keepdim=True)).bfloat16().contiguous()
    before = ops.COUNTS["ns_kernel"]
    want, one = M._launches(x, steps), M._one_kernel(x, steps)
    got = M.newton_schulz(x, steps)
    torch.cuda.synchronize()
    L.check_error_word()
    assert ops.COUNTS["ns_kernel"] == before + 1 + M.in_one_kernel(n, r, c, steps)
    # the same products, summed in the same order and rounded to bf16 at the same three places of an iteration
    assert torch.equal(one, want) and torch.equal(got, want)
