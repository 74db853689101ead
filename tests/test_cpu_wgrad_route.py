"""Which way a weight gradient that autograd gets back is computed: written by the GEMM, or its contraction shared out."""
import pytest

from them_bones_b200.ops.cuda import _wgrad_direct

# n, k, rows, us written directly, us with the contraction shared out (148 SMs)
MEASURED = [(128, 128, 1000, 9.3, 16.5), (256, 128, 2048, 13.3, 11.4), (128, 128, 4096, 21.4, 12.6), (256, 256, 1000, 9.4, 23.0), (256, 256, 3072, 17.5, 15.1),
            (1024, 256, 1000, 9.4, 23.4), (1024, 256, 4096, 22.3, 16.0), (768, 768, 4096, 23.0, 17.6), (1024, 1024, 4096, 24.8, 20.3), (1280, 1280, 2048, 14.7, 19.9),
            (1280, 1280, 6144, 33.5, 30.1), (2560, 1280, 4096, 25.4, 40.0), (2560, 1280, 8192, 45.0, 50.5), (3840, 1280, 2048, 26.8, 39.7), (3840, 1280, 4096, 45.8, 51.6),
            (3840, 1280, 8192, 83.8, 74.1), (3840, 1280, 12288, 121.8, 100.1), (5120, 1280, 4096, 45.7, 55.3), (5120, 1280, 8192, 84.4, 92.8),
            (5120, 1280, 16384, 178.5, 164.6), (1280, 5120, 16384, 175.7, 165.8), (4096, 1024, 8192, 55.2, 61.2), (5120, 1280, 24576, 307.9, 243.2)]


@pytest.mark.parametrize("n,k,rows,direct,shared", MEASURED)
def test_the_faster_route_is_taken_where_they_are_apart(n, k, rows, direct, shared):
    assert abs(direct - shared) > 0.05 * min(direct, shared)
    assert _wgrad_direct(n, k, rows, 148) == (direct < shared)


def test_edges():
    assert not _wgrad_direct(1280, 1280, 0, 148) and _wgrad_direct(8, 8, 1, 148) and _wgrad_direct(8, 8, 1984, 148)
    # one wave of tiles more or less: what counts is the device's SMs
    assert not _wgrad_direct(3840, 1280, 8192, 148) and _wgrad_direct(3840, 1280, 8192, 150)
