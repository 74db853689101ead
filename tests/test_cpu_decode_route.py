"""Which of its two kernels a decode step's layers and its head take: the one measured faster on both sides of each line."""
import pytest

from them_bones_b200.utils import decode as D


@pytest.mark.parametrize("width,batch,rows", [(128, 1, True), (128, 16, True), (256, 1, True), (256, 8, True), (384, 1, False), (384, 20, True), (512, 8, False),
                                              (640, 4, False), (768, 16, False), (896, 1, True), (896, 16, True), (1024, 1, True)])
def test_layers(width, batch, rows):
    assert D.use_rows(batch, width, width, 4 * width, 148) == rows


@pytest.mark.parametrize("k,n,batch,rows", [(1280, 65536, 16, False), (1280, 65536, 20, False), (1280, 65536, 28, False), (1280, 65536, 33, True), (1280, 65536, 64, True),
                                            (1024, 32768, 20, False), (1024, 32768, 36, True), (1536, 65536, 18, True), (1024, 131072, 28, True), (1024, 131072, 16, False),
                                            (256, 65536, 20, False), (256, 65536, 64, False), (256, 8192, 24, False), (256, 8192, 64, True)])
def test_head(k, n, batch, rows):
    assert D.head_on_rows(batch, n, k) == rows
