"""The depthwise-conv + SwiGLU kernel where a stage takes several images: small grids, batches that are no multiple of what fits, borders
between images, against PyTorch in fp32."""
import pytest
import torch

from test_swiglu_tiles_gpu import test_tiles as check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,hg,wg,C,with_bias", [(300, 1, 1, 64, True), (257, 2, 2, 128, True), (200, 3, 5, 72, False), (161, 4, 4, 64, True),
                                                 (152, 7, 7, 128, True), (299, 8, 8, 64, False), (298, 1, 20, 64, True), (150, 8, 12, 136, True)])
def test_images(B, hg, wg, C, with_bias):
    check(B, hg, wg, C, with_bias)
