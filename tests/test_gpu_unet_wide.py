"""Convolutions of images at least 128 pixels wide (a tile is part of one image row), with the tolerance of the other
forward convolution tests, 4e-3 (bf16 outputs)."""
import pytest
import torch

from test_gpu_unet import test_conv_forward as conv_forward

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def cuda_required():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


ROW_CASES = [
    # (B, H, W, c0, c1, cout, taps)
    (1, 3, 128, 32, 0, 32, 9),         # few tiles: the general kernel
    (1, 1300, 128, 32, 0, 32, 9),      # resident filter, two rows an item, a partial round of items
    (3, 417, 128, 32, 0, 32, 9),       # odd heights: the last item has one row
    (1, 650, 256, 32, 0, 64, 9),
    (2, 160, 512, 64, 32, 32, 9),      # two sources, a ring of filter blocks
    (1, 640, 256, 64, 0, 64, 9),
    (1, 620, 256, 32, 0, 96, 9),       # one row an item
    (1, 320, 512, 128, 64, 64, 9),
    (1, 1240, 128, 64, 0, 384, 9),     # output channels in two tiles
    (1, 610, 256, 128, 0, 256, 9),
]


@pytest.mark.parametrize("case", ROW_CASES)
def test_wide_conv_forward(case):
    conv_forward(case)
