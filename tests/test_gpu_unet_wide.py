"""Convolutions of images at least 128 pixels wide (a tile is part of one image row), with the tolerance of the other
forward convolution tests, 4e-3 (bf16 outputs); and the backward pass, whose weight gradients run on a stream forked
from the caller's, on other streams and under graph capture (FP32 sums in another order: 1e-5 of the gradient)."""
import pytest
import torch

from sarsolver_gb300.unet import UNet
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


@pytest.mark.parametrize("H,W", [(128, 128), (64, 256)])
def test_backward_on_streams_and_captured(H, W):
    net = UNet(base_channels=32, seed=7)
    g = torch.Generator(device="cuda")
    g.manual_seed(8)
    x, go = (torch.complex(torch.randn(1, H, W, device="cuda", generator=g), torch.randn(1, H, W, device="cuda", generator=g))
             for _ in range(2))

    def step():
        net.zero_grad()
        net.forward(x)
        net.backward(go)
        return net.grads()

    ref = step().clone()
    close = lambda t: float((t - ref).norm() / ref.norm()) < 1.0e-5
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        assert all(close(step()) for _ in range(3))
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = step()
    for _ in range(3):
        out.zero_()
        graph.replay()
        assert close(out)
    assert net.flags() == 0
