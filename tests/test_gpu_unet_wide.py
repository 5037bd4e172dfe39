"""Convolutions of images at least 128 pixels wide (a tile is part of one image row), with the tolerance of the other
forward convolution tests, 4e-3 (bf16 outputs); and the backward pass, whose weight gradients run on a stream forked
from the caller's, on other streams and under graph capture (FP32 sums in another order: 1e-5 of the gradient)."""
import ctypes

import pytest
import torch
import torch.nn.functional as F

from sarsolver_gb300 import _lib
from sarsolver_gb300.unet import UNet
from test_gpu_unet import ptr, test_conv_forward as conv_forward

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


WGRAD_CASES = [
    # (B, H, W, c0, c1, cout): blocks of 32 and 64 input and output channels in all combinations, one source and two, rows
    # of one tile and of several, odd heights, more K blocks than CTAs
    (1, 3, 128, 32, 0, 32), (2, 37, 256, 32, 0, 32), (1, 130, 512, 32, 0, 32), (1, 5, 128, 32, 0, 64), (1, 33, 256, 96, 0, 64),
    (1, 9, 128, 64, 0, 32), (3, 21, 256, 64, 32, 32), (1, 64, 512, 64, 32, 32), (1, 7, 128, 64, 0, 64), (2, 40, 256, 128, 64, 64),
    (1, 16, 256, 32, 32, 96), (1, 24, 128, 256, 128, 128), (1, 12, 384, 32, 0, 32),
]


@pytest.mark.parametrize("case", WGRAD_CASES)
def test_wide_weight_gradient(case):
    """Weight gradients of images at least 128 wide against FP64: exact products of bf16 values, truncated FP32 sums over some
    twenty blocks of 128 pixels (2e-6) and FP32 additions of the splits; 1e-5."""
    B, H, W, c0, c1, cout = case
    g = torch.Generator(device="cuda")
    g.manual_seed(9)
    rand = lambda c: torch.randn(B, H, W, c, device="cuda", generator=g).bfloat16()
    x0, x1, dz = rand(c0), rand(c1) if c1 else None, rand(cout)
    dw = torch.zeros(cout, 9, c0 + c1, device="cuda")
    flags = torch.zeros(4, dtype=torch.int32, device="cuda")
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    _lib.check(_lib.load().sar_conv2d_wgrad_bf16(ptr(x0), c0, ptr(x1), c1, ptr(dz), cout, B, H, W, 9, ptr(dw), ptr(flags), stream),
               "conv wgrad")
    torch.cuda.synchronize()
    assert int(flags[0]) == 0
    x = F.pad((x0 if x1 is None else torch.cat([x0, x1], -1)).double(), (0, 0, 1, 1, 1, 1))
    z = dz.double().reshape(-1, cout)
    for tap in range(9):
        want = z.T @ x[:, tap // 3:tap // 3 + H, tap % 3:tap % 3 + W].reshape(-1, c0 + c1)
        assert float((dw[:, tap].double() - want).norm() / want.norm()) < 1.0e-5


@pytest.mark.parametrize("B,H,W", [(1, 64, 128), (2, 96, 256), (1, 272, 512)])
def test_bias_gradient_beside_the_weights(B, H, W):
    """The sums of dZ that the weight gradient's CTAs form: the last 3x3 layer's bias, with every ReLU mask open (a bias of
    100) and gradients of one sign, so that dZ = W^T g in bf16; FP32 sums against FP64, 1e-5 (2e-3 a rounding of dZ that
    differs, of which there are few)."""
    net = UNet(base_channels=32, seed=11)
    l, top = net.layers[13], net.layers[14]
    p = net.params().clone()
    p[l["bias_offset"]:l["bias_offset"] + l["cout"]] = 100.0
    net.set_params(p)
    g = torch.Generator(device="cuda")
    g.manual_seed(12)
    x = torch.complex(torch.randn(B, H, W, device="cuda", generator=g), torch.randn(B, H, W, device="cuda", generator=g))
    go = torch.complex(torch.rand(B, H, W, device="cuda", generator=g), torch.zeros(B, H, W, device="cuda"))
    net.zero_grad()
    net.forward(x)
    net.backward(go)
    w = p[top["weight_offset"]:top["weight_offset"] + l["cout"]].bfloat16().double()   # the real output's row
    dz = (go.real.bfloat16().double()[..., None] * w).float().bfloat16().double()
    want = dz.sum(dim=(0, 1, 2))
    got = net.grads()[l["bias_offset"]:l["bias_offset"] + l["cout"]].double()
    assert float((got - want).norm() / want.norm()) < 1.0e-5 and net.flags() == 0
