"""Counts off a multiple of 8, padded to whole lines of 64 or whole sectors of 16: both rules on either side of their line, for
channels and features, alone and together, in all three passes against float64."""
import pytest
import torch

import portdnn_b200 as pd
from gpu_util import TORCH_DTYPES
from test_gpu_cluster_gemm import _check, _rand

pytestmark = pytest.mark.gpu

# channels, features: 41, 130 -> sectors (48, 144); 50, 100, 150, 250 -> lines (64, 128, 192, 256); 40, 136 stay as they are
COUNTS = [(41, 130), (50, 100), (100, 150), (49, 50), (130, 41), (250, 148), (40, 150), (100, 136), (147, 149)]


@pytest.mark.parametrize("dtype", ["f16", "bf16"])
@pytest.mark.parametrize("win", [1, 3])
@pytest.mark.parametrize("c,k", COUNTS)
def test_passes(c, k, win, dtype):
    n, h, w = 3, 13, 18
    dt, g, lo = TORCH_DTYPES[dtype], torch.Generator(device="cuda").manual_seed(c * 7 + k), win // 2
    p = pd.conv_params(n, h, w, c, k, win, 1)
    x, dy, b = _rand(g, n, h, w, c).to(dt), _rand(g, n, h, w, k).to(dt), _rand(g, k).to(dt)
    wt = (_rand(g, win, win, c, k) / (win * win * c) ** 0.5).to(dt)
    w64, x64, dy64 = wt.double().permute(3, 2, 0, 1), x.double().permute(0, 3, 1, 2), dy.double().permute(0, 3, 1, 2)
    nhwc, conv, back = lambda t: t.permute(0, 2, 3, 1), torch.nn.functional.conv2d, torch.nn.functional.conv_transpose2d
    ref, mag = nhwc(conv(x64, w64, padding=lo)), nhwc(conv(x64.abs(), w64.abs(), padding=lo))
    y = pd.conv2d(pd.FORWARD, x.reshape(-1), wt.reshape(-1), p, bias=b, activation=pd.ACT_RELU).view(ref.shape)
    _check(y, (ref + b.double()).relu(), mag + b.double().abs(), dtype, before_bias=ref)
    ref, mag = nhwc(back(dy64, w64, padding=lo)), nhwc(back(dy64.abs(), w64.abs(), padding=lo))
    dx = pd.conv2d(pd.INPUT_BACKPROP, dy.reshape(-1), wt.reshape(-1), p).view(ref.shape)
    _check(dx, ref, mag, dtype)
    grad = lambda a, d: torch.nn.grad.conv2d_weight(a, w64.shape, d, padding=lo).permute(2, 3, 1, 0)
    ref, mag = grad(x64, dy64), grad(x64.abs(), dy64.abs())
    dw = pd.conv2d(pd.FILTER_BACKPROP, x.reshape(-1), dy.reshape(-1), p, output_f32=True).view(ref.shape)
    assert ((dw.double() - ref).abs() - 2.0 ** -20 * mag).max() <= 0
