"""fp32 convolutions as three TF32 products with A in tensor memory: all three passes against the oracle at the edges of
the tiles (channel boxes of 32, two filter taps to a tile, column tiles of 64 and 128, the filter's lo part ahead of
the kernel and inside it) and the fp32 epilogue's bias and activations beside the last column."""
import numpy as np
import pytest
import torch

import portdnn_b200 as pd
from conftest import rel_err
from gpu_util import TOL, assert_no_device_error, to_dev, to_host

pytestmark = pytest.mark.gpu

# n, h, w, c, k, window, stride
SHAPES = [
    (1, 5, 5, 4, 4, 3, 1),        # one partial tile of everything
    (2, 13, 11, 32, 36, 3, 1),    # one channel box of four; odd number of taps, two to a tile
    (2, 13, 11, 36, 100, 2, 1),   # the second box of a tap holds four channels
    (1, 17, 15, 64, 64, 3, 2),    # two full boxes to a tap, parity classes
    (1, 17, 15, 68, 132, 3, 1),   # one tap to a tile, a column tile of four columns
    (2, 40, 40, 64, 48, 1, 1),    # 2048 pixels and more, 64 columns backwards: the filter is split in the kernel
    (2, 40, 40, 68, 64, 1, 1),    # ... and 68: ahead of it
    (3, 56, 56, 128, 128, 3, 1),  # several tiles to a CTA
    (4, 16, 16, 3, 64, 3, 1),     # packed few-channel form, filter rows two to a tile
    # column tiles of 16 and 32: rings of seven stages
    (2, 20, 20, 128, 16, 3, 1),   # one tile of 36 steps
    (8, 64, 64, 96, 24, 3, 1),    # forward: two tiles to a CTA; filter gradient: 1024 steps
    (8, 64, 64, 24, 96, 3, 1),    # input gradient: two tiles to a CTA
    (3, 65, 63, 128, 32, 1, 1),
]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("activation", [pd.ACT_NONE, pd.ACT_RELU, pd.ACT_TANH, pd.ACT_RELU6])
def test_forward(orc, shape, activation):
    n, h, w, c, k, win, st = shape
    rng = np.random.default_rng(1)
    p, po = pd.conv_params(n, h, w, c, k, win, st), orc.conv_params(n, h, w, c, k, win, st)
    x = rng.uniform(-1, 1, n * h * w * c).astype(np.float32)
    wt = (rng.uniform(-1, 1, win * win * c * k) * 8 * np.sqrt(1.0 / (win * win * c))).astype(np.float32)
    b = rng.standard_normal(k).astype(np.float32)
    y = to_host(pd.conv2d(pd.FORWARD, to_dev(x, "f32"), to_dev(wt, "f32"), p, bias=to_dev(b, "f32"), activation=activation))
    assert_no_device_error()
    ref = orc.conv2d(orc.FORWARD, x, wt, po).reshape(-1, k) + b
    ref = {pd.ACT_NONE: ref, pd.ACT_RELU: np.maximum(ref, 0), pd.ACT_TANH: np.tanh(ref), pd.ACT_RELU6: np.clip(ref, 0, 6)}[activation]
    # (sums of up to 1152 products of order one, outputs clipped to order one: the bound of the unclipped sums, which are
    # about eight times larger, still holds where the largest output is one)
    assert rel_err(y, ref.ravel()) <= TOL["f32"]


@pytest.mark.parametrize("shape", SHAPES)
def test_backprops(orc, shape):
    n, h, w, c, k, win, st = shape
    rng = np.random.default_rng(2)
    p, po = pd.conv_params(n, h, w, c, k, win, st), orc.conv_params(n, h, w, c, k, win, st)
    x = rng.uniform(-1, 1, n * h * w * c).astype(np.float32)
    wt = (rng.uniform(-1, 1, win * win * c * k) * np.sqrt(1.0 / (win * win * c))).astype(np.float32)
    dy = rng.standard_normal(n * p.out_rows * p.out_cols * k).astype(np.float32)
    dw = to_host(pd.conv2d(pd.FILTER_BACKPROP, to_dev(x, "f32"), to_dev(dy, "f32"), p))
    assert rel_err(dw, orc.conv2d(orc.FILTER_BACKPROP, x, dy, po)) <= TOL["f32"]
    dx = to_host(pd.conv2d(pd.INPUT_BACKPROP, to_dev(dy, "f32"), to_dev(wt, "f32"), p))
    assert rel_err(dx, orc.conv2d(orc.INPUT_BACKPROP, dy, wt, po)) <= TOL["f32"]
    assert_no_device_error()


@pytest.mark.parametrize("shape", SHAPES)
def test_relu_gradient_in_the_epilogue(shape):
    """The masked input gradient is the unmasked one with zeros wherever the forward output is not positive."""
    n, h, w, c, k, win, st = shape
    rng = np.random.default_rng(5)
    p = pd.conv_params(n, h, w, c, k, win, st)
    fwd = to_dev(rng.standard_normal(n * h * w * c).astype(np.float32), "f32")
    wt = to_dev(rng.standard_normal(win * win * c * k).astype(np.float32), "f32")
    dy = to_dev(rng.standard_normal(n * p.out_rows * p.out_cols * k).astype(np.float32), "f32")
    plain = pd.conv2d(pd.INPUT_BACKPROP, dy, wt, p)
    masked = pd.conv2d(pd.INPUT_BACKPROP, dy, wt, p, relu_forward_output=fwd)
    assert_no_device_error()
    assert torch.equal(masked, torch.where(fwd > 0, plain, torch.zeros_like(plain)))
