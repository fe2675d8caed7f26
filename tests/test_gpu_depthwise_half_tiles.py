"""fp16 depthwise 3x3 layers of more than 4 MB run on TMA tiles, smaller ones on strips, with the same sums in the same order: a
batch equals its images, bit for bit."""
import pytest
import torch

import portdnn_b200 as pd
from gpu_util import assert_no_device_error

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h,w,c,st", [(57, 61, 24, 1), (29, 15, 136, 1), (14, 14, 576, 1), (7, 9, 960, 1), (13, 8, 264, 1), (15, 120, 40, 1),
                                      (56, 57, 144, 2), (30, 31, 88, 2), (9, 14, 520, 2), (7, 7, 8, 2)])
def test_a_batch_is_its_images(h, w, c, st):
    g = torch.Generator(device="cuda").manual_seed(h * c)
    n = (5 << 20) // (2 * h * w * c) + 2
    p, one = pd.depthwise_params(n, h, w, c, 1, 3, st), pd.depthwise_params(1, h, w, c, 1, 3, st)
    x = torch.randn(n, h * w * c, device="cuda", generator=g).half()
    dy = torch.randn(n, p.out_rows * p.out_cols * c, device="cuda", generator=g).half()
    wt = torch.randn(9 * c, device="cuda", generator=g).half()
    some = [0, 1, n // 2, n - 2, n - 1]
    y = pd.depthwise_conv2d(pd.FORWARD, x.reshape(-1), wt, p).view(n, -1)
    assert all(torch.equal(y[i], pd.depthwise_conv2d(pd.FORWARD, x[i], wt, one)) for i in some)
    dx = pd.depthwise_conv2d(pd.INPUT_BACKPROP, dy.reshape(-1), wt, p).view(n, -1)
    assert all(torch.equal(dx[i], pd.depthwise_conv2d(pd.INPUT_BACKPROP, dy[i], wt, one)) for i in some)
    assert_no_device_error()


def test_infinite_weights_meet_pixels_only():
    n, h, w, c = 24, 33, 35, 96
    p = pd.depthwise_params(n, h, w, c, 1, 3, 1)
    wt = torch.full((9, c), 0.5, device="cuda", dtype=torch.half)
    wt[0] = float("inf")  # the tap above and to the left
    y = pd.depthwise_conv2d(pd.FORWARD, torch.ones(n * h * w * c, device="cuda", dtype=torch.half), wt.reshape(-1), p).view(n, h, w, c)
    assert torch.isinf(y[:, 1:, 1:]).all()
    assert torch.isfinite(y[:, 0]).all() and torch.isfinite(y[:, :, 0]).all()
    assert (y[:, 0, 1:-1] == 3.0).all() and (y[:, 1:-1, 0] == 3.0).all()
