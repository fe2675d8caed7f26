"""The depthwise 3x3 kernels on TMA tiles against the oracle: sizes around their tiles of 14 or 8 (stride 1) or 4
(stride 2) columns and two rows to a strip, one and several chunks of channels, and values at the image's edges
that belong to no product.  Which kernel ran is read from a trace."""
import numpy as np
import pytest
import torch

import portdnn_b200 as pd
from gpu_util import assert_no_device_error, rounded, to_dev, to_host

pytestmark = pytest.mark.gpu

# n, h, w, c, stride, same
SHAPES = [
    (1, 3, 3, 8, 1, False),      # one output: too few tiles for the filter gradient
    (9, 7, 7, 24, 1, True),      # odd rows: the last strip has one
    (8, 8, 8, 40, 1, True),
    (4, 9, 17, 144, 1, True),    # one column beyond two tiles
    (5, 33, 16, 72, 1, False),
    (8, 6, 7, 960, 1, True),     # several chunks
    (8, 5, 5, 520, 2, True),     # the last chunk partly beyond the channels
    (9, 5, 5, 520, 1, True),
    (2, 9, 28, 40, 1, True),     # two whole tiles of 14 columns
    (2, 9, 27, 40, 1, True),     # ... the second one short of a column
    (1, 30, 40, 24, 1, True),    # three, the last of 12 columns
    (3, 15, 18, 32, 2, True),
    (2, 64, 9, 16, 2, False),
    (40, 14, 14, 64, 1, True),   # several tiles to a block
]
# Products of 16-bit values are exact in fp32; a sum of m terms in any order is off by at most m * 2^-24 of the sum of
# magnitudes, the rounding of the result by 2^-11 or 2^-8 of its value.
ULP = {"f16": 2.0 ** -11, "bf16": 2.0 ** -8, "f32": 2.0 ** -24}


def traced(call, kernel, ran=True):
    """What the call returns; kernel was launched by it, or was not.  (Without a tracer nothing is known of it.)"""
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA], acc_events=True) as trace:
        out = call()
        torch.cuda.synchronize()
    names = [e.key for e in trace.key_averages() if "kernel<" in e.key]
    assert not names or any(kernel in n for n in names) == ran, names
    return out


@pytest.mark.parametrize("dtype", ["f16", "bf16", "f32"])
@pytest.mark.parametrize("shape", SHAPES)
def test_filter_gradient(orc, dtype, shape):
    n, h, w, c, st, same = shape
    rng = np.random.default_rng(3)
    p, po = pd.depthwise_params(n, h, w, c, 1, 3, st, same), orc.depthwise_params(n, h, w, c, 1, 3, st, same)
    x = rounded(rng.standard_normal(n * h * w * c).astype(np.float32), dtype)
    dy = rounded(rng.standard_normal(n * p.out_rows * p.out_cols * c).astype(np.float32), dtype)
    xd, dyd = to_dev(x, dtype), to_dev(dy, dtype)
    got = to_host(traced(lambda: pd.depthwise_conv2d(pd.FILTER_BACKPROP, xd, dyd, p), "depthwise_filter_tile_kernel", shape != SHAPES[0]))
    assert_no_device_error()
    ref = orc.depthwise_conv2d(orc.FILTER_BACKPROP, x, dy, po)
    size = orc.depthwise_conv2d(orc.FILTER_BACKPROP, np.abs(x), np.abs(dy), po)
    terms = n * p.out_rows * p.out_cols
    # (the oracle's own fp32 sums are off by as much again)
    assert np.all(np.abs(got - ref) <= 2 * (terms + 1) * 2.0 ** -24 * size + ULP[dtype] * np.abs(ref) + 2.0 ** -24)


@pytest.mark.parametrize("size,c", [(56, 144), (112, 32)])
def test_error_of_long_fp32_sums(size, c):
    """128 images, products of random sign, against float64.  A chain of L additions of products of variance one leaves an
    error of 0.45 * 2^-24 * sqrt(L / 2) of the root of the number of terms: 2e-7 for sums of up to 28 products that are
    then added up over the 64 tiles of a thread, 3e-7 for chains of 500, 8e-7 for one of 1800."""
    n = 128
    p = pd.depthwise_params(n, size, size, c, 1, 3, 1, True)
    g = torch.Generator(device="cuda").manual_seed(1)
    x, dy = (torch.randn(n, size, size, c, device="cuda", generator=g) for _ in range(2))
    dw = pd.depthwise_conv2d(pd.FILTER_BACKPROP, x.view(-1), dy.view(-1), p).view(3, 3, c)
    assert_no_device_error()
    xp = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1))
    ref = torch.stack([torch.stack([(xp[:, r:r + size, s:s + size].double() * dy).sum((0, 1, 2)) for s in range(3)]) for r in range(3)])
    assert (dw - ref).square().mean().sqrt() <= 3.2e-7 * (n * size * size) ** 0.5


@pytest.mark.parametrize("dtype", ["f16", "f32"])
def test_edge_values_stay_out_of_other_taps(dtype):
    """VALID windows on 10 x 11 pixels: the last row and column are read by the last tap of each direction only."""
    n, h, w, c = 16, 10, 11, 16
    p = pd.depthwise_params(n, h, w, c, 1, 3, 1, False)
    x = torch.zeros(n, h, w, c)
    x[:, -1] = float("inf")
    x[:, :, -1] = float("inf")
    dy = torch.ones(n, p.out_rows, p.out_cols, c)
    dw = pd.depthwise_conv2d(pd.FILTER_BACKPROP, to_dev(x.numpy().ravel(), dtype), to_dev(dy.numpy().ravel(), dtype), p)
    dw = dw.float().cpu().view(3, 3, c)
    assert_no_device_error()
    assert torch.equal(dw[:2, :2], torch.zeros(2, 2, c))
    assert torch.isinf(dw[2]).all() and torch.isinf(dw[:, 2]).all()


@pytest.mark.parametrize("dtype", ["f16", "bf16", "f32"])
@pytest.mark.parametrize("shape,kernel", [
    ((16, 10, 11, 16, 1), "depthwise_filter_tile_kernel"),
    ((9, 9, 15, 24, 2), "depthwise_filter_tile_kernel"),
    ((1, 5, 6, 16, 1), "depthwise_filter_backprop_rows_kernel"),  # few tiles
    ((2, 7, 9, 10, 2), "depthwise_filter_backprop_rows_kernel"),  # no whole packets
    ((3, 11, 10, 16, 3), "depthwise_filter_backprop_partial9_kernel")])
def test_infinities_meet_their_own_products_only(dtype, shape, kernel):
    """SAME windows: what stands outside the image, and for outputs that do not exist, is no term of a sum."""
    n, h, w, c, st = shape
    p = pd.depthwise_params(n, h, w, c, 1, 3, st, True)
    rng = np.random.default_rng(6)
    x = rounded(rng.standard_normal(n * h * w * c).astype(np.float32), dtype).reshape(n, h, w, c)
    dy = rounded(rng.standard_normal(n * p.out_rows * p.out_cols * c).astype(np.float32), dtype).reshape(n, p.out_rows, p.out_cols, c)
    dy[0, 0, 0, 0] = dy[-1, 0, -1, 2] = dy[0, -1, 0, 4] = dy[-1, -1, -1, 6] = np.inf
    x[0, 0, 0, 1] = x[-1, 0, -1, 3] = x[0, -1, 0, 5] = x[-1, -1, -1, 7] = -np.inf
    xd, dyd = to_dev(x.ravel(), dtype), to_dev(dy.ravel(), dtype)
    dw = to_host(traced(lambda: pd.depthwise_conv2d(pd.FILTER_BACKPROP, xd, dyd, p), kernel)).reshape(3, 3, c)
    assert_no_device_error()
    ref, size = np.zeros((3, 3, c)), np.zeros((3, 3, c))
    for r in range(3):
        for s in range(3):
            oh = [o for o in range(p.out_rows) if 0 <= o * st - p.pad_rows + r < h]
            ow = [o for o in range(p.out_cols) if 0 <= o * st - p.pad_cols + s < w]
            a = x[:, [o * st - p.pad_rows + r for o in oh]][:, :, [o * st - p.pad_cols + s for o in ow]].astype(np.float64)
            b = dy[:, oh][:, :, ow].astype(np.float64)
            ref[r, s], size[r, s] = (a * b).sum((0, 1, 2)), np.abs(a * b).sum((0, 1, 2))
    finite = np.isfinite(ref)
    assert finite.sum() >= 9 * (c - 8) and not finite.all()
    assert np.array_equal(dw[~finite], ref[~finite], equal_nan=True)
    terms = n * p.out_rows * p.out_cols
    dw, ref, size = dw[finite], ref[finite], size[finite]
    assert np.all(np.abs(dw - ref) <= (terms + 1) * 2.0 ** -24 * size + ULP[dtype] * np.abs(ref) + 2.0 ** -24)


@pytest.mark.parametrize("dtype", ["f16", "bf16", "f32"])
@pytest.mark.parametrize("shape", SHAPES)
def test_forward_and_input_gradient(orc, dtype, shape):
    n, h, w, c, st, same = shape
    rng = np.random.default_rng(4)
    p, po = pd.depthwise_params(n, h, w, c, 1, 3, st, same), orc.depthwise_params(n, h, w, c, 1, 3, st, same)
    x = rounded(rng.standard_normal(n * h * w * c).astype(np.float32), dtype)
    f = rounded(rng.standard_normal(9 * c).astype(np.float32), dtype)
    dy = rounded(rng.standard_normal(n * p.out_rows * p.out_cols * c).astype(np.float32), dtype)
    xd, fd, dyd = to_dev(x, dtype), to_dev(f, dtype), to_dev(dy, dtype)
    tiles = "depthwise_forward_tile_kernel"
    y = to_host(traced(lambda: pd.depthwise_conv2d(pd.FORWARD, xd, fd, p), tiles, dtype == "bf16"))
    dx = to_host(traced(lambda: pd.depthwise_conv2d(pd.INPUT_BACKPROP, dyd, fd, p), tiles, dtype == "bf16" and st == 1))
    assert_no_device_error()
    # nine products: at most nine roundings of partial sums (fp16 kernels may hold them in fp16) and one of the result
    for got, ref, size in ((y, orc.depthwise_conv2d(orc.FORWARD, x, f, po), orc.depthwise_conv2d(orc.FORWARD, np.abs(x), np.abs(f), po)),
                           (dx, orc.depthwise_conv2d(orc.INPUT_BACKPROP, dy, f, po),
                            orc.depthwise_conv2d(orc.INPUT_BACKPROP, np.abs(dy), np.abs(f), po))):
        assert np.all(np.abs(got - ref) <= 10 * (2.0 ** -24 if dtype == "bf16" else ULP[dtype]) * size + ULP[dtype] * np.abs(ref) + 2.0 ** -24)


def test_infinite_weight_meets_the_image_only():
    """bf16: a tap outside the image is no term of the sum, whatever its weight."""
    n, h, w, c = 1, 9, 10, 16
    p = pd.depthwise_params(n, h, w, c, 1, 3, 1, True)
    f = torch.zeros(3, 3, c)
    f[0, 0] = float("inf")
    y = pd.depthwise_conv2d(pd.FORWARD, to_dev(np.ones(n * h * w * c), "bf16"), to_dev(f.numpy().ravel(), "bf16"), p)
    y = y.float().cpu().view(h, w, c)
    assert torch.equal(y[0], torch.zeros(w, c)) and torch.equal(y[:, 0], torch.zeros(h, c))
    assert torch.isinf(y[1:, 1:]).all()


def test_rows_of_more_than_four_billion_elements():
    """bf16: the second of two rows starts more than 2^31 words into the output."""
    w, c = 2 ** 22 + 5, 1024
    if torch.cuda.get_device_properties(0).total_memory < 50e9:
        pytest.skip("needs two tensors of 17 GB")
    p = pd.depthwise_params(1, 2, w, c, 1, 3, 1, True)
    g = torch.Generator(device="cuda").manual_seed(2)
    x = torch.empty(2, w, c, device="cuda", dtype=torch.bfloat16).normal_(generator=g)
    f = torch.randn(3, 3, c, device="cuda", generator=g).bfloat16()
    y = pd.depthwise_conv2d(pd.FORWARD, x.view(-1), f.view(-1), p).view(2, w, c)
    assert_no_device_error()
    for at in (0, w // 2, w - 40):
        part = torch.nn.functional.pad(x[:, max(at - 1, 0):at + 41].double(), (0, 0, at == 0, at + 40 == w, 1, 1))
        terms = torch.stack([part[r:r + 2, s:s + 40] * f[r, s].double() for r in range(3) for s in range(3)])
        ref, size = terms.sum(0), terms.abs().sum(0)
        assert ((y[:, at:at + 40].double() - ref).abs() <= 10 * 2.0 ** -24 * size + 2.0 ** -8 * ref.abs() + 2.0 ** -24).all()
