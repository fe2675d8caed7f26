"""Operators on tensors of more than half of the L2 cache begin with the last image; the result of a batch is that of its
images one by one, bit for bit.  The splits of a filter gradient go through such a batch side by side."""
import pytest
import torch

import portdnn_b200 as pd
from gpu_util import TORCH_DTYPES, assert_no_device_error

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["f16", "f32"])
@pytest.mark.parametrize("case", ["pool3_s1", "pool3_s2", "pool2", "depthwise_s1", "depthwise_s2", "conv1x1", "conv1x1_pair"])
def test_a_batch_is_its_images(case, dtype):
    dt, g = TORCH_DTYPES[dtype], torch.Generator(device="cuda").manual_seed(3)
    conv = case.startswith("conv")
    h, w, c, k = (31, 45, 512, 128) if case == "conv1x1_pair" else (61, 45, 136, 72) if conv else (61, 45, 136, 136)
    n = (80 << 20) // (h * w * c * dt.itemsize) + 1
    x = torch.randn(n, h, w, c, device="cuda", generator=g).to(dt)
    stride = 2 if case.endswith("s2") or case == "pool2" else 1
    wt = (torch.randn(9 * c * (k if conv else 1), device="cuda", generator=g) * 0.1).to(dt)

    def params(m):
        if case.startswith("pool"):
            return pd.pool_params(m, h, w, c, 2 if case == "pool2" else 3, stride, case != "pool2")
        return pd.conv_params(m, h, w, c, k, 1, 1) if conv else pd.depthwise_params(m, h, w, c, 1, 3, stride)

    p = params(n)
    dy = torch.randn(n, p.out_rows, p.out_cols, k, device="cuda", generator=g).to(dt)

    def run(lo, hi):
        q, xs, ds = params(hi - lo), x[lo:hi].reshape(-1), dy[lo:hi].reshape(-1)
        if case.startswith("pool"):
            y = pd.pooling(pd.POOL_MAX, 0, xs, q)
            return y, pd.pooling_max_grad(pd.POOL_MAX, xs, y, ds, q)
        if conv:
            return pd.conv2d(pd.FORWARD, xs, wt[:c * k], q), pd.conv2d(pd.INPUT_BACKPROP, ds, wt[:c * k], q)
        return pd.depthwise_conv2d(pd.FORWARD, xs, wt, q), pd.depthwise_conv2d(pd.INPUT_BACKPROP, ds, wt, q)

    whole = run(0, n)
    parts = [run(lo, min(lo + 5, n)) for lo in range(0, n, 5)]
    for i, a in enumerate(whole):
        assert torch.equal(a, torch.cat([q[i] for q in parts]))
    assert_no_device_error()


@pytest.mark.parametrize("dtype", ["f16", "bf16"])
@pytest.mark.parametrize("h,w,c,k,win,st", [(57, 61, 64, 64, 3, 1), (57, 61, 256, 256, 1, 1), (113, 97, 3, 64, 7, 2), (29, 30, 136, 520, 1, 2)])
def test_filter_gradient(h, w, c, k, win, st, dtype):
    """Against float64 sums of the same products: fp32 additions of at most 2^-20 of the terms' magnitudes, as for smaller batches."""
    dt, g = TORCH_DTYPES[dtype], torch.Generator(device="cuda").manual_seed(4)
    one = pd.conv_params(1, h, w, c, k, win, st)
    n = (72 << 20) // (2 * max(h * w * c, one.out_rows * one.out_cols * k)) + 1
    p = pd.conv_params(n, h, w, c, k, win, st)
    x = torch.randn(n, h, w, c, device="cuda", generator=g).to(dt)
    dy = torch.randn(n, p.out_rows, p.out_cols, k, device="cuda", generator=g).to(dt)
    below, right = (max((o - 1) * st + win - s - pad, 0) for o, s, pad in ((p.out_rows, h, p.pad_rows), (p.out_cols, w, p.pad_cols)))
    ref = mag = 0
    for lo in range(0, n, 8):
        xs = torch.nn.functional.pad(x[lo:lo + 8].double().permute(0, 3, 1, 2), (p.pad_cols, right, p.pad_rows, below))
        ds = dy[lo:lo + 8].double().permute(0, 3, 1, 2)
        grad = lambda a, b: torch.nn.grad.conv2d_weight(a, (k, c, win, win), b, stride=st).permute(2, 3, 1, 0)
        ref, mag = ref + grad(xs, ds), mag + grad(xs.abs(), ds.abs())
    dw = pd.conv2d(pd.FILTER_BACKPROP, x.reshape(-1), dy.reshape(-1), p, output_f32=True).view(ref.shape)
    assert ((dw.double() - ref).abs() - 2.0 ** -20 * mag).max() <= 0
    added = torch.zeros_like(dw).reshape(-1)
    pd.conv2d(pd.FILTER_BACKPROP, x.reshape(-1), dy.reshape(-1), p, out=added, output_f32=True, accumulate=True)
    assert ((added.view(ref.shape).double() - ref).abs() - 2.0 ** -20 * mag).max() <= 0
    assert_no_device_error()
