"""Pairs of row tiles, and pairs of CTAs in filter gradients, on tensors that are read from the end: an odd number of tiles of
pixels, whose last pair, half empty, is visited first; pixel splits of whole filter tiles that go through the batch side by
side."""
import pytest
import torch

import portdnn_b200 as pd
from gpu_util import TORCH_DTYPES, assert_no_device_error
from launched import launched

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["f16", "bf16"])
def test_row_tiles_in_pairs(dtype):
    """1024 -> 128 forward and 128 <- 1024 backward, 1x1: 16 reduction steps, 317 row tiles, 159 pairs for 148 SMs; 83 MB are read.
    The images in fives, which fill too few pairs, have the same results, bit for bit."""
    dt, g = TORCH_DTYPES[dtype], torch.Generator(device="cuda").manual_seed(8)
    n, h, w, wide, narrow = 29, 31, 45, 1024, 128
    assert -(-n * h * w // 128) == 317
    x = torch.randn(n, h, w, wide, device="cuda", generator=g).to(dt)
    f = (torch.randn(wide * narrow, device="cuda", generator=g) * 0.05).to(dt)
    for which, c, k in ((pd.FORWARD, wide, narrow), (pd.INPUT_BACKPROP, narrow, wide)):
        run = lambda t: pd.conv2d(which, t.reshape(-1), f, pd.conv_params(t.shape[0], h, w, c, k, 1, 1)).view(-1, h, w, narrow)  # noqa: E731
        whole = run(x)
        kernels = launched(lambda: run(x))
        assert len(kernels) == 1 and "umma_gemm_kernel" in kernels[0].name and (kernels[0].threads, kernels[0].blocks) == (384, 148)
        assert torch.equal(whole, torch.cat([run(x[i:i + 5]) for i in range(0, n, 5)]))
        wt = f.double().view(wide, narrow) if which == pd.FORWARD else f.double().view(narrow, wide).T
        ref, mag = x.double() @ wt, x.double().abs() @ wt.abs()
        unit = {"f16": 2.0 ** -11, "bf16": 2.0 ** -8}[dtype]
        assert ((whole.double() - ref).abs() - (unit * (ref.abs() + 2.0 ** -13) * 1.01 + 2.0 ** -20 * mag)).max() <= 0
    assert_no_device_error()


@pytest.mark.parametrize("dtype", ["f16", "bf16"])
@pytest.mark.parametrize("c,k,win", [(512, 256, 1), (256, 512, 3)])
def test_filter_tiles_on_pairs_of_ctas(c, k, win, dtype):
    """Against float64 sums of the same products: fp32 additions of at most 2^-20 of the terms' magnitudes."""
    dt, g = TORCH_DTYPES[dtype], torch.Generator(device="cuda").manual_seed(9)
    n, h, w = 27, 53, 49
    p = pd.conv_params(n, h, w, c, k, win, 1)
    x, dy = torch.randn(n, h, w, c, device="cuda", generator=g).to(dt), torch.randn(n, h, w, k, device="cuda", generator=g).to(dt)
    assert max(x.numel(), dy.numel()) * 2 > 64 << 20
    call = lambda: pd.conv2d(pd.FILTER_BACKPROP, x.reshape(-1), dy.reshape(-1), p, output_f32=True)  # noqa: E731
    kernels = [k_ for k_ in launched(call) if "umma_gemm" in k_.name]
    assert len(kernels) == 1 and "filter_pair" in kernels[0].name
    ref = mag = 0
    for i in range(n):
        xs, ds = x[i:i + 1].double().permute(0, 3, 1, 2), dy[i:i + 1].double().permute(0, 3, 1, 2)
        grad = lambda a, b: torch.nn.grad.conv2d_weight(a, (k, c, win, win), b, padding=win // 2).permute(2, 3, 1, 0)  # noqa: E731
        ref, mag = ref + grad(xs, ds), mag + grad(xs.abs(), ds.abs())
    dw = call().view(ref.shape)
    assert ((dw.double() - ref).abs() - 2.0 ** -20 * mag).max() <= 0
    added = dw.clone().reshape(-1)
    pd.conv2d(pd.FILTER_BACKPROP, x.reshape(-1), dy.reshape(-1), p, out=added, output_f32=True, accumulate=True)
    assert ((added.view(ref.shape).double() - 2 * ref).abs() - 2.0 ** -19 * mag).max() <= 0
    assert_no_device_error()
