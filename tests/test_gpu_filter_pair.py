"""Filter gradients of whole 256 x 256 tiles.  On clusters of two CTAs (umma_gemm_filter_pair_kernel), where every
split has 16 pixel boxes or more: one and several splits, the last of them shorter, several tiles either way,
stride 2, pixel boxes cut at each edge, and the three ways the sums end (added to an fp32 gradient, written as
fp32, reduced to the tensors' type); and on tiles of one CTA below that."""
import pytest
import torch

import portdnn_b200 as pd
from gpu_util import TORCH_DTYPES, assert_no_device_error

pytestmark = pytest.mark.gpu

# n, h, w, c, k, window, stride
SHAPES = [
    (24, 14, 14, 256, 256, 3, 1),
    (70, 9, 11, 256, 512, 1, 1),
    (33, 15, 17, 512, 256, 3, 2),
    (17, 8, 8, 768, 768, 3, 1),  # more tiles than clusters: one split
]
# at 148 SMs: splits, boxes of the others / of the last split; edges at which boxes of 64 pixels are cut
PAIR_SHAPES = [
    (17, 8, 8, 768, 768, 3, 1),     # 1, 17
    (43, 14, 14, 256, 256, 3, 1),   # 8, 19 / 14; images
    (131, 21, 19, 256, 512, 1, 1),  # 36, 26 / 25; columns, rows, images
    (67, 11, 13, 512, 512, 3, 2),   # 2, 26 / 25; columns, images
    (37, 29, 27, 512, 256, 3, 2),   # 4, 34 / 31; rows, images
]


@pytest.mark.parametrize("dtype", ["f16", "bf16"])
@pytest.mark.parametrize("shape", SHAPES + PAIR_SHAPES[1:])
def test_filter_gradient(shape, dtype):
    kernel = "umma_gemm_filter_pair_kernel" if shape in PAIR_SHAPES else "umma_gemm_kernel"
    n, h, w, c, k, win, st = shape
    dt, g = TORCH_DTYPES[dtype], torch.Generator(device="cuda").manual_seed(c + k)
    p = pd.conv_params(n, h, w, c, k, win, st)
    x = torch.randn(n, h, w, c, device="cuda", generator=g).to(dt)
    dy = torch.randn(n, p.out_rows, p.out_cols, k, device="cuda", generator=g).to(dt)
    below, right = (max((o - 1) * st + win - s - pad, 0) for o, s, pad in ((p.out_rows, h, p.pad_rows), (p.out_cols, w, p.pad_cols)))
    xp = torch.nn.functional.pad(x.double(), (0, 0, p.pad_cols, right, p.pad_rows, below))
    d2 = dy.double().reshape(-1, k)
    ref, mag = torch.empty(win, win, c, k, device="cuda", dtype=torch.float64), torch.empty(win, win, c, k, device="cuda", dtype=torch.float64)
    for r in range(win):
        for s in range(win):
            a = xp[:, r:r + (p.out_rows - 1) * st + 1:st, s:s + (p.out_cols - 1) * st + 1:st].reshape(-1, c)
            ref[r, s], mag[r, s] = a.T @ d2, a.abs().T @ d2.abs()
    # fp32 sums that lose at most 2^-20 of the magnitudes of their terms, then at most one rounding
    slack = 2.0 ** -20 * mag
    f32 = pd.conv2d(pd.FILTER_BACKPROP, x.reshape(-1), dy.reshape(-1), p, output_f32=True).view(ref.shape)
    assert pd.last_gemm_kernel() == kernel
    assert ((f32.double() - ref).abs() <= slack).all()
    own = pd.conv2d(pd.FILTER_BACKPROP, x.reshape(-1), dy.reshape(-1), p).view(ref.shape)
    assert pd.last_gemm_kernel() == kernel
    unit = 2.0 ** -11 if dtype == "f16" else 2.0 ** -8
    assert ((own.double() - ref).abs() <= slack + 1.01 * unit * ref.abs()).all()
    total = torch.ones_like(f32).reshape(-1)
    pd.conv2d(pd.FILTER_BACKPROP, x.reshape(-1), dy.reshape(-1), p, out=total, output_f32=True, accumulate=True)
    assert pd.last_gemm_kernel() == kernel
    assert ((total.view(ref.shape).double() - 1.0 - ref).abs() <= slack + 2.0 ** -20).all()
    assert_no_device_error()
