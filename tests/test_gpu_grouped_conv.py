"""Grouped convolutions whose groups share the column tiles of one launch (umma_gemm_grouped_kernel) against a
double-precision convolution: every group width it takes, a last tile with fewer groups, windows with and
without halo copies, stride 2, both filter layouts, bias and activation."""
import pytest
import torch

import portdnn_b200 as pd
from gpu_util import TORCH_DTYPES, assert_no_device_error

pytestmark = pytest.mark.gpu

UNIT = {"f16": 2.0 ** -11, "bf16": 2.0 ** -8}

# n, h, w, groups, channels per group, features per group, window, stride
SHAPES = [
    (2, 16, 24, 32, 16, 16, 3, 1),  # halo copies, resident tile per CTA
    (3, 13, 11, 6, 16, 16, 3, 1),   # a last tile of two groups, ragged rows
    (2, 15, 14, 8, 32, 32, 3, 2),   # parity maps
    (1, 9, 10, 7, 32, 64, 1, 1),    # a last tile of one group
    (2, 12, 12, 5, 48, 64, 3, 1),   # three slices of a step
    (2, 14, 14, 6, 64, 64, 3, 1),
    (2, 14, 14, 6, 64, 64, 5, 1),   # a filter too large to stay in shared memory: one GEMM per group
    (1, 1, 1, 5, 16, 64, 1, 1),     # tiles of 256 features, one pixel
]


@pytest.mark.parametrize("dtype", ["f16", "bf16"])
@pytest.mark.parametrize("fhwc", [False, True])
@pytest.mark.parametrize("shape", SHAPES)
def test_grouped_forward(shape, fhwc, dtype):
    n, h, w, groups, cg, kg, win, st = shape
    c, k, dt = groups * cg, groups * kg, TORCH_DTYPES[dtype]
    g = torch.Generator(device="cuda").manual_seed(c + k)
    p = pd.conv_params(n, h, w, c, k, win, st, groups=groups, filter_format=2 if fhwc else 0)
    x = torch.randn(n, h, w, c, device="cuda", generator=g).to(dt)
    wt = (torch.randn(win, win, cg, k, device="cuda", generator=g) / (win * win * cg) ** 0.5).to(dt)
    b = torch.randn(k, device="cuda", generator=g).to(dt)
    x[0, 0, 0, :cg] = float("inf")  # an overflow in the first group stays there
    below, right = (max((o - 1) * st + win - s - pad, 0) for o, s, pad in ((p.out_rows, h, p.pad_rows), (p.out_cols, w, p.pad_cols)))
    xp = torch.nn.functional.pad(x.double().permute(0, 3, 1, 2), (p.pad_cols, right, p.pad_rows, below))
    w64 = wt.double().permute(3, 2, 0, 1)
    ref = torch.nn.functional.conv2d(xp[:, cg:], w64[kg:], stride=st, groups=groups - 1).permute(0, 2, 3, 1)
    mag = torch.nn.functional.conv2d(xp[:, cg:].abs(), w64[kg:].abs(), stride=st, groups=groups - 1).permute(0, 2, 3, 1)
    wd = wt.permute(3, 0, 1, 2).contiguous() if fhwc else wt
    before = pd.launch_count()
    y = pd.conv2d(pd.FORWARD, x.reshape(-1), wd.reshape(-1), p).view(n, p.out_rows, p.out_cols, k)[..., kg:].double()
    assert pd.launch_count() - before == 2
    assert pd.last_gemm_kernel() == ("umma_gemm_multi_kernel" if win == 5 else "umma_gemm_grouped_kernel")
    yb = pd.conv2d(pd.FORWARD, x.reshape(-1), wd.reshape(-1), p, bias=b, activation=pd.ACT_RELU)
    yb = yb.view(n, p.out_rows, p.out_cols, k)[..., kg:].double()
    assert_no_device_error()
    # one rounding of a sum whose fp32 additions lose at most 2^-20 of the terms' magnitudes; with a bias the
    # sum is rounded before it is added
    bound = UNIT[dtype] * (ref.abs() + 2.0 ** -13) * 1.01 + 2.0 ** -20 * mag
    assert ((y - ref).abs() <= bound).all()
    refb = (ref + b[kg:].double()).relu()
    assert ((yb - refb).abs() <= bound + UNIT[dtype] * refb * 1.01).all()
