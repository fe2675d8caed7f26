"""Filter gradients of few-channel stems: four filter rows to a tile where the packed pixel has 4 channels (16 bits, even
column stride), two where it has 8; windows that fill the last tile and windows that do not."""
import pytest
import torch

import portdnn_b200 as pd
from gpu_util import TORCH_DTYPES, assert_no_device_error
from test_gpu_cluster_gemm import _rand

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["f16", "bf16"])
@pytest.mark.parametrize("n,h,w,c,k,win,st", [(2, 33, 41, 3, 64, 7, 2), (3, 64, 64, 3, 32, 3, 2), (1, 30, 21, 4, 72, 5, 2), (2, 17, 19, 1, 136, 8, 2),
                                              (2, 21, 22, 3, 64, 4, 2), (2, 20, 24, 3, 64, 2, 2), (2, 19, 23, 5, 64, 7, 2), (2, 19, 23, 3, 64, 3, 1)])
def test_against_float64(n, h, w, c, k, win, st, dtype):
    dt, g = TORCH_DTYPES[dtype], torch.Generator(device="cuda").manual_seed(h * c + k)
    p = pd.conv_params(n, h, w, c, k, win, st)
    x, dy = _rand(g, n, h, w, c).to(dt), _rand(g, n, p.out_rows, p.out_cols, k).to(dt)
    below, right = (max((o - 1) * st + win - s - pad, 0) for o, s, pad in ((p.out_rows, h, p.pad_rows), (p.out_cols, w, p.pad_cols)))
    xp = torch.nn.functional.pad(x.double().permute(0, 3, 1, 2), (p.pad_cols, right, p.pad_rows, below))
    grad = lambda a, b: torch.nn.grad.conv2d_weight(a, (k, c, win, win), b, stride=st).permute(2, 3, 1, 0)
    ref, mag = grad(xp, dy.double().permute(0, 3, 1, 2)), grad(xp.abs(), dy.double().abs().permute(0, 3, 1, 2))
    dw = pd.conv2d(pd.FILTER_BACKPROP, x.reshape(-1), dy.reshape(-1), p, output_f32=True)
    assert ((dw.view(ref.shape).double() - ref).abs() - 2.0 ** -20 * mag).max() <= 0
    before = dw.clone()
    pd.conv2d(pd.FILTER_BACKPROP, x.reshape(-1), dy.reshape(-1), p, out=dw, output_f32=True, accumulate=True)
    assert ((dw - 2 * before).abs().view(ref.shape).double() <= 2.0 ** -20 * mag).all()
    rounded = pd.conv2d(pd.FILTER_BACKPROP, x.reshape(-1), dy.reshape(-1), p)
    assert torch.equal(rounded, before.to(dt))
    assert_no_device_error()
