"""GEMMs of at most two tiles to an SM: one tile to a CTA, two CTAs to an SM, the staging slices in the place of the ring
(the solo form of umma_gemm_kernel), in all three passes, and launches that overlap their predecessors."""
import pytest
import torch

import portdnn_b200 as pd
from gpu_util import TORCH_DTYPES
from test_gpu_cluster_gemm import _check, _rand

pytestmark = pytest.mark.gpu

# n, h, w, c, k, window
SHAPES = [
    (1, 8, 16, 64, 64, 1),      # one tile, one step
    (2, 9, 15, 72, 200, 3),     # ragged rows, columns and blocks
    (9, 16, 16, 136, 64, 1),    # fewer steps than stages
    (37, 16, 8, 256, 1024, 1),  # tiles of 128 columns, exactly two to an SM of 148
    (38, 16, 8, 256, 1024, 1),  # one row of tiles more: the persistent form
    (5, 12, 20, 520, 72, 1),    # a long reduction
    (3, 10, 11, 40, 320, 5),
]


@pytest.mark.parametrize("dtype", ["f16", "bf16"])
@pytest.mark.parametrize("fhwc", [False, True])
@pytest.mark.parametrize("shape", SHAPES)
def test_passes(shape, fhwc, dtype):
    n, h, w, c, k, win = shape
    dt, g, lo = TORCH_DTYPES[dtype], torch.Generator(device="cuda").manual_seed(h * c + k), win // 2
    p = pd.conv_params(n, h, w, c, k, win, 1, filter_format=2 if fhwc else 0)
    x, dy, b = _rand(g, n, h, w, c).to(dt), _rand(g, n, h, w, k).to(dt), _rand(g, k).to(dt)
    wt = (_rand(g, win, win, c, k) / (win * win * c) ** 0.5).to(dt)
    wd = (wt.permute(3, 0, 1, 2).contiguous() if fhwc else wt).reshape(-1)
    w64, x64, dy64 = wt.double().permute(3, 2, 0, 1), x.double().permute(0, 3, 1, 2), dy.double().permute(0, 3, 1, 2)
    nhwc = lambda t: t.permute(0, 2, 3, 1)
    conv = torch.nn.functional.conv2d
    ref, mag = nhwc(conv(x64, w64, padding=lo)), nhwc(conv(x64.abs(), w64.abs(), padding=lo))
    for const in (False, True):
        y = pd.conv2d(pd.FORWARD, x.reshape(-1), wd, p, bias=b, activation=pd.ACT_RELU, constant_filter=const).view(ref.shape)
        _check(y, (ref + b.double()).relu(), mag + b.double().abs(), dtype, before_bias=ref)
    back = torch.nn.functional.conv_transpose2d
    ref, mag = nhwc(back(dy64, w64, padding=lo)), nhwc(back(dy64.abs(), w64.abs(), padding=lo))
    keep = _rand(g, n, h, w, c).relu().to(dt)
    dx = pd.conv2d(pd.INPUT_BACKPROP, dy.reshape(-1), wd, p, relu_forward_output=keep.reshape(-1)).view(ref.shape)
    _check(dx, ref * (keep > 0), mag, dtype)
    if not fhwc:  # fp32 sums: what their additions lose, no rounding to 16 bits
        grad = lambda a, d: torch.nn.grad.conv2d_weight(a, w64.shape, d, padding=lo).permute(2, 3, 1, 0)
        ref, mag = grad(x64, dy64), grad(x64.abs(), dy64.abs())
        dw = pd.conv2d(pd.FILTER_BACKPROP, x.reshape(-1), dy.reshape(-1), p, output_f32=True).view(ref.shape)
        assert ((dw.double() - ref).abs() - 2.0 ** -20 * mag).max() <= 0


def test_each_launch_waits_for_its_predecessor():
    """A chain of layers each of which reads what the one before has written, with and without a pause between them."""
    n, h, c = 24, 14, 256
    g = torch.Generator(device="cuda").manual_seed(1)
    p = pd.conv_params(n, h, h, c, c, 1, 1)
    ws = [(_rand(g, c * c) * (2.0 / c) ** 0.5).half() for _ in range(16)]
    x = _rand(g, n * h * h * c).half()

    def run(pause):
        a = x
        for w in ws:
            a = pd.conv2d(pd.FORWARD, a, w, p, activation=pd.ACT_RELU, constant_filter=True)
            if pause:
                torch.cuda.synchronize()
        return a

    want = run(True)
    for _ in range(5):
        assert torch.equal(run(False), want)
