"""GEMMs of few tiles whose reduction is shared by the CTAs of a cluster (umma_gemm_cluster_kernel): forward
pass, stride-1 input backprop with its fused forms, and matmul, at 2, 4 and 8 CTAs to a tile, with
ragged rows, columns and reduction blocks."""
import pytest
import torch

import portdnn_b200 as pd
from gpu_util import TORCH_DTYPES, assert_no_device_error

pytestmark = pytest.mark.gpu

UNIT = {"f16": 2.0 ** -11, "bf16": 2.0 ** -8}  # half a unit in the last place: one rounding


def _rand(g, *shape):
    return torch.randn(*shape, device="cuda", generator=g, dtype=torch.float64)


def _check(got, ref, magnitude, dtype, before_bias=None):
    """One rounding of a sum whose fp32 additions lose at most 2^-20 of the sum of the terms' magnitudes.  With
    a bias the sum is rounded before it is added, so half a unit of that sum joins half a unit of the result
    (whichever is the larger of the two)."""
    assert_no_device_error()
    rounded = ref.abs() if before_bias is None else ref.abs() + before_bias.abs()
    bound = UNIT[dtype] * (rounded + 2.0 ** -13) * 1.01 + 2.0 ** -20 * magnitude
    worst = ((got.double() - ref).abs() - bound).max()
    assert worst <= 0, float(worst)


# n, h, w, c, k, window, stride
SHAPES = [
    (1, 7, 7, 512, 512, 3, 1),     # 8 CTAs, one ragged row tile
    (1, 14, 14, 1024, 256, 1, 1),  # 4
    (1, 28, 40, 520, 136, 1, 1),   # 2, last reduction block and column tile of 8
    (1, 13, 11, 72, 40, 3, 1),     # taps of two blocks, the second of 8 channels; fewer columns than a tile
    (1, 15, 17, 256, 200, 3, 2),   # strided: parity maps
    (1, 5, 6, 136, 72, 5, 1),
]


@pytest.mark.parametrize("dtype", ["f16", "bf16"])
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("fhwc", [False, True])
@pytest.mark.parametrize("any_order", [False, True])
def test_conv(shape, dtype, fhwc, any_order):
    n, h, w, c, k, win, st = shape
    dt, g = TORCH_DTYPES[dtype], torch.Generator(device="cuda").manual_seed(h * c + k)
    p = pd.conv_params(n, h, w, c, k, win, st, filter_format=2 if fhwc else 0)
    x, wt, b = _rand(g, n, h, w, c).to(dt), (_rand(g, win, win, c, k) / (win * win * c) ** 0.5).to(dt), _rand(g, k).to(dt)
    wd = wt.permute(3, 0, 1, 2).contiguous() if fhwc else wt
    below, right = (max((o - 1) * st + win - s - pad, 0) for o, s, pad in ((p.out_rows, h, p.pad_rows), (p.out_cols, w, p.pad_cols)))
    xp = torch.nn.functional.pad(x.double().permute(0, 3, 1, 2), (p.pad_cols, right, p.pad_rows, below))
    w64 = wt.double().permute(3, 2, 0, 1)
    ref = torch.nn.functional.conv2d(xp, w64, stride=st).permute(0, 2, 3, 1)
    mag = torch.nn.functional.conv2d(xp.abs(), w64.abs(), stride=st).permute(0, 2, 3, 1)
    y = pd.conv2d(pd.FORWARD, x.reshape(-1), wd.reshape(-1), p, any_order=any_order).view(ref.shape)
    assert pd.last_gemm_kernel() == ("umma_gemm_cluster_kernel" if any_order else "umma_gemm_kernel")
    _check(y, ref, mag, dtype)
    assert torch.equal(y, pd.conv2d(pd.FORWARD, x.reshape(-1), wd.reshape(-1), p, constant_filter=True,
                                    any_order=any_order).view(ref.shape))
    bits = torch.zeros(y.numel() // 8, dtype=torch.uint8, device="cuda")
    yb = pd.conv2d(pd.FORWARD, x.reshape(-1), wd.reshape(-1), p, bias=b, activation=pd.ACT_RELU, relu_bitmask=bits,
                   any_order=any_order).view(ref.shape)
    _check(yb, (ref + b.double()).relu(), mag + b.double().abs(), dtype, before_bias=ref)
    unpacked = (bits[:, None] >> torch.arange(8, device="cuda", dtype=torch.uint8)) & 1
    assert torch.equal(unpacked.view(ref.shape).bool(), yb > 0)


@pytest.mark.parametrize("dtype", ["f16", "bf16", "f32"])
@pytest.mark.parametrize("shape", SHAPES)
def test_an_image_alone_and_in_a_batch(shape, dtype):
    """Without any_order an image's result has the same bits whatever is beside it."""
    _, h, w, c, k, win, st = shape
    dt, g = TORCH_DTYPES[dtype], torch.Generator(device="cuda").manual_seed(h * c + k)
    x, wt, b = _rand(g, 5, h, w, c).to(dt), (_rand(g, win, win, c, k) / (win * win * c) ** 0.5).to(dt), _rand(g, k).to(dt)
    call = lambda xs: pd.conv2d(pd.FORWARD, xs.reshape(-1), wt.reshape(-1), pd.conv_params(len(xs), h, w, c, k, win, st),
                                bias=b, activation=pd.ACT_RELU, constant_filter=True).view(len(xs), -1)
    for many in (2, 3, 5):
        together = call(x[:many])
        assert all(torch.equal(together[i], call(x[i:i + 1])[0]) for i in range(many))
    assert_no_device_error()


@pytest.mark.parametrize("dtype", ["f16", "bf16"])
@pytest.mark.parametrize("shape", [s for s in SHAPES if s[6] == 1] + [(1, 12, 10, 24, 520, 1, 1), (3, 5, 6, 136, 72, 5, 1), (1, 14, 14, 256, 1024, 1, 1)])
def test_input_backprop(shape, dtype):
    n, h, w, c, k, win, _ = shape
    dt, g = TORCH_DTYPES[dtype], torch.Generator(device="cuda").manual_seed(h + c + k)
    p = pd.conv_params(n, h, w, c, k, win, 1)
    dy, wt = _rand(g, n, h, w, k).to(dt), (_rand(g, win, win, c, k) / (win * win * k) ** 0.5).to(dt)
    w64, lo = wt.double().permute(3, 2, 0, 1), win // 2
    back = lambda a, f: torch.nn.functional.conv_transpose2d(a.permute(0, 3, 1, 2), f, padding=lo).permute(0, 2, 3, 1)
    ref, mag = back(dy.double(), w64), back(dy.double().abs(), w64.abs())
    call = lambda **kw: pd.conv2d(pd.INPUT_BACKPROP, dy.reshape(-1), wt.reshape(-1), p, **kw).view(ref.shape)
    plain = call()
    # (fewer than eight blocks of 64 features, one tap: nothing to share)
    assert pd.last_gemm_kernel() == ("umma_gemm_kernel" if win == 1 and k <= 7 * 64 else "umma_gemm_cluster_kernel")
    _check(plain, ref, mag, dtype)
    fwd, before = _rand(g, n, h, w, c).relu().to(dt), _rand(g, n, h, w, c).to(dt)
    keep = fwd > 0
    assert torch.equal(call(relu_forward_output=fwd.reshape(-1)), plain * keep)
    bits = (keep.reshape(-1, 8).to(torch.uint8) << torch.arange(8, device="cuda", dtype=torch.uint8)).sum(1).to(torch.uint8)
    assert torch.equal(call(relu_bitmask=bits), plain * keep)
    out = before.clone().reshape(-1)
    call(out=out, accumulate=1, relu_forward_output=fwd.reshape(-1))
    assert torch.equal(out.view(ref.shape), (plain + before) * keep)


@pytest.mark.parametrize("dtype", ["f16", "bf16"])
@pytest.mark.parametrize("batches,m,k,n,tr", [(1, 250, 2048, 1000, False), (1, 250, 1000, 2048, True), (3, 30, 520, 72, False),
                                              (1, 1, 4096, 8, True), (2, 129, 512, 64, False)])
def test_matmul(batches, m, k, n, tr, dtype):
    dt, g = TORCH_DTYPES[dtype], torch.Generator(device="cuda").manual_seed(m + n)
    a, b = _rand(g, batches, m, k).to(dt), (_rand(g, batches, k, n) / k ** 0.5).to(dt)
    bd = b.transpose(1, 2).contiguous() if tr else b
    out = pd.matmul(a.reshape(-1), bd.reshape(-1), batches, m, k, n, transpose_rhs=tr).view(batches, m, n)
    assert pd.last_gemm_kernel() == "umma_gemm_cluster_kernel"
    _check(out, a.double() @ b.double(), a.double().abs() @ b.double().abs(), dtype)


@pytest.mark.parametrize("dtype", ["f16", "bf16"])
@pytest.mark.parametrize("batch", [2, 5])
@pytest.mark.parametrize("shape", [(7, 7, 512, 512, 3, 1), (13, 11, 72, 40, 3, 1), (15, 17, 256, 200, 3, 2), (14, 14, 1024, 256, 1, 1)])
def test_small_batches_in_any_order(shape, batch, dtype):
    """Several images to a row tile, and a last row tile that is not full."""
    h, w, c, k, win, st = shape
    dt, g = TORCH_DTYPES[dtype], torch.Generator(device="cuda").manual_seed(h * c + k + batch)
    p = pd.conv_params(batch, h, w, c, k, win, st)
    x, wt = _rand(g, batch, h, w, c).to(dt), (_rand(g, win, win, c, k) / (win * win * c) ** 0.5).to(dt)
    below, right = (max((o - 1) * st + win - s - pad, 0) for o, s, pad in ((p.out_rows, h, p.pad_rows), (p.out_cols, w, p.pad_cols)))
    xp = torch.nn.functional.pad(x.double().permute(0, 3, 1, 2), (p.pad_cols, right, p.pad_rows, below))
    w64 = wt.double().permute(3, 2, 0, 1)
    ref = torch.nn.functional.conv2d(xp, w64, stride=st).permute(0, 2, 3, 1)
    mag = torch.nn.functional.conv2d(xp.abs(), w64.abs(), stride=st).permute(0, 2, 3, 1)
    y = pd.conv2d(pd.FORWARD, x.reshape(-1), wt.reshape(-1), p, any_order=True).view(ref.shape)
    assert pd.last_gemm_kernel() == "umma_gemm_cluster_kernel"
    _check(y, ref, mag, dtype)
    assert_no_device_error()


@pytest.mark.parametrize("dtype", ["f16", "bf16"])
@pytest.mark.parametrize("shape", [(3, 90, 71, 64, 136, 3), (2, 100, 100, 520, 248, 1), (3, 80, 80, 72, 192, 3)])
def test_one_wide_column_tile(shape, dtype):
    """129 to 255 features and a row tile for every SM: one column tile of 192 or 256, its last columns not there."""
    n, h, w, c, k, win = shape
    dt, g = TORCH_DTYPES[dtype], torch.Generator(device="cuda").manual_seed(h * c + k)
    p = pd.conv_params(n, h, w, c, k, win, 1)
    x, wt = _rand(g, n, h, w, c).to(dt), (_rand(g, win, win, c, k) / (win * win * c) ** 0.5).to(dt)
    w64 = wt.double().permute(3, 2, 0, 1)
    xp = x.double().permute(0, 3, 1, 2)
    ref = torch.nn.functional.conv2d(xp, w64, padding=win // 2).permute(0, 2, 3, 1)
    mag = torch.nn.functional.conv2d(xp.abs(), w64.abs(), padding=win // 2).permute(0, 2, 3, 1)
    _check(pd.conv2d(pd.FORWARD, x.reshape(-1), wt.reshape(-1), p).view(ref.shape), ref, mag, dtype)
    assert_no_device_error()
