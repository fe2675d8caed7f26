"""fp32 tiles on the CUDA cores (simt_gemm.cu): fp32 convolutions of odd channel and feature counts in all three
passes, filters in both orders, and matrix products of odd sizes, against float64."""
import pytest
import torch
import torch.nn.functional as F

import portdnn_b200 as pd

pytestmark = pytest.mark.gpu

DT = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}
# rounding of the result, then of up to n fp32 additions of terms of one size, whose errors add up as sqrt(n)
ULP = {"f32": 2.0 ** -24, "f16": 2.0 ** -11, "bf16": 2.0 ** -8}


def _rel(got, ref):
    return ((got.double() - ref).norm() / ref.norm().clamp(min=1e-30)).item()


def _bound(dtype, terms):
    return ULP[dtype] + 2.0 ** -24 * (terms ** 0.5 + 4)


# (images, rows, cols, channels, features, window, stride, dtype): one term and one output; tiles of 64 and of 128 rows with
# remainders; clusters of 1 to 8 blocks; a long sum in slices; strides that leave a phase without taps; more than one chunk
# of terms to a tap; 16-bit layers too small for padded copies
SHAPES = [(1, 1, 1, 1, 1, 1, 1, "f32"), (2, 9, 11, 17, 33, 3, 1, "f32"), (3, 20, 17, 37, 65, 3, 2, "f32"), (1, 8, 9, 133, 77, 5, 1, "f32"),
          (5, 30, 31, 13, 19, 1, 2, "f32"), (8, 60, 61, 14, 18, 1, 1, "f32"), (2, 13, 16, 5, 130, 2, 3, "f32"), (16, 40, 41, 66, 97, 3, 1, "f32"),
          (2, 13, 15, 21, 11, 1, 1, "f16"), (1, 9, 7, 13, 29, 3, 3, "bf16"), (2, 21, 19, 16, 24, 3, 4, "f16")]


def _reference(x, w, p, dy):
    """Output and gradients in float64, NHWC and HWCF."""
    x = x.double().cpu().permute(0, 3, 1, 2).requires_grad_()
    w = w.double().cpu().permute(3, 2, 0, 1).requires_grad_()
    below = max((p.out_rows - 1) * p.stride_rows + p.window_rows - p.in_rows - p.pad_rows, 0)
    right = max((p.out_cols - 1) * p.stride_cols + p.window_cols - p.in_cols - p.pad_cols, 0)
    y = F.conv2d(F.pad(x, (p.pad_cols, right, p.pad_rows, below)), w, stride=(p.stride_rows, p.stride_cols))[:, :, :p.out_rows, :p.out_cols]
    y.backward(dy.double().cpu().permute(0, 3, 1, 2))
    return y.detach().permute(0, 2, 3, 1), x.grad.permute(0, 2, 3, 1), w.grad.permute(2, 3, 1, 0)


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("fhwc", [False, True])
def test_passes(shape, fhwc):
    n, h, w, c, k, win, st, dtype = shape
    p = pd.conv_params(n, h, w, c, k, win, st, filter_format=2 if fhwc else 0)
    g = torch.Generator(device="cuda").manual_seed(3)
    rand = lambda *s: torch.randn(*s, device="cuda", generator=g).to(DT[dtype])  # noqa: E731
    x, f, dy = rand(n, h, w, c), rand(win, win, c, k), rand(n, p.out_rows, p.out_cols, k)
    y, dx, df = _reference(x, f, p, dy)
    order = (3, 0, 1, 2) if fhwc else (0, 1, 2, 3)
    stored = f.permute(order).contiguous().reshape(-1)
    xf, dyf = x.reshape(-1), dy.reshape(-1)
    assert _rel(pd.conv2d(pd.FORWARD, xf, stored, p).cpu().view(y.shape), y) <= _bound(dtype, win * win * c)
    assert _rel(pd.conv2d(pd.INPUT_BACKPROP, dyf, stored, p).cpu().view(dx.shape), dx) <= _bound(dtype, win * win * k)
    got = pd.conv2d(pd.FILTER_BACKPROP, xf, dyf, p).cpu().view(df.permute(order).shape)
    assert _rel(got, df.permute(order)) <= _bound(dtype, dy.numel() // k)
    again = pd.conv2d(pd.FILTER_BACKPROP, xf, dyf, p).cpu().view(got.shape)
    assert torch.equal(got, again)


def test_a_tap_outside_the_image_has_no_term():
    """Filters and gradients that are infinite where only the border meets them."""
    p = pd.conv_params(1, 5, 5, 7, 9, 3, 1)
    x, w = torch.ones(5 * 5 * 7, device="cuda"), torch.ones(3, 3, 7, 9, device="cuda")
    w[0, 0, 0, 0] = float("inf")
    args = (x, w.reshape(-1), p)
    assert torch.equal(pd.conv2d(pd.FORWARD, *args), pd.conv2d(pd.FORWARD, *args, algorithm=pd.ALGO_DIRECT))
    dy = torch.ones(5 * 5 * 9, device="cuda")
    args = (dy, w.reshape(-1), p)
    assert torch.equal(pd.conv2d(pd.INPUT_BACKPROP, *args), pd.conv2d(pd.INPUT_BACKPROP, *args, algorithm=pd.ALGO_DIRECT))
    dy[0] = float("inf")
    args = (x, dy, p)
    assert torch.equal(pd.conv2d(pd.FILTER_BACKPROP, *args), pd.conv2d(pd.FILTER_BACKPROP, *args, algorithm=pd.ALGO_DIRECT))


def test_an_image_alone_and_in_a_batch():
    one, many = pd.conv_params(1, 14, 15, 45, 51, 3, 1), pd.conv_params(40, 14, 15, 45, 51, 3, 1)
    g = torch.Generator(device="cuda").manual_seed(5)
    x = torch.randn(40 * 14 * 15 * 45, device="cuda", generator=g)
    w = torch.randn(9 * 45 * 51, device="cuda", generator=g)
    y = pd.conv2d(pd.FORWARD, x, w, many).view(40, -1)
    for i in (0, 39):
        assert torch.equal(pd.conv2d(pd.FORWARD, x.view(40, -1)[i].contiguous(), w, one), y[i])


@pytest.mark.parametrize("dtype", ["f32", "f16", "bf16"])
@pytest.mark.parametrize("tl,tr", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("sizes", [(1, 1, 1, 1), (1, 2, 1009, 543), (3, 65, 17, 33), (1, 127, 15, 31), (1, 250, 513, 129), (2, 130, 301, 20), (2000, 3, 5, 2)])
def test_products(sizes, tl, tr, dtype):
    b, m, k, n = sizes
    g = torch.Generator(device="cuda").manual_seed(7)
    lhs = torch.randn(b, k, m, device="cuda", generator=g).to(DT[dtype]) if tl else torch.randn(b, m, k, device="cuda", generator=g).to(DT[dtype])
    rhs = torch.randn(b, n, k, device="cuda", generator=g).to(DT[dtype]) if tr else torch.randn(b, k, n, device="cuda", generator=g).to(DT[dtype])
    out = torch.randn(b, m, n, device="cuda", generator=g).to(DT[dtype])
    ref = (lhs.double().mT if tl else lhs.double()) @ (rhs.double().mT if tr else rhs.double())
    got = pd.matmul(lhs.reshape(-1), rhs.reshape(-1), b, m, k, n, tl, tr).view(b, m, n)
    assert _rel(got, ref) <= _bound(dtype, k)
    ref = ref + 0.5 * out.double()
    pd.matmul(lhs.reshape(-1), rhs.reshape(-1), b, m, k, n, tl, tr, beta=0.5, out=out.view(-1))
    assert _rel(out, ref) <= _bound(dtype, k)
