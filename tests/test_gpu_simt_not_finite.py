"""fp32 tiles with infinities and NaN: a tap outside the image has no term, in every pass, order of the filter and form of the
sum; the second look that this takes is no slower than a few calls."""
import pytest
import torch

import portdnn_b200 as pd

pytestmark = pytest.mark.gpu

# images, rows, cols, channels, features, window, stride: remainders; strides that leave a phase without taps; sums shared by
# clusters and cut into slices; windows larger than the image; no tap outside
SHAPES = [(2, 9, 11, 17, 33, 3, 1), (3, 20, 17, 37, 65, 3, 2), (2, 13, 16, 5, 130, 2, 3), (8, 60, 61, 14, 18, 3, 1), (1, 8, 9, 133, 77, 5, 1),
          (2, 3, 2, 21, 23, 5, 1), (5, 30, 31, 13, 19, 1, 2), (8, 60, 61, 14, 18, 1, 1)]


def _same(got, want):
    """Equal where not finite, else apart by fp32 sums in another order (the direct kernel's): their terms are below 2^5 each."""
    got, want = got.double(), want.double()
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isinf(), want.isinf())
    assert torch.equal(got[got.isinf()], want[want.isinf()])
    ok = want.isfinite()
    assert not ok.any() or (got - want)[ok].norm() <= 2.0 ** -19 * want[ok].norm().clamp(min=1)


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("fhwc", [False, True])
def test_against_the_direct_kernel(shape, fhwc):
    n, h, w, c, k, win, st = shape
    p = pd.conv_params(n, h, w, c, k, win, st, filter_format=2 if fhwc else 0)
    g = torch.Generator(device="cuda").manual_seed(5)
    x, f = torch.randn(n, h, w, c, device="cuda", generator=g), torch.randn(win, win, c, k, device="cuda", generator=g)
    dy = torch.randn(n, p.out_rows, p.out_cols, k, device="cuda", generator=g)
    f[0, 0, 0, 0] = float("inf")
    f[-1, -1, c - 1, 1] = -float("inf")
    f[0, -1, 0, k - 1] = float("nan")
    dy[0, 0, 0, 0] = float("inf")
    dy[n - 1, -1, -1, 2] = float("nan")
    order = (3, 0, 1, 2) if fhwc else (0, 1, 2, 3)
    f = f.permute(order).contiguous().reshape(-1)
    x, dy = x.reshape(-1), dy.reshape(-1)
    for which, a, b in ((pd.FORWARD, x, f), (pd.INPUT_BACKPROP, dy, f), (pd.FILTER_BACKPROP, x, dy)):
        _same(pd.conv2d(which, a, b, p), pd.conv2d(which, a, b, p, algorithm=pd.ALGO_DIRECT))


def test_the_second_look_takes_a_few_calls():
    p = pd.conv_params(24, 60, 61, 66, 97, 3, 1)
    g = torch.Generator(device="cuda").manual_seed(6)
    x = torch.randn(24 * 60 * 61 * 66, device="cuda", generator=g)
    dy = torch.randn(24 * 60 * 61 * 97, device="cuda", generator=g)

    def time():
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        pd.conv2d(pd.FILTER_BACKPROP, x, dy, p)
        a.record()
        for _ in range(3):
            pd.conv2d(pd.FILTER_BACKPROP, x, dy, p)
        b.record()
        b.synchronize()
        return a.elapsed_time(b)

    clean = time()
    dy[:97] = float("nan")  # one pixel: all of the gradient
    assert time() <= 8 * clean  # one pass more, one term at a time: about four
