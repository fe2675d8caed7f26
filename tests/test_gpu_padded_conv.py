"""16-bit convolutions whose channel or feature count is not a multiple of 8, or whose tensors start off a
16-byte boundary: the tensor-core kernels on padded copies (padded_conv.cu) against the general direct
kernel, which reads the tensors as they are."""
import numpy as np
import pytest
import torch

import portdnn_b200 as pd
from gpu_util import assert_no_device_error, rounded, to_dev, to_host

pytestmark = pytest.mark.gpu

# Both sides add exact products in fp32 and round once (the forward pass with a bias twice): where the two
# orders of the sums fall on different sides of a rounding boundary they differ by one unit in the last
# place, 2^-10 (f16) or 2^-7 (bf16) of a value at most, in a small share of the values.  In the 2-norm that
# stays below half a unit.
HALF_UNIT = {"f16": 2.0 ** -11, "bf16": 2.0 ** -8}

SHAPES = [
    # n, h, w, c, k, window, stride: odd counts on either side, both, one multiple of 8, fewer than 8 channels,
    # packets of 1, 2 and 4 elements, stride 2
    (2, 23, 31, 13, 150, 3, 1),
    (3, 21, 17, 100, 152, 3, 1),
    (3, 21, 17, 104, 149, 1, 1),
    (2, 30, 33, 33, 65, 3, 2),
    (2, 64, 64, 3, 42, 7, 2),
    (9, 28, 28, 9, 257, 1, 1),
]


def _tensors(shape, dtype, fhwc=False):
    n, h, w, c, k, win, st = shape
    rng = np.random.default_rng(c + k)
    p = pd.conv_params(n, h, w, c, k, win, st, filter_format=2 if fhwc else 0)
    x = rng.standard_normal(n * h * w * c).astype(np.float32)
    wt = (rng.standard_normal(win * win * c * k) / np.sqrt(win * win * c)).astype(np.float32)
    dy = rng.standard_normal(n * p.out_rows * p.out_cols * k).astype(np.float32)
    b = rng.standard_normal(k).astype(np.float32)
    return (p,) + tuple(to_dev(rounded(t, dtype), dtype) for t in (x, wt, dy, b))


def _close(got, ref, dtype):
    assert_no_device_error()
    d = got.double() - ref.double()
    assert torch.isfinite(got.double()).all()
    assert d.norm() <= HALF_UNIT[dtype] * ref.double().norm()


def _off_boundary(t):
    """The same values two bytes off a 16-byte boundary."""
    r = torch.empty(t.numel() + 8, dtype=t.dtype, device=t.device)[1:1 + t.numel()]
    return r.copy_(t)


@pytest.mark.parametrize("dtype", ["f16", "bf16"])
@pytest.mark.parametrize("shape", SHAPES)
def test_passes_against_direct(shape, dtype):
    p, x, w, dy, b = _tensors(shape, dtype)
    for kw in ({}, {"bias": b, "activation": pd.ACT_RELU}):
        _close(pd.conv2d(pd.FORWARD, x, w, p, **kw), pd.conv2d(pd.FORWARD, x, w, p, algorithm=pd.ALGO_DIRECT, **kw), dtype)
    for which, a, f in ((pd.INPUT_BACKPROP, dy, w), (pd.FILTER_BACKPROP, x, dy)):
        ref = pd.conv2d(which, a, f, p, algorithm=pd.ALGO_DIRECT)
        _close(pd.conv2d(which, a, f, p), ref, dtype)
        _, elems = pd.conv2d_workspace_size(which, pd.F16 if dtype == "f16" else pd.BF16, p, pd.ALGO_IM2COL)
        ws = torch.full((elems + 1,), float("nan"), dtype=x.dtype, device="cuda")[1:]  # (its contents must not matter)
        _close(pd.conv2d(which, a, f, p, workspace=ws), ref, dtype)


@pytest.mark.parametrize("shape", [(2, 23, 31, 13, 150, 3, 1), (2, 20, 20, 64, 64, 3, 1)])
def test_filter_layout_and_boundaries(shape):
    p, x, w, dy, b = _tensors(shape, "f16")
    x, w, dy, b = (_off_boundary(t) for t in (x, w, dy, b))
    for which, a, f, kw in ((pd.FORWARD, x, w, {"bias": b}), (pd.INPUT_BACKPROP, dy, w, {}), (pd.FILTER_BACKPROP, x, dy, {})):
        ref = pd.conv2d(which, a, f, p, algorithm=pd.ALGO_DIRECT, **kw)
        out = _off_boundary(torch.zeros_like(ref))
        _close(pd.conv2d(which, a, f, p, out=out, **kw), ref, "f16")
    p, x, w, dy, b = _tensors(shape, "f16", fhwc=True)
    for which, a, f in ((pd.FORWARD, x, w), (pd.INPUT_BACKPROP, dy, w)):
        _close(pd.conv2d(which, a, f, p), pd.conv2d(which, a, f, p, algorithm=pd.ALGO_DIRECT), "f16")


@pytest.mark.parametrize("channels,features", [(13, 150), (16, 150), (13, 152)])
def test_fused_backprop_forms(channels, features):
    p, x, w, dy, _ = _tensors((2, 23, 31, channels, features, 3, 1), "f16")
    before = to_dev(np.random.default_rng(0).standard_normal(x.numel()).astype(np.float32), "f16")
    got, ref = before.clone(), before.clone()
    kw = {"accumulate": 1, "relu_forward_output": x}
    pd.conv2d(pd.INPUT_BACKPROP, dy, w, p, out=got, **kw)
    pd.conv2d(pd.INPUT_BACKPROP, dy, w, p, algorithm=pd.ALGO_DIRECT, out=ref, **kw)
    # (the sum with the earlier contents is rounded once more)
    assert (got.double() - ref.double()).norm() <= 2 * HALF_UNIT["f16"] * ref.double().norm()
    dw = torch.ones(w.numel(), dtype=torch.float32, device="cuda")
    pd.conv2d(pd.FILTER_BACKPROP, x, dy, p, out=dw, output_f32=True, accumulate=1)
    plain = pd.conv2d(pd.FILTER_BACKPROP, x, dy, p, algorithm=pd.ALGO_DIRECT)
    _close(dw - 1.0, plain, "f16")


@pytest.mark.parametrize("dtype", ["f16", "bf16"])
@pytest.mark.parametrize("size,c,k,win", [(7, 20, 30, 3), (14, 20, 30, 3), (28, 20, 30, 3), (28, 12, 20, 1), (9, 100, 150, 1)])
def test_an_image_alone_and_in_a_batch(size, c, k, win, dtype):
    """Whichever kernel a ragged layer runs on, it is the same one for every batch: an image's result has the same
    bits whatever is beside it."""
    g = torch.Generator(device="cuda").manual_seed(size * c)
    dt = torch.float16 if dtype == "f16" else torch.bfloat16
    x, w, b = (torch.randn(n, device="cuda", generator=g).to(dt) for n in (64 * size * size * c, win * win * c * k, k))
    x = x.view(64, -1)

    def call(images):
        p = pd.conv_params(len(images), size, size, c, k, win, 1)
        return pd.conv2d(pd.FORWARD, images.reshape(-1), w, p, bias=b, activation=pd.ACT_RELU).view(len(images), -1)

    together = call(x)
    for first, many in ((0, 1), (5, 1), (8, 2), (30, 9)):
        assert torch.equal(together[first:first + many], call(x[first:first + many]))
    assert_no_device_error()
