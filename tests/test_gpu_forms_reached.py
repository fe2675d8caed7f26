"""The shapes of other tests beside the form of kernel that they run in, read from the kernel nodes of a captured graph, and shapes for
the forms that those do not reach."""
import pytest
import torch

import portdnn_b200 as pd
from gpu_util import TORCH_DTYPES, assert_no_device_error
from launched import launched
from test_gpu_simt_gemm import SHAPES as TILE_SHAPES
from test_gpu_simt_gemm import test_passes as passes_against_float64
from test_gpu_solo_gemm import SHAPES as SOLO_SHAPES

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _sms():
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the sizes are those of 148 SMs")


@pytest.mark.parametrize("shape", SOLO_SHAPES)
def test_small_ctas(shape):
    n, h, w, c, k, win = shape
    p = pd.conv_params(n, h, w, c, k, win, 1)
    x, f, b = (torch.ones(m, device="cuda", dtype=torch.half) for m in (n * h * w * c, win * win * c * k, k))
    kernel, = launched(lambda: pd.conv2d(pd.FORWARD, x, f, p, bias=b, activation=pd.ACT_RELU))
    assert (kernel.threads == 192 and kernel.shared_bytes < 114 * 1024) == (n != 38)


# 16-bit layers whose three passes run on fp32 tiles
MORE_SHAPES = [(4, 21, 19, 16, 180, 3, 4, "f16"), (5, 22, 17, 17, 181, 3, 4, "bf16")]
# the passes that run on tiles, the others being too small (a thread to an output) or copied
ON_TILES = ["", "fib", "fib", "fib", "b", "fib", "i", "fib", "", "", "f", "fib", "fib"]


@pytest.mark.parametrize("shape,passes", list(zip(TILE_SHAPES + MORE_SHAPES, ON_TILES, strict=True)))
def test_passes_on_fp32_tiles(shape, passes):
    n, h, w, c, k, win, st, dtype = shape
    p = pd.conv_params(n, h, w, c, k, win, st)
    for letter, which in (("f", pd.FORWARD), ("i", pd.INPUT_BACKPROP), ("b", pd.FILTER_BACKPROP)):
        n_in, n_fil, _ = pd.api.conv_sizes(which, p)
        a, b = (torch.ones(m, device="cuda", dtype=TORCH_DTYPES[dtype]) for m in (n_in, n_fil))
        names = [kernel.name for kernel in launched(lambda: pd.conv2d(which, a, b, p))]
        assert any("simt_gemm_kernel" in name for name in names) == (letter in passes), (letter, names)


@pytest.mark.parametrize("shape", MORE_SHAPES)
@pytest.mark.parametrize("fhwc", [False, True])
def test_16_bit_layers_on_fp32_tiles(shape, fhwc):
    passes_against_float64(shape, fhwc)


@pytest.mark.parametrize("h,w,c,st", [(57, 61, 24, 1), (29, 15, 136, 1), (14, 14, 576, 1), (7, 9, 960, 1), (13, 8, 264, 1), (15, 120, 40, 1),
                                      (56, 57, 144, 2), (30, 31, 88, 2), (9, 14, 520, 2), (7, 7, 8, 2)])
def test_depthwise_fp16_tiles_and_strips(h, w, c, st):
    """Tensors of more than 8 MB on tiles, those of 8 channels and single images on strips: the same results, bit for bit."""
    g = torch.Generator(device="cuda").manual_seed(h * c)
    n = (9 << 20) // (2 * h * w * c) + 2
    p, one = pd.depthwise_params(n, h, w, c, 1, 3, st), pd.depthwise_params(1, h, w, c, 1, 3, st)
    x = torch.randn(n, h * w * c, device="cuda", generator=g).half()
    dy = torch.randn(n, p.out_rows * p.out_cols * c, device="cuda", generator=g).half()
    wt = torch.randn(9 * c, device="cuda", generator=g).half()
    on_tiles = lambda images, q: "forward_tile_kernel" in launched(lambda: pd.depthwise_conv2d(pd.FORWARD, images, wt, q))[0].name  # noqa: E731
    assert on_tiles(x.reshape(-1), p) == (c > 8) and not on_tiles(x[0], one)
    y = pd.depthwise_conv2d(pd.FORWARD, x.reshape(-1), wt, p).view(n, -1)
    dx = pd.depthwise_conv2d(pd.INPUT_BACKPROP, dy.reshape(-1), wt, p).view(n, -1)
    for i in (0, 1, n // 2, n - 2, n - 1):
        assert torch.equal(y[i], pd.depthwise_conv2d(pd.FORWARD, x[i], wt, one))
        assert torch.equal(dx[i], pd.depthwise_conv2d(pd.INPUT_BACKPROP, dy[i], wt, one))
    assert_no_device_error()
