"""Which kernel or grid a call takes on either side of a rule's line, read from the kernel nodes of a captured graph.  The lines
themselves were measured; the figures stand beside the rules."""
import pytest
import torch

import portdnn_b200 as pd
from gpu_util import TORCH_DTYPES
from launched import launched

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _sms():
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the sizes are those of 148 SMs")


def _rand(n, dtype):
    return torch.randn(n, device="cuda").to(TORCH_DTYPES[dtype])


@pytest.mark.parametrize("n,h,w,c,dtype", [(24, 45, 62, 96, "f16"), (10, 17, 24, 688, "f16"), (39, 31, 28, 64, "f32"), (30, 60, 59, 40, "bf16")])
def test_short_walks_stay_within_one_wave(n, h, w, c, dtype):
    """Stride-2 gradients, depthwise and of 3x3 pools: threads by the length of their walks, 512 to an SM at most where the
    walks are shorter than four rows."""
    p = pd.depthwise_params(n, h, w, c, 1, 3, 2)
    dy, f = _rand(n * p.out_rows * p.out_cols * c, dtype), _rand(9 * c, dtype)
    kernels = launched(lambda: pd.depthwise_conv2d(pd.INPUT_BACKPROP, dy, f, p))
    assert len(kernels) == 1 and "depthwise_ibp_s2_kernel" in kernels[0].name
    assert 148 * 256 < kernels[0].blocks * kernels[0].threads <= 148 * 512 + 256
    q = pd.pool_params(n, h, w, c, 3, 2, True)
    x = _rand(n * h * w * c, dtype)
    y = pd.pooling(pd.POOL_MAX, 0, x, q)
    kernels = [k for k in launched(lambda: pd.pooling_max_grad(pd.POOL_MAX, x, y, dy, q)) if "pool_max_grad_s2" in k.name]
    assert len(kernels) == 1 and 148 * 256 < kernels[0].blocks * kernels[0].threads <= 148 * 512 + 256


@pytest.mark.parametrize("n,h,c,dtype,most", [(64, 28, 2048, "f16", 444), (64, 28, 904, "f16", 444), (64, 28, 1664, "bf16", 444), (128, 14, 640, "f32", 444),
                                              (16, 56, 1024, "f32", 888)])
def test_statistics_take_whole_waves(n, h, c, dtype, most):
    """Three blocks to an SM, in one wave or, fp32 tensors well beyond the L2 cache, two; no block more."""
    p, size = pd.batchnorm_params(n, h, h, c, True), n * h * h * c
    x, dy, v = _rand(size, dtype), _rand(size, dtype), _rand(c, dtype).abs()
    for call, limit in ((lambda: pd.batchnorm_forward(x, v, v, v, v, p), most), (lambda: pd.batchnorm_gradient(x, dy, v, p), 444)):
        kernels = [k for k in launched(call) if "batchnorm_moments_kernel" in k.name]
        assert len(kernels) == 1 and limit * 3 // 4 < kernels[0].blocks <= limit


@pytest.mark.parametrize("c", [904, 936, 1000, 1016, 888])
def test_threads_of_a_gradient_keep_their_channels(c):
    """16-bit training gradients: the threads are a multiple of the packets of a pixel, also where a wave has no room for more
    than four of their units."""
    n, h = 118, 8
    p, size = pd.batchnorm_params(n, h, h, c, True), n * h * h * c
    x, dy, g = _rand(size, "bf16"), _rand(size, "bf16"), _rand(c, "bf16")
    kernels = [k for k in launched(lambda: pd.batchnorm_gradient(x, dy, g, p)) if "grad_training_vec" in k.name]
    assert len(kernels) == 1 and kernels[0].blocks * kernels[0].threads % (c // 8) == 0


# n, h, c, k, window, pass; one tile to a CTA or persistent CTAs of two pipelines
@pytest.mark.parametrize("layer,which,solo", [
    ((24, 14, 256, 256, 3), pd.FORWARD, True),          # 168 tiles of 36 steps, the filter in whole lines
    ((24, 14, 256, 200, 3), pd.FORWARD, False),         # rows of 400 bytes
    ((24, 14, 264, 256, 3), pd.INPUT_BACKPROP, True),
    ((24, 14, 256, 264, 3), pd.INPUT_BACKPROP, False),
    ((24, 14, 256, 128, 1), pd.FORWARD, True),          # at most one tile to an SM
    ((36, 28, 64, 64, 1), pd.FORWARD, True),            # 221 tiles, the filter in whole lines
    ((36, 28, 64, 72, 1), pd.FORWARD, True),            # one step: whatever the filter's rows are
    ((36, 28, 512, 24, 1), pd.FORWARD, False),          # eight steps, rows of 48 bytes
    ((60, 24, 32, 16, 3), pd.FORWARD, False),
    ((10, 54, 1024, 64, 1), pd.FORWARD, True),          # 228 tiles: beyond 1.42 to an SM
])
def test_small_ctas(layer, which, solo):
    p = pd.conv_params(layer[0], layer[1], layer[1], *layer[2:], 1)
    n_in, n_fil, _ = pd.api.conv_sizes(which, p)
    x, f = _rand(n_in, "bf16"), _rand(n_fil, "bf16")
    kernels = [k for k in launched(lambda: pd.conv2d(which, x, f, p)) if "umma_gemm_kernel" in k.name]
    assert len(kernels) == 1
    # the persistent form has two pipelines, 384 threads, and one CTA to an SM
    assert (kernels[0].threads == 192 and kernels[0].shared_bytes < 114 * 1024) == solo
    assert solo or kernels[0].blocks <= 148


@pytest.mark.parametrize("layer,which,dtype,kernel", [
    ((24, 28, 2, 2, 7), pd.FORWARD, "f32", "simt_gemm_kernel"),             # sums of 98 terms
    ((24, 28, 5, 2, 3), pd.FORWARD, "f32", "direct_forward_kernel"),        # two columns, 45 terms
    ((24, 28, 5, 6, 3), pd.FORWARD, "f32", "direct_forward_kernel"),        # 45 terms, 212 thousand multiply-adds an image
    ((24, 60, 5, 6, 3), pd.FORWARD, "f32", "simt_gemm_kernel"),             # a million
    ((1, 30, 9, 89, 1), pd.INPUT_BACKPROP, "f32", "direct_input_backprop_kernel"),
    ((1, 30, 9, 91, 1), pd.INPUT_BACKPROP, "f32", "simt_gemm_kernel"),
    ((5, 4, 270, 14, 2), pd.INPUT_BACKPROP, "f16", "direct_input_backprop_kernel"),
    ((5, 4, 270, 18, 2), pd.INPUT_BACKPROP, "f16", "umma_gemm"),            # copies
    ((1, 7, 13, 20, 1), pd.FILTER_BACKPROP, "f16", "direct_filter_backprop_kernel"),
    ((2, 7, 13, 20, 1), pd.FILTER_BACKPROP, "f16", "umma_gemm"),
])
def test_odd_layers(layer, which, dtype, kernel):
    p = pd.conv_params(layer[0], layer[1], layer[1], *layer[2:], 1)
    n_in, n_fil, _ = pd.api.conv_sizes(which, p)
    x, f = _rand(n_in, dtype), _rand(n_fil, dtype)
    assert any(kernel in k.name for k in launched(lambda: pd.conv2d(which, x, f, p)))


# products that a thread to an output had been faster at than the tiles that took them, and one that tiles are faster at
@pytest.mark.parametrize("m,k,n,dtype,tiles", [(844, 101, 38, "bf16", False), (267, 144, 13, "f32", False), (74, 110, 1028, "f16", False), (1000, 2000, 501, "f16", True)])
def test_odd_products(m, k, n, dtype, tiles):
    a, b = _rand(m * k, dtype), _rand(k * n, dtype)
    kernels = launched(lambda: pd.matmul(a, b, 1, m, k, n))
    assert len(kernels) == 1 and ("simt_gemm_kernel" in kernels[0].name) == tiles


@pytest.mark.parametrize("n,h,c,stride,tiles", [(16, 28, 96, 1, False), (48, 28, 96, 1, True), (24, 56, 32, 2, False), (64, 56, 32, 2, True), (64, 112, 8, 1, False),
                                                (64, 112, 16, 1, True)])
def test_depthwise_half(n, h, c, stride, tiles):
    p = pd.depthwise_params(n, h, h, c, 1, 3, stride)
    x, f = _rand(n * h * h * c, "f16"), _rand(9 * c, "f16")
    kernels = launched(lambda: pd.depthwise_conv2d(pd.FORWARD, x, f, p))
    assert len(kernels) == 1 and ("depthwise_forward_tile_kernel" in kernels[0].name) == tiles


@pytest.mark.parametrize("n,h,window,narrow", [(2, 38, 3, False), (24, 64, 3, True), (24, 64, 7, True), (24, 64, 5, False), (40, 112, 5, True)])
def test_stem_filter_gradients(n, h, window, narrow):
    p = pd.conv_params(n, h, h, 3, 64, window, 2)
    x, dy = _rand(n * h * h * 3, "f16"), _rand(n * p.out_rows * p.out_cols * 64, "f16")
    kernels = launched(lambda: pd.conv2d(pd.FILTER_BACKPROP, x, dy, p))
    assert any("pack_small_c_input_narrow" in k.name for k in kernels) == narrow


@pytest.mark.parametrize("c,k,window,wide", [(100, 150, 3, (128, 192)), (100, 150, 1, (112, 160)), (59, 121, 1, (64, 128)), (50, 49, 3, (64, 64)), (50, 49, 1, (64, 64)),
                                             (49, 130, 3, (64, 144)), (57, 114, 1, (64, 128))])
def test_widths_of_padded_copies(c, k, window, wide):
    """Whole lines of 64 where they are at most 1.3 times as much, 1.1 for windows of one pixel; else whole sectors of 16."""
    p, q = pd.conv_params(4, 30, 30, c, k, window, 1), pd.conv_params(4, 30, 30, *wide, window, 1)
    _, elems = pd.conv2d_workspace_size(pd.FORWARD, pd.F16, p, pd.ALGO_IM2COL)
    _, inner = pd.conv2d_workspace_size(pd.FORWARD, pd.F16, q, pd.ALGO_IM2COL)
    sizes = (2 * 3600 * q.channels, 2 * 3600 * q.features, 2 * window * window * q.channels * q.features, 2 * q.features, 2 * inner)
    assert 2 * elems == sum(-(-n // 256) * 256 for n in sizes) + 256
