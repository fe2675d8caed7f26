"""Pooling forms with kernels of their own - max-pool gradients of windows that do not overlap, and global
average pools - at the sizes where they can go wrong: windows cut by the edge, rows and columns that no window
covers, ties, NaN; fewer pixels than threads to a packet, a last tile of few packets."""
import numpy as np
import pytest
import torch

import portdnn_b200 as pd
from gpu_util import to_dev, to_host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["f32", "f16"])
@pytest.mark.parametrize("with_nan", [False, True])
@pytest.mark.parametrize("rows,cols,window,same", [(8, 6, 2, False), (7, 9, 2, False), (7, 9, 2, True), (11, 5, 3, False),
                                                   (11, 8, 3, True), (5, 5, 5, False), (3, 2, 2, False)])
def test_max_grad_of_disjoint_windows(rows, cols, window, same, with_nan, dtype):
    n, c = 2, 8
    rng = np.random.default_rng(rows * cols)
    p = pd.pool_params(n, rows, cols, c, window, window, same)
    assert p.pad_rows == p.pad_cols == 0  # (else: windows of the general path)
    x = rng.integers(-2, 3, (n, rows, cols, c)).astype(np.float32)  # many ties
    op = pd.POOL_MAX
    if with_nan:
        op = pd.POOL_MAX_WITH_NAN
        x[rng.random(x.shape) < 0.1] = np.nan
    dy = rng.integers(1, 9, (n, p.out_rows, p.out_cols, c)).astype(np.float32)
    y = pd.pooling(op, 0, to_dev(x.ravel(), dtype), p)
    dx = pd.pooling_max_grad(op, to_dev(x.ravel(), dtype), y, to_dev(dy.ravel(), dtype), p)
    ref, yv = np.zeros_like(x), to_host(y).reshape(dy.shape)
    for i in range(n):
        for r in range(p.out_rows):
            for s in range(p.out_cols):
                for k in range(c):
                    win = x[i, r * window:(r + 1) * window, s * window:(s + 1) * window, k]
                    top = yv[i, r, s, k]
                    hits = np.argwhere((win == top) | (np.isnan(win) & np.isnan(top)))
                    ref[i, r * window + hits[0][0], s * window + hits[0][1], k] = dy[i, r, s, k]
    assert np.array_equal(to_host(dx).reshape(ref.shape), ref)


@pytest.mark.parametrize("dtype", ["f32", "f16", "bf16"])
@pytest.mark.parametrize("n,rows,cols,c", [(1, 1, 1, 8), (2, 1, 5, 264), (3, 7, 7, 256), (1, 9, 8, 1288), (150, 2, 3, 2048)])
def test_global_average(n, rows, cols, c, dtype):
    rng = np.random.default_rng(c)
    p = pd.pool_params(n, rows, cols, c, 1, 1, False)
    p.window_rows, p.window_cols, p.out_rows, p.out_cols = rows, cols, 1, 1
    x = to_dev(rng.standard_normal((n, rows * cols, c)).astype(np.float32), dtype)
    dy = to_dev(rng.standard_normal((n, 1, c)).astype(np.float32), dtype)
    y, dx = pd.pooling(pd.POOL_AVERAGE, 0, x.reshape(-1), p), pd.pooling(pd.POOL_AVERAGE, 1, dy.reshape(-1), p)
    unit = {"f32": 2.0 ** -24, "f16": 2.0 ** -11, "bf16": 2.0 ** -8}[dtype]
    # one rounding to the type, and fp32 sums of at most 72 terms and one division
    ref = x.double().mean(1)
    bound = unit * (ref.abs() + 2.0 ** -13) * 1.01 + 73 * 2.0 ** -24 * x.double().abs().mean(1)
    assert ((y.view(n, c).double() - ref).abs() <= bound).all()
    share = (dy.float() / torch.full_like(dy, rows * cols, dtype=torch.float32)).to(dy.dtype)
    assert torch.equal(dx.view(n, rows * cols, c), share.expand(n, rows * cols, c))


def test_global_average_of_more_than_four_billion_elements():
    """8.6 GB on the image side: offsets beyond 32 bits in both directions."""
    n, rows, cols, c = 21000, 10, 10, 2048
    p = pd.pool_params(n, rows, cols, c, 1, 1, False)
    p.window_rows, p.window_cols, p.out_rows, p.out_cols = rows, cols, 1, 1
    dy = torch.randn(n, c, device="cuda", generator=torch.Generator(device="cuda").manual_seed(0)).half()
    dx = pd.pooling(pd.POOL_AVERAGE, 1, dy.reshape(-1), p).view(n, rows * cols, c)
    share = (dy.float() / torch.full_like(dy, 100.0, dtype=torch.float32)).half()
    for i in (0, 1, 10485, 10486, 20971, 20972, n - 1):  # about the images at 2^31 and 2^32 elements
        assert torch.equal(dx[i], share[i].expand(rows * cols, c))
    y = pd.pooling(pd.POOL_AVERAGE, 0, dx.reshape(-1), p).view(n, c)
    # a hundred equal values: exact products of the sum up to 100 fp32 roundings, one division and one rounding
    assert ((y.float() - share.float()).abs() <= 2.0 ** -11 * 1.1 * share.float().abs() + 2.0 ** -25).all()
