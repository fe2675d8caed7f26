"""Pooling forms with kernels of their own - max-pool gradients of windows that do not overlap - at the sizes
where they can go wrong: windows cut by the edge, rows and columns that no window covers, ties, NaN."""
import numpy as np
import pytest
import torch

import portdnn_b200 as pd
from gpu_util import to_dev, to_host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["f32", "f16"])
@pytest.mark.parametrize("with_nan", [False, True])
@pytest.mark.parametrize("rows,cols,window,same", [(8, 6, 2, False), (7, 9, 2, False), (7, 9, 2, True), (11, 5, 3, False),
                                                   (10, 8, 3, True), (5, 5, 5, False), (3, 2, 2, False)])
def test_max_grad_of_disjoint_windows(rows, cols, window, same, with_nan, dtype):
    n, c = 2, 8
    rng = np.random.default_rng(rows * cols)
    p = pd.pool_params(n, rows, cols, c, window, window, same)
    if p.pad_rows or p.pad_cols:
        pytest.skip("padded on the low side: windows of the general path")
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
