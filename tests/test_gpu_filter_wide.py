"""Filter gradients of 129 to 192 features: one column tile of 192, its last columns not there (and, with few steps,
two of 128)."""
import numpy as np
import pytest

import portdnn_b200 as pd
from conftest import rel_err
from gpu_util import TOL, assert_no_device_error, rounded, to_dev, to_host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["f16", "bf16"])
@pytest.mark.parametrize("shape", [(16, 45, 47, 40, 136, 3, 1), (40, 65, 63, 72, 192, 1, 1), (30, 41, 40, 136, 184, 3, 2), (6, 33, 35, 64, 152, 5, 1),
                                   (2, 13, 11, 40, 136, 3, 1)])
@pytest.mark.parametrize("output_f32", [False, True])
def test_filter_gradient(orc, dtype, shape, output_f32):
    n, h, w, c, k, win, st = shape
    rng = np.random.default_rng(6)
    p, po = pd.conv_params(n, h, w, c, k, win, st), orc.conv_params(n, h, w, c, k, win, st)
    x = rounded(rng.uniform(-1, 1, n * h * w * c).astype(np.float32), dtype)
    dy = rounded(rng.standard_normal(n * p.out_rows * p.out_cols * k).astype(np.float32), dtype)
    ref = orc.conv2d(orc.FILTER_BACKPROP, x, dy, po)
    dw = pd.conv2d(pd.FILTER_BACKPROP, to_dev(x, dtype), to_dev(dy, dtype), p, output_f32=output_f32)
    assert rel_err(to_host(dw), ref) <= TOL[dtype]
    if output_f32:  # every pixel split adds its tiles
        pd.conv2d(pd.FILTER_BACKPROP, to_dev(x, dtype), to_dev(dy, dtype), p, out=dw, output_f32=True, accumulate=True)
        assert rel_err(to_host(dw), 2 * ref) <= TOL[dtype]
    assert_no_device_error()
