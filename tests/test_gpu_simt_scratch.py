"""Slices of a long filter gradient on the CUDA cores: reported by the query, in the caller's scratch where there is some, done
without where no memory is to be had."""
import pytest
import torch

import portdnn_b200 as pd
from portdnn_b200 import api
from test_gpu_scratch_limits import no_memory

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fhwc", [False, True])
@pytest.mark.parametrize("layer", [(64, 56, 56, 13, 15, 1), (16, 40, 41, 66, 97, 3)])
def test_scratch_of_a_long_filter_gradient(layer, fhwc):
    p = pd.conv_params(*layer, 1, filter_format=2 if fhwc else 0)
    n_in, n_fil, n_out = api.conv_sizes(pd.FILTER_BACKPROP, p)
    g = torch.Generator(device="cuda").manual_seed(n_in)
    x, dy = torch.randn(n_in, device="cuda", generator=g), torch.randn(n_fil, device="cuda", generator=g)
    required, elems = pd.conv2d_workspace_size(pd.FILTER_BACKPROP, pd.F32, p, pd.ALGO_IM2COL)
    assert required == 0 and elems > 0 and elems % n_out == 0
    ref = pd.conv2d(pd.FILTER_BACKPROP, x, dy, p)
    ws = torch.full((elems,), float("nan"), device="cuda")
    torch.cuda.synchronize()
    with no_memory():
        before = pd.launch_count()
        assert torch.equal(pd.conv2d(pd.FILTER_BACKPROP, x, dy, p, workspace=ws), ref)
        assert pd.launch_count() - before == 2  # tiles, and the sum of the slices
    assert ws.isfinite().all()
    # too little of it: eight chains of a slice of all pixels then, apart by their additions.  m additions of products of random
    # sign are off by 2^-24 / sqrt 3 of each of m sums that grow as a root: 2^-24 sqrt(m / 6) of the last one.
    chain = p.batch * p.out_rows * p.out_cols / 8
    short = torch.full((elems - 1,), float("nan"), device="cuda")
    few = (1 << 20) // 4 + 1  # (a small block may still be had from the pool)
    with no_memory():
        got = pd.conv2d(pd.FILTER_BACKPROP, x, dy, p, workspace=short)
    assert (got.double() - ref.double()).norm() <= 2.0 ** -24 * (chain / 6) ** 0.5 * ref.double().norm()
    assert elems < few or short.isnan().all()


def test_nothing_is_reported_where_no_slices_run():
    for args, which, dtype in (((2, 9, 11, 17, 33, 3, 1), pd.FILTER_BACKPROP, pd.F32), ((16, 40, 41, 66, 97, 3, 1), pd.FORWARD, pd.F32),
                               ((16, 40, 41, 66, 97, 3, 1), pd.INPUT_BACKPROP, pd.F32)):
        assert pd.conv2d_workspace_size(which, dtype, pd.conv_params(*args), pd.ALGO_IM2COL) == (0, 0)
    assert pd.conv2d_workspace_size(pd.FILTER_BACKPROP, pd.F32, pd.conv_params(16, 40, 41, 66, 97, 3, 1), pd.ALGO_DIRECT) == (0, 0)
