"""Padded copies to whole lines or sectors are up to a third larger than copies to multiples of 8, which layers fall back to: where
the wider copies have more elements than the kernels count, and where the scratch that is there holds only the smaller ones."""
import pytest
import torch

import portdnn_b200 as pd
from portdnn_b200 import api

MOST = 0xF0000000  # elements of a copy


def _up(n, unit):
    return (n + unit - 1) // unit * unit


@pytest.mark.gpu
def test_layers_whose_wider_copies_have_too_many_elements():
    """100 channels: copies to 128 have too many elements, to 104 not; a little more, and neither is to be had."""
    for images, padded in ((700, True), (MOST // (224 * 224 * 104) + 1, False)):
        p = pd.conv_params(images, 224, 224, 100, 64, 1, 1)
        assert images * 224 * 224 * 128 >= MOST
        for which in (pd.FORWARD, pd.INPUT_BACKPROP, pd.FILTER_BACKPROP):
            _, elems = pd.conv2d_workspace_size(which, pd.F16, p, pd.ALGO_IM2COL)
            assert (elems >= images * 224 * 224 * 104) == padded, (which, images, elems)


def _bytes_by_eights(which, p):
    """Scratch of copies to multiples of 8 of tensors of which both counts are off it: x, y, filter, bias, each on 256 bytes,
    and what the padded layer asks for itself."""
    c, k, taps = _up(p.channels, 8), _up(p.features, 8), p.window_rows * p.window_cols
    q = pd.conv_params(p.batch, p.in_rows, p.in_cols, c, k, p.window_rows, p.stride_rows)
    _, inner = pd.conv2d_workspace_size(which, pd.F16, q, pd.ALGO_IM2COL)
    x, y = p.batch * p.in_rows * p.in_cols * c, p.batch * p.out_rows * p.out_cols * k
    return sum(_up(n, 256) for n in (2 * x, 2 * y, (4 if which == pd.FILTER_BACKPROP else 2) * taps * c * k, 2 * k, 2 * inner)) + 256


@pytest.mark.gpu
@pytest.mark.parametrize("which", [pd.FORWARD, pd.INPUT_BACKPROP, pd.FILTER_BACKPROP])
def test_scratch_for_multiples_of_eight(which):
    """The caller's scratch, poisoned, and no memory beside it: the results are those of the wider copies but for the order in which
    a filter gradient's pixels are added up; with a little less the call has no scratch at all."""
    from test_gpu_scratch_limits import _near, _rand, no_memory
    p = pd.conv_params(9, 33, 35, 100, 150, 3, 1)
    n_in, n_fil, _ = api.conv_sizes(which, p)
    a, b = _rand(n_in), _rand(n_fil, 0.05)
    ref = pd.conv2d(which, a, b, p)
    size = _bytes_by_eights(which, p)
    _, elems = pd.conv2d_workspace_size(which, pd.F16, p, pd.ALGO_IM2COL)
    assert size < 2 * elems
    ws = torch.full((size // 2,), float("nan"), dtype=torch.half, device="cuda")
    launches = {}
    with no_memory():
        for name, scratch in (("eights", ws), ("less", ws[:-64]), ("none", None)):
            before = pd.launch_count()
            got = pd.conv2d(which, a, b, p, workspace=scratch)
            launches[name] = pd.launch_count() - before
            _near(got, ref)
    assert launches["eights"] > launches["less"] == launches["none"]  # copies, GEMM, cut; the general kernel alone
