"""Layers that use scratch of the library's own where there is memory, and have a kernel that needs none: they
run where no memory is to be had.  The device's stream-ordered allocations come from a small pool here, and what
it has is taken."""
import ctypes
from contextlib import contextmanager

import pytest
import torch

import portdnn_b200 as pd
from portdnn_b200 import api
from gpu_util import assert_no_device_error

pytestmark = pytest.mark.gpu


class _PoolProps(ctypes.Structure):
    """cudaMemPoolProps: pinned device memory without handles."""
    _fields_ = [("alloc_type", ctypes.c_int), ("handle_types", ctypes.c_int), ("location_type", ctypes.c_int),
                ("location_id", ctypes.c_int), ("security", ctypes.c_void_p), ("max_size", ctypes.c_size_t),
                ("usage", ctypes.c_ushort), ("reserved", ctypes.c_ubyte * 54)]


@contextmanager
def no_memory():
    """No stream-ordered allocation of a MiB or more succeeds inside."""
    rt, dev = ctypes.CDLL("libcudart.so.12"), torch.cuda.current_device()
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    before, pool, blocks = ctypes.c_void_p(), ctypes.c_void_p(), []
    props = _PoolProps(1, 0, 1, dev, None, 1 << 20, 0)
    torch.cuda.synchronize()
    assert rt.cudaDeviceGetMemPool(ctypes.byref(before), dev) == 0
    assert rt.cudaMemPoolCreate(ctypes.byref(pool), ctypes.byref(props)) == 0
    assert rt.cudaDeviceSetMemPool(dev, pool) == 0
    try:
        refused = False
        while not refused and len(blocks) < 256:  # (the limit is rounded up to the driver's own granularity)
            block = ctypes.c_void_p()
            refused = rt.cudaMallocAsync(ctypes.byref(block), ctypes.c_size_t(1 << 20), stream) != 0
            if not refused:
                blocks.append(block)
        rt.cudaGetLastError()
        if not refused:
            pytest.skip("this driver does not limit a pool")
        yield
        torch.cuda.synchronize()
    finally:
        for block in blocks:
            assert rt.cudaFreeAsync(block, stream) == 0
        torch.cuda.synchronize()
        assert rt.cudaDeviceSetMemPool(dev, before) == 0
        assert rt.cudaMemPoolDestroy(pool) == 0


def _rand(n, scale=1.0):
    return torch.randn(n, device="cuda", generator=torch.Generator(device="cuda").manual_seed(n)).mul_(scale).half()


def _near(got, ref):
    """Two fp32 sums of the same products, each rounded once to fp16: apart by a unit in the last place in few
    places, below half a unit in the 2-norm."""
    assert_no_device_error()
    assert (got.double() - ref.double()).norm() <= 2.0 ** -11 * ref.double().norm()


@pytest.mark.parametrize("which", [pd.FORWARD, pd.INPUT_BACKPROP, pd.FILTER_BACKPROP])
def test_padded_copies(which):
    p = pd.conv_params(8, 28, 28, 100, 150, 1, 1)  # copies of 1.3 and 1.9 MB
    n_in, n_fil, _ = api.conv_sizes(which, p)
    a, b = _rand(n_in), _rand(n_fil, 0.1)
    ref = pd.conv2d(which, a, b, p)
    with no_memory():
        got = pd.conv2d(which, a, b, p)
    _near(got, ref)


def test_packed_filter_of_a_grouped_layer():
    p = pd.conv_params(2, 14, 14, 64 * 64, 64 * 64, 3, 1, groups=64)  # 4.7 MB
    n_in, n_fil, _ = api.conv_sizes(pd.FORWARD, p)
    x, w = _rand(n_in), _rand(n_fil, 0.02)
    before = pd.launch_count()
    ref = pd.conv2d(pd.FORWARD, x, w, p)
    assert pd.launch_count() - before == 2  # packing, and all groups in one launch
    _, elems = pd.conv2d_workspace_size(pd.FORWARD, pd.F16, p, pd.ALGO_IM2COL)
    assert elems == n_fil
    ws = torch.full((elems,), float("nan"), dtype=torch.half, device="cuda")
    with no_memory():
        _near(pd.conv2d(pd.FORWARD, x, w, p), ref)
        assert torch.equal(pd.conv2d(pd.FORWARD, x, w, p, workspace=ws), ref)


def test_partial_sums_of_whole_filter_tiles():
    p = pd.conv_params(17, 8, 8, 768, 768, 3, 1)  # 21 MB
    n_in, n_fil, _ = api.conv_sizes(pd.FILTER_BACKPROP, p)
    x, dy = _rand(n_in), _rand(n_fil)
    ref = pd.conv2d(pd.FILTER_BACKPROP, x, dy, p)
    with no_memory():
        got = pd.conv2d(pd.FILTER_BACKPROP, x, dy, p)
    _near(got, ref)


@pytest.mark.parametrize("dtype,layer", [
    (torch.float32, (2, 16, 16, 64, 768, 5)),  # two taps to a tile: two pieces of 4.9 MB
    (torch.half, (8, 16, 16, 400, 192, 5)),    # one column tile of 192: two pieces of 7.7 MB
    (torch.half, (8, 56, 56, 64, 64, 3))])     # many pieces
@pytest.mark.parametrize("accumulate", [False, True])
def test_partial_sums_of_a_split_filter_gradient(dtype, layer, accumulate):
    """Without memory the reduction runs in one piece."""
    p = pd.conv_params(*layer, 1)
    n_in, n_fil, n_out = api.conv_sizes(pd.FILTER_BACKPROP, p)
    x, dy = _rand(n_in).to(dtype), _rand(n_fil, 0.02).to(dtype)
    _, elems = pd.conv2d_workspace_size(pd.FILTER_BACKPROP, pd.F32 if dtype == torch.float32 else pd.F16, p, pd.ALGO_IM2COL)
    assert elems > 0
    kw = {"accumulate": True, "output_f32": True} if accumulate else {}
    out = [torch.zeros(n_out, device="cuda", dtype=torch.float32 if accumulate else dtype) for _ in range(2)]
    pd.conv2d(pd.FILTER_BACKPROP, x, dy, p, out=out[0], **kw)
    with no_memory():
        pd.conv2d(pd.FILTER_BACKPROP, x, dy, p, out=out[1], **kw)
    _near(out[1], out[0])
