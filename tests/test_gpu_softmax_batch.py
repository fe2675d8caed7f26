"""A pixel's softmax is the same, bit for bit, alone, beside few others and beside many."""
import pytest
import torch

import portdnn_b200 as pd
from gpu_util import TORCH_DTYPES
from launched import launched

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["f16", "bf16", "f32"])
@pytest.mark.parametrize("packets", [33, 64, 65, 97, 125, 128])
def test_alone_and_beside_others(packets, dtype):
    dt, g = TORCH_DTYPES[dtype], torch.Generator(device="cuda").manual_seed(packets)
    c, rows = packets * 16 // dt.itemsize, 148 * 16 + 2
    x = (torch.randn(rows, c, device="cuda", generator=g) * 3).to(dt)
    many = pd.softmax(x.reshape(-1), rows, 1, 1, c).view(rows, c)
    few = pd.softmax(x[:500].reshape(-1), 500, 1, 1, c).view(500, c)
    assert torch.equal(few, many[:500])
    assert torch.equal(pd.softmax(x[7].contiguous(), 1, 1, 1, c), many[7])


@pytest.mark.parametrize("dtype,channels,rows,by_rows", [
    ("f16", 1000, 148 * 16, True), ("f16", 1000, 148 * 16 + 1, False), ("f16", 512, 148 * 6, True), ("f16", 512, 148 * 6 + 1, False),
    ("f32", 500, 148 * 6, True), ("f32", 500, 148 * 6 + 1, False), ("f32", 128, 8, False)])
def test_where_four_warps_take_a_pixel(dtype, channels, rows, by_rows):
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the numbers of pixels are those of 148 SMs")
    x = torch.randn(rows * channels, device="cuda").to(TORCH_DTYPES[dtype])
    kernels = launched(lambda: pd.softmax(x, rows, 1, 1, channels))
    assert len(kernels) == 1 and ("softmax_forward_row_kernel" in kernels[0].name) == by_rows
