"""Softmax of few pixels: four warps to a pixel, up to one wave of blocks, beside the one-warp form with more pixels; packets that
fill the block and packets that do not; rows whose maximum lies anywhere, equal values, infinities."""
import pytest
import torch

import portdnn_b200 as pd
from gpu_util import TORCH_DTYPES

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["f16", "bf16", "f32"])
@pytest.mark.parametrize("rows", [1, 250, 148 * 16, 148 * 16 + 1])
@pytest.mark.parametrize("packets", [33, 64, 125, 127, 128])
def test_forward(rows, packets, dtype):
    dt, g = TORCH_DTYPES[dtype], torch.Generator(device="cuda").manual_seed(rows + packets)
    c = packets * 16 // dt.itemsize
    x = (torch.randn(rows, c, device="cuda", generator=g) * 5).to(dt)
    x[0] = 1.0
    if rows > 1:
        x[1, ::3] = -float("inf")
    y = pd.softmax(x.reshape(-1), rows, 1, 1, c).view(rows, c)
    ref = torch.softmax(x.double(), 1)
    # the exponentials and their sum in fp32 (a few units in the last place), one rounding of the result
    unit = {"f16": 2.0 ** -11, "bf16": 2.0 ** -8, "f32": 2.0 ** -20}[dtype]
    floor = {"f16": 2.0 ** -25, "bf16": 0.0, "f32": 0.0}[dtype]  # (half the smallest fp16)
    assert ((y.double() - ref).abs() <= ref * (unit + 2.0 ** -19) + floor + 1e-38).all()
