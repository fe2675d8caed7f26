"""A pixel's softmax is the same, bit for bit, alone, beside few others and beside many."""
import pytest
import torch

import portdnn_b200 as pd
from gpu_util import TORCH_DTYPES

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
