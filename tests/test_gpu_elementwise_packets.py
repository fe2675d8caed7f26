"""Elementwise operators that have kernels of their own (ReLU, ReLU6, the ReLU gradient, sums of tensors of one shape) against the
general forms, at remainders of the packets in flight, with NaN, infinities and zeros of both signs."""
import pytest
import torch

import portdnn_b200 as pd
from gpu_util import TORCH_DTYPES

pytestmark = pytest.mark.gpu

PACKETS = 148 * 16 * 256  # of one pass of the grid
SIZES = [8, 64, 8 * 255, 8 * (PACKETS - 1), 8 * (PACKETS + 3), 8 * (4 * PACKETS + 1), 8 * (2 * PACKETS) - 8, 13]


def _values(n, dtype, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    t = torch.randn(n, device="cuda", generator=g) * 4
    for i, v in enumerate((float("nan"), float("inf"), -float("inf"), 0.0, -0.0, 6.0, 5.9999, 6.0001)):
        t[i % n::101] = v
    return t.to(TORCH_DTYPES[dtype])


def _same(a, b):
    assert torch.equal(a.isnan(), b.isnan()) and torch.equal(a.nan_to_num(nan=0.0), b.nan_to_num(nan=0.0))


@pytest.mark.parametrize("dtype", ["f16", "bf16", "f32"])
@pytest.mark.parametrize("n", SIZES)
def test_against_definitions(n, dtype):
    x, y = _values(n, dtype, 1), _values(n, dtype, 2)
    zero = torch.zeros_like(x)
    # fmaxf(NaN, 0) is 0
    _same(pd.pointwise(pd.ACT_RELU, x), torch.where(x > 0, x, zero))
    _same(pd.pointwise(pd.ACT_RELU6, x), torch.where(x > 0, x, zero).clamp(max=6))
    _same(pd.pointwise_grad(pd.ACT_RELU, x, y), torch.where(x > 0, y, zero))
    _same(pd.pointwise_grad(pd.ACT_RELU6, x, y), torch.where((x > 0) & (x < 6), y, zero))
    for op, f in ((pd.BINARY_ADD, torch.add), (pd.BINARY_SUB, torch.sub), (pd.BINARY_MUL, torch.mul)):
        _same(pd.binaryop(op, x, [n], y, [n]), f(x.float(), y.float()).to(x.dtype))
    if n % 4 == 0:  # several extents of one shape, and in place
        out = x.clone()
        pd.binaryop(pd.BINARY_ADD, out, [n // 4, 4], y, [n // 4, 4], out=out)
        _same(out, (x.float() + y.float()).to(x.dtype))
