"""Argument checks of the native front end that need no GPU: what a wrong call raises."""
import pytest
import torch

import portdnn_b200 as pd

P = pd.conv_params(1, 8, 8, 8, 8, 3, 1)
X = torch.zeros(512)


@pytest.mark.parametrize("call, error", [
    (lambda: pd.conv2d(pd.FORWARD, X, X, P), ValueError),                              # not on a GPU
    (lambda: pd.conv2d(pd.FORWARD, "x", X, P), TypeError),                             # not a tensor
    (lambda: pd.conv2d(pd.FORWARD, X, X, pd.pool_params(1, 8, 8, 8, 2, 2)), TypeError),  # another operator's parameters
    (lambda: pd.depthwise_conv2d(pd.FORWARD, X, X, pd.depthwise_params(1, 8, 8, 8, 1, 3, 1)), ValueError),
    (lambda: pd.pooling(pd.POOL_MAX, 0, X, pd.pool_params(1, 8, 8, 8, 2, 2)), ValueError),
    (lambda: pd.pointwise(pd.ACT_RELU, X), ValueError),
    (lambda: pd.matmul(X, X, 1, 8, 8, 8), ValueError),
    (lambda: pd.binaryop(pd.BINARY_ADD, X, [512], X, [512]), ValueError),
    (lambda: pd.softmax(X, 1, 8, 8, 8), ValueError),
])
def test_wrong_calls_raise(call, error):
    with pytest.raises(error):
        call()
