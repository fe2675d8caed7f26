"""Argument checks of the native front end that need no GPU: what a wrong call raises."""
import os

import pytest
import torch

import portdnn_b200 as pd
from portdnn_b200 import api, build

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


@pytest.mark.parametrize("call", [
    lambda: pd.conv2d("0", X, X, P),
    lambda: pd.conv2d(0.5, X, X, P),
    lambda: pd.conv2d(pd.FORWARD, X, X, P, algorithm="4"),
    lambda: pd.depthwise_conv2d(0.5, X, X, pd.depthwise_params(1, 8, 8, 8, 1, 3, 1)),
    lambda: pd.pooling("0", 0, X, pd.pool_params(1, 8, 8, 8, 2, 2)),
    lambda: pd.pooling(pd.POOL_MAX, 0.5, X, pd.pool_params(1, 8, 8, 8, 2, 2)),
    lambda: pd.pointwise("1", X),
    lambda: pd.pointwise_grad(1.5, X, X),
    lambda: pd.bias_add(X, X, "8"),
    lambda: pd.bias_add(X, X, 8.5),
    lambda: pd.softmax(X, 1.0, 8, 8, 8),
    lambda: pd.matmul(X, X, 1, 8.5, 8, 8),
])
def test_texts_and_fractions_are_no_integers(call):
    """Before anything else is looked at, an argument that has to be a whole number is one."""
    with pytest.raises(TypeError):
        call()


def test_the_extension_of_another_torch_is_not_loaded(monkeypatch):
    """It is compiled against torch's headers: under another torch it counts as not built, and says so."""
    built = api.front_path()
    assert os.path.exists(built)
    monkeypatch.setattr(torch, "__version__", "0.0.0")
    monkeypatch.setattr(api, "_F", None)
    assert api.front_path() != built and build.needs_build()
    with pytest.raises(ImportError, match="portdnn_b200.build"):
        pd.pointwise(pd.ACT_RELU, X)
