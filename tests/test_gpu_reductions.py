"""The fixed-order second stage of the split reductions (column_sums.cuh), through operators that end in it:
few rows of partial sums (one thread per column), row counts around the 32 lanes and the four loads each
lane has in flight, and column counts that leave the last block ragged."""
import numpy as np
import pytest

import portdnn_b200 as pd
from gpu_util import to_dev, to_host

pytestmark = pytest.mark.gpu

# A sum of n fp32 terms in lanes of at most n / 256 and trees of at most 10 levels, against float64.  The
# terms are of order 1 and of both signs, so errors are measured against the sum of their magnitudes.
BOUND = 2.0 ** -23


@pytest.mark.parametrize("rows,channels", [(64, 1), (64 * 8, 33), (64 * 9 + 1, 31), (64 * 33 - 5, 40), (64 * 130, 12), (64 * 700 + 3, 64)])
def test_batchnorm_sums(rows, channels):
    rng = np.random.default_rng(rows)
    x = rng.standard_normal((rows, channels)).astype(np.float32)
    dy = rng.standard_normal((rows, channels)).astype(np.float32)
    one, zero = np.ones(channels, np.float32), np.zeros(channels, np.float32)
    p = pd.batchnorm_params(1, 1, rows, channels, True, 1e-3, 0.0)
    _, mean, var = pd.batchnorm_forward(to_dev(x, "f32"), *(to_dev(t, "f32") for t in (zero, one, zero, one)), p)
    _, dbeta, dgamma = pd.batchnorm_gradient(to_dev(x, "f32"), to_dev(dy, "f32"), to_dev(one, "f32"), p)
    x64, dy64 = x.astype(np.float64), dy.astype(np.float64)
    xc = x64 - x64.mean(0)
    steps = rows / 256 + 12
    assert np.all(np.abs(to_host(mean) - x64.mean(0)) <= BOUND * steps * np.abs(x64).mean(0))
    assert np.all(np.abs(to_host(var) - (xc ** 2).mean(0)) <= BOUND * (steps + 4) * (xc ** 2).mean(0))
    assert np.all(np.abs(to_host(dbeta) - dy64.sum(0)) <= BOUND * (steps + 2) * np.abs(dy64).sum(0))
    ref = (dy64 * xc).sum(0) / np.sqrt((xc ** 2).mean(0) + 1e-3)
    assert np.all(np.abs(to_host(dgamma) - ref) <= BOUND * (steps + 8) * np.abs(dy64 * xc).sum(0))


@pytest.mark.parametrize("batch,rows,channels", [(1, 5, 3), (2, 33, 40), (40, 28, 72)])
def test_depthwise_filter_gradient(batch, rows, channels):
    rng = np.random.default_rng(channels)
    p = pd.depthwise_params(batch, rows, rows, channels, 1, 3, 1)
    x = rng.standard_normal((batch, rows, rows, channels)).astype(np.float32)
    dy = rng.standard_normal((batch, rows, rows, channels)).astype(np.float32)
    dw = to_host(pd.depthwise_conv2d(pd.FILTER_BACKPROP, to_dev(x.ravel(), "f32"), to_dev(dy.ravel(), "f32"), p))
    xp = np.pad(x.astype(np.float64), ((0, 0), (1, 1), (1, 1), (0, 0)))
    for r in range(3):
        for c in range(3):
            terms = xp[:, r:r + rows, c:c + rows] * dy
            got = dw.reshape(3, 3, channels)[r, c]
            bound = BOUND * (batch * rows * rows / 256 + 30) * np.abs(terms).sum((0, 1, 2))
            assert np.all(np.abs(got - terms.sum((0, 1, 2))) <= bound)


@pytest.mark.parametrize("dtype", ["f32", "f16"])
@pytest.mark.parametrize("rows,channels", [(1, 8), (37, 128), (9, 256), (250, 1000), (3, 1032)])
def test_softmax_gradient(rows, channels, dtype):
    """Packets of a lane from one to the four it holds, and the widths before and behind them."""
    rng = np.random.default_rng(channels)
    y = np.exp(rng.standard_normal((rows, channels)))
    y = to_dev((y / y.sum(1, keepdims=True)).astype(np.float32), dtype)
    dy = to_dev(rng.standard_normal((rows, channels)).astype(np.float32), dtype)
    dx = pd.softmax(y.reshape(-1), rows, 1, 1, channels, gradient=dy.reshape(-1)).view(rows, channels).double()
    y64, dy64 = y.double(), dy.double()
    terms = y64 * dy64
    ref = (dy64 - terms.sum(1, keepdim=True)) * y64
    unit = 2.0 ** -24 if dtype == "f32" else 2.0 ** -11
    # one rounding to the type (smallest f16 numbers: 2^-25), fp32 sums of at most channels / 32 + 5 additions in a row
    slack = BOUND * (channels / 32 + 8) * (terms.abs().sum(1, keepdim=True) + dy64.abs()) * y64
    assert ((dx - ref).abs() <= unit * ref.abs() * 1.01 + slack + (2.0 ** -25 if dtype == "f16" else 0.0)).all()


@pytest.mark.parametrize("dtype", ["f32", "bf16"])
@pytest.mark.parametrize("rows,channels", [(1, 8), (31, 8), (64, 136), (97, 128), (5000, 264), (40000, 8)])
def test_batchnorm_moments_far_from_zero(rows, channels, dtype):
    """The one-pass moments where the mean is large against the deviations: fewer rows than row lanes, slices
    that end inside a batch, channel tiles with idle lanes."""
    rng = np.random.default_rng(rows)
    x = to_dev((32.0 + rng.standard_normal((rows, channels))).astype(np.float32), dtype)
    dy = to_dev((8.0 + rng.standard_normal((rows, channels))).astype(np.float32), dtype)
    one, zero = (to_dev(np.full(channels, v, np.float32), dtype) for v in (1.0, 0.0))
    p = pd.batchnorm_params(1, 1, rows, channels, True, 1e-3, 0.0)
    out, mean, var = (t.double().view(-1, channels) for t in pd.batchnorm_forward(x.reshape(-1), zero, one, zero, one, p))
    dx, dbeta, dgamma = (t.double().view(-1, channels) for t in pd.batchnorm_gradient(x.reshape(-1), dy.reshape(-1), one, p))
    x64, dy64 = x.double(), dy.double()
    m, xc = x64.mean(0), x64 - x64.mean(0)
    v, dc = (xc ** 2).mean(0), dy64 - dy64.mean(0)
    # one rounding to the type, and fp32 means with an error of a few units of 32 (or 8), which enters the sums
    # around them twice
    unit = 2.0 ** -24 if dtype == "f32" else 2.0 ** -8
    near = lambda got, ref, slack: bool(((got - ref).abs() <= 1.01 * unit * ref.abs() + slack).all())
    e = 2.0 ** -24 * (rows / 256 + 12)
    assert near(out, x64 / (1 + 1e-3) ** 0.5, 2.0 ** -20 * x64.abs())
    assert near(mean[0], m, 33 * e)
    assert near(var[0], v, 2 * 33 * e * xc.abs().mean(0) + 4 * e * v)
    assert near(dbeta[0], dy64.sum(0), 9 * e * rows)
    sd = (v + 1e-3).sqrt()
    cov = (xc * dc).sum(0)
    cov_slack = 33 * e * dc.abs().sum(0) + 9 * e * xc.abs().sum(0) + 4 * e * (xc * dc).abs().sum(0)
    assert near(dgamma[0], cov / sd, cov_slack / sd * 1.01 + 33 * e * (cov / sd).abs() / sd ** 2)
    ref = (dc - xc * (cov / rows / (v + 1e-3))) / sd
    share = cov.abs() / rows / (v + 1e-3)
    slack = (9 * e + 2.0 ** -20 * dy64.abs() + (33 * e + 2.0 ** -20 * x64.abs()) * share + xc.abs() * (cov_slack / rows + 66 * e * share) / (v + 1e-3)) / sd
    assert near(dx, ref, 2 * slack)
