"""The fixed-order second stage of the split reductions (column_sums.cuh), through operators that end in it:
few rows of partial sums (one thread per column), row counts around the 32 lanes and the four loads each
lane has in flight, and column counts that leave the last block ragged."""
import numpy as np
import pytest
import torch

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


def _batch_statistics(x, dy):
    """Batch mean and variance, and the gradients, of fp32 rows x channels; the same in float64."""
    rows, channels = x.shape
    one, zero = np.ones(channels, np.float32), np.zeros(channels, np.float32)
    p = pd.batchnorm_params(1, 1, rows, channels, True, 1e-3, 0.0)
    _, mean, var = pd.batchnorm_forward(to_dev(x, "f32"), *(to_dev(t, "f32") for t in (zero, one, zero, one)), p)
    dx, dbeta, dgamma = pd.batchnorm_gradient(to_dev(x, "f32"), to_dev(dy, "f32"), to_dev(one, "f32"), p)
    got = [to_host(t).astype(np.float64) for t in (mean, var, dgamma, dbeta)] + [to_host(dx).astype(np.float64).reshape(x.shape)]
    with np.errstate(all="ignore"):
        x64, dy64 = x.astype(np.float64), dy.astype(np.float64)
        xc = x64 - x64.mean(0)
        v = (xc ** 2).mean(0)
        cov = ((dy64 - dy64.mean(0)) * xc).sum(0)
        dx64 = (dy64 - dy64.mean(0) - xc * cov / rows / (v + 1e-3)) / np.sqrt(v + 1e-3)
        return got, [x64.mean(0), v, cov / np.sqrt(v + 1e-3), dy64.sum(0), dx64]


@pytest.mark.parametrize("rows,channels", [(40, 8), (1000, 24), (6001, 136)])
@pytest.mark.parametrize("mean,deviation,dy_mean", [(1e3, 1.0, 0.0), (1e3, 1.0, 8.0), (2e19, 1e17, 1.0), (-3e19, 1e16, 0.0)])
def test_batchnorm_moments_ignore_the_mean(rows, channels, mean, deviation, dy_mean):
    """The variance and the sums with the gradient are as exact far from zero as near it, and finite where
    the square of the mean is not (a mean is known to 2^-24 of itself, which enters neither)."""
    rng = np.random.default_rng(rows)
    x = (mean + deviation * rng.standard_normal((rows, channels))).astype(np.float32)
    dy = (dy_mean + rng.standard_normal((rows, channels))).astype(np.float32)
    got, ref = _batch_statistics(x, dy)
    # a lane's sums of at most 4 + rows / 64 rows lose 2^-24 of themselves with each, and the terms are up to twice
    # the squared deviations (the subtracted value is not the mean); then three levels of merging
    u = 2.0 ** -24 * (2 * (4 + rows / 256) + 8)
    magnitude = np.abs((x - ref[0]) * (dy - dy.astype(np.float64).mean(0))).sum(0) / np.sqrt(ref[1] + 1e-3)
    assert np.all(np.abs(got[1] - ref[1]) <= u * ref[1])
    assert np.all(np.abs(got[2] - ref[2]) <= 2 * u * (magnitude + np.abs(ref[2])))
    assert np.all(np.isfinite(got[4]))


@pytest.mark.parametrize("rows", [64, 1000, 6001])
@pytest.mark.parametrize("at", [0, 3, 63])
def test_batchnorm_moments_of_one_row(rows, at):
    """A channel that is the same everywhere but in one row, which a lane may have subtracted from the others."""
    x = np.full((rows, 8), 5.0, np.float32)
    x[at] = 1000.0 + np.arange(8)
    dy = np.random.default_rng(at).standard_normal((rows, 8)).astype(np.float32)
    got, ref = _batch_statistics(x, dy)
    # the lane of that row adds up to 4 + rows / 256 terms that are together up to 1 + rows / 256 / 4 times their
    # squared deviations
    u = 2.0 ** -24 * (8 + rows / 64) * (1 + rows / 1024)
    assert np.all(np.abs(got[1] - ref[1]) <= u * ref[1])


@pytest.mark.parametrize("rows,channels", [(40, 8), (1000, 24)])
def test_batchnorm_infinities(rows, channels):
    """What an infinity or a NaN makes of the results: what the formulas make of it, in the channel it is in."""
    rng = np.random.default_rng(rows)
    x, dy = (rng.standard_normal((rows, channels)).astype(np.float32) for _ in range(2))
    inf, last = np.float32(np.inf), rows - 1
    x[last, 0] = 3.0
    x[2, 1] = -3.0
    dy[last, 0] = inf              # dgamma = inf * (3 - mean) / deviation
    dy[2, 1] = inf                 # the same with -3
    dy[1, 2], dy[last, 2] = inf, -inf  # dbeta = NaN
    x[5, 3] = inf                  # mean = inf, variance = NaN
    dy[7, 4] = np.nan
    x[0, 5], x[1, 5] = 3e38, -3e38  # the variance overflows
    got, ref = _batch_statistics(x, dy)
    mean, var, dgamma, dbeta, dx = got
    assert dgamma[0] == np.inf and dgamma[1] == -np.inf and dbeta[0] == dbeta[1] == np.inf
    assert np.isnan(dbeta[2])
    assert mean[3] == np.inf and np.isnan(var[3]) and np.isnan(dgamma[3]) and np.isfinite(dbeta[3])
    assert np.isfinite(mean[4]) and np.isfinite(var[4]) and np.isnan(dgamma[4]) and np.isnan(dbeta[4])
    assert np.isfinite(mean[5]) and var[5] == np.inf
    for t, r in zip(got[:4], ref):
        assert np.allclose(t[6:], r[6:], rtol=1e-4, atol=1e-4)
    assert np.all(np.isfinite(dx[:, 6:])) and not np.any(np.isfinite(dx[:, :2]))


def test_batchnorm_of_very_many_channels():
    """More channel tiles than a grid's second extent holds (65535 of 128 channels)."""
    rows, channels = 3, 65536 * 128 + 8
    g = torch.Generator(device="cuda").manual_seed(1)
    x, dy = (torch.randn(rows, channels, device="cuda", generator=g).half() for _ in range(2))
    one, zero = torch.ones(channels, device="cuda").half(), torch.zeros(channels, device="cuda").half()
    p = pd.batchnorm_params(1, 1, rows, channels, True, 1e-3, 0.0)
    _, mean, var = pd.batchnorm_forward(x.view(-1), zero, one, zero, one, p)
    _, dbeta, _ = pd.batchnorm_gradient(x.view(-1), dy.view(-1), one, p)
    v, m = torch.var_mean(x.float(), 0, correction=0)
    # one rounding of fp32 sums of three terms
    for got, ref in ((mean, m), (var, v), (dbeta, dy.float().sum(0))):
        assert ((got.float() - ref).abs() <= 2.0 ** -11 * 1.01 * ref.abs() + 2.0 ** -20).all()
