"""Batch normalisation in training, fp32: what the statistics and gradients of many rows lose against float64, however
long the run of rows is that a thread adds up."""
import pytest
import torch

import portdnn_b200 as pd

pytestmark = pytest.mark.gpu


def _off(got, ref):
    return ((got.double() - ref).norm() / ref.norm()).item()


# Largest relative errors of mean and gradient of gamma with threads of half as many rows that subtract the mean of their
# first four, as measured with these inputs (5.7e-7, 6.0e-7 and 1.8e-7, 2.3e-7); a deviation that is subtracted wrongly or a
# longer chain of additions shows as twice that.
@pytest.mark.parametrize("n,h,c,gamma,mean", [(128, 56, 64, 5.7e-7, 1.8e-7), (100, 56, 256, 6.1e-7, 2.3e-7)])
@pytest.mark.parametrize("shift", [0.0, 30.0])
def test_many_rows(n, h, c, gamma, mean, shift):
    g = torch.Generator(device="cuda").manual_seed(1)
    p, rows = pd.batchnorm_params(n, h, h, c, True), n * h * h
    x = torch.randn(rows, c, device="cuda", generator=g) + shift
    dy = torch.randn(rows, c, device="cuda", generator=g) + 0.1
    one, zero = torch.ones(c, device="cuda"), torch.zeros(c, device="cuda")
    _, m, v = pd.batchnorm_forward(x.view(-1), zero, one, zero, one, p)
    dx, dbeta, dgamma = pd.batchnorm_gradient(x.view(-1), dy.view(-1), one, p)
    xd, d = x.double(), dy.double()
    mu, var = xd.mean(0), xd.var(0, unbiased=False)
    normed = (xd - mu) / (var + p.epsilon).sqrt()
    assert _off(m, (1 - p.momentum) * mu) <= mean
    assert _off(v, p.momentum + (1 - p.momentum) * var) <= 2.0 ** -24
    dg, db = (d * normed).sum(0), d.sum(0)
    assert _off(dgamma, dg) <= gamma
    assert _off(dbeta, db) <= 2.0 ** -23
    assert _off(dx.view(rows, c), (d - db / rows - normed * (dg / rows)) / (var + p.epsilon).sqrt()) <= 2.0 ** -23


@pytest.mark.parametrize("value", [float("inf"), -float("inf"), float("nan")])
def test_one_value_that_is_not_finite(value):
    """It stays in its channel: the others are those without it, bit for bit."""
    n, h, c = 40, 40, 64
    g = torch.Generator(device="cuda").manual_seed(2)
    p, rows = pd.batchnorm_params(n, h, h, c, True), n * h * h
    x, dy = torch.randn(rows, c, device="cuda", generator=g), torch.randn(rows, c, device="cuda", generator=g)
    one, zero = torch.ones(c, device="cuda"), torch.zeros(c, device="cuda")

    def run():
        y, m, v = pd.batchnorm_forward(x.view(-1), zero, one, zero, one, p)
        dx, dbeta, dgamma = pd.batchnorm_gradient(x.view(-1), dy.view(-1), one, p)
        return [t.view(-1, c) for t in (y, m, v, dx, dbeta, dgamma)]

    clean = run()
    for row, channel in ((0, 3), (77, 10), (rows - 1, 63)):
        x[row, channel] = value
    hit = [3, 10, 63]
    rest = [i for i in range(c) if i not in hit]
    got = run()
    for a, b in zip(got, clean):
        assert torch.equal(a[:, rest], b[:, rest])
    assert not got[1][:, hit].isfinite().any() and got[2][:, hit].isnan().all() and got[5][:, hit].isnan().all()
    if value == value:
        assert (got[1][:, hit] == value).all()
