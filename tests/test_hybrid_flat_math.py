"""Division, roots, softplus, sigmoid and tanh without branches, one by one over the ranges they are stated for, against 64-bit values."""
from __future__ import annotations

import pytest
import torch

INF = float("inf")


def _points(lo, hi, signs=False):
    """Every power of two of the range with mantissas at random, at one and just below two, and its ends."""
    g = torch.Generator().manual_seed(7)
    e = torch.arange(-126, 128, dtype=torch.float64)
    m = torch.cat((torch.rand(8000, generator=g, dtype=torch.float64) + 1, torch.tensor([1.0, 1 + 2.0 ** -23, 2 - 2.0 ** -23], dtype=torch.float64)))
    x = (torch.exp2(e)[:, None] * m).float().flatten()
    x = torch.cat((x[(x >= lo) & (x <= hi)], torch.tensor([lo, hi])))
    return torch.cat((x, -x, torch.zeros(1))) if signs else x


def _evaluate(which, x, by=1.0):
    from mdi_llm_b200.ops import hybrid as H

    x = x.cuda()
    y = torch.empty_like(x)
    assert H.lib().hyb_flat_math(which, x.data_ptr(), by, y.data_ptr(), x.numel(), torch.cuda.current_stream().cuda_stream) == 0
    return y.double().cpu()


def _worst(got, want, least=-149):
    """Largest difference in units in the last place of the wanted value; values that fp32 does not have, and zeros, have to be met exactly."""
    fits = (want.abs() < 2.0 ** 128) & (want != 0)
    assert torch.equal(got[~fits], want[~fits].float().double())
    _, e = torch.frexp(want[fits])
    return ((got[fits] - want[fits]).abs() / torch.exp2(torch.clamp(e.double() - 24, min=least))).max().item()


@pytest.mark.gpu
def test_inverse():
    x = _points(1.0, 1e37)
    assert _worst(_evaluate(0, x), 1 / x.double()) <= 0.51
    x = _points(1e37, 2.0 ** 126)
    assert _worst(_evaluate(0, x), 1 / x.double()) <= 1
    assert (_evaluate(0, torch.tensor([1.1 * 2.0 ** 126, 3.4e38, INF])) == 0).all()


@pytest.mark.gpu
def test_inverse_root():
    x = _points(2.0 ** -126, 1e37)
    assert _worst(_evaluate(1, x), x.double().rsqrt()) <= 1
    x = torch.cat((_points(1e37, 3.4e38), torch.tensor([INF])))
    assert _worst(_evaluate(1, x), x.double().rsqrt()) <= 2


@pytest.mark.gpu
@pytest.mark.parametrize("by", [2.0 ** -20, 1e-3, 0.3, 1.0, 3.0, 5.0, 16.0, 1 - 2.0 ** -24, 1e3, 2.0 ** 20])
def test_divided(by):
    x = torch.cat((_points(2.0 ** -100, 3.4e38, signs=True), torch.tensor([INF, -INF])))
    by = torch.tensor(by).item()
    want = x.double() / by
    got, over = _evaluate(2, x, by), want.abs() > 3.4e38  # (at the very end of the range the rounded product may be infinite before the quotient is)
    assert _worst(got[~over], want[~over]) <= 0.51
    assert (got[over].abs() > 3.39e38).all() and torch.equal(got[over].sign(), want[over].sign())


@pytest.mark.gpu
def test_softplus():
    x = torch.cat((_points(2.0 ** -30, 3.4e38, signs=True), torch.linspace(-87, 30, 400001), torch.tensor([INF, -INF])))
    x = x[~((x < -87) & (x > -110))]  # (results below 2^-126 keep fewer digits)
    want = torch.where(x < -110, 0.0, torch.clamp(x.double(), min=0) + torch.log1p(torch.exp(-x.double().abs())))
    assert _worst(_evaluate(3, x), want) <= 3
    x = torch.linspace(-110, -87, 10001)
    assert (_evaluate(3, x) - torch.exp(x.double())).abs().max() <= 4 * 2.0 ** -149


@pytest.mark.gpu
def test_sigmoid():
    x = torch.cat((_points(2.0 ** -30, 87.0, signs=True), torch.linspace(-87, 30, 400001), torch.tensor([88.0, 1e4, INF])))
    assert _worst(_evaluate(4, x), torch.sigmoid(x.double())) <= 3
    assert (_evaluate(4, torch.tensor([-89.0, -1e4, -INF])) == 0).all()


@pytest.mark.gpu
def test_small_tanh():
    x = torch.cat((_points(2.0 ** -126, 0.75, signs=True), torch.linspace(-0.75, 0.75, 4000001)))
    assert _worst(_evaluate(5, x), torch.tanh(x.double())) <= 0.75
