"""The arclength slope s / sqrt(1 + s^2) of an edge (the integer root and one
FP64 product) against extended precision, over the magnitudes of s that its
branches cover: rms, bias and largest error.

The line is flat in pairs of sites, so every second edge has slope zero and,
without a field, the gradient of a pair's sites is the one slope beside them,
with nothing rounded after it (tension 1, spacing 1, the heights chosen so
that their differences are exact).

Bars, in ulps of the slope: the root and the product round to nearest once
each, and an error of the root's half ulp is up to one ulp of the slope: 1.5 at
most, and sqrt(1/12 + 2^2/12) = 0.65 rms if that factor were always 2 (it is
spread between 1/2 and 2: 0.29 sqrt(1 + 4/3) = 0.44 for a uniform logarithm);
0.55 is what FP64's own root and division give. Rounding to nearest is itself
one-sided where the root is within a few ulps of 1 (slopes about 2^-26), so the
bias is measured against the correctly rounded root times s: the two differ for
one slope in a thousand, by an ulp either way, and the difference's mean over
2^17 slopes scatters by 1e-4; 0.005 is a fiftieth of rounding's own spread.

With a spacing that is no power of two the difference of heights is divided by
it and rounded once more (a quarter of an ulp more in the square of the rms);
its reciprocal's own rounding must not appear, which would move every slope of
the line the same way by up to an ulp."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
LD = np.longdouble


@pytest.mark.parametrize("lo,hi", [(-34, -29), (-28, -20), (-10, -4), (-4, -1), (-1, 1), (1, 6), (6, 8)])
def test_slope_rounds_to_nearest(Q, lo, hi):
    import torch
    rng = np.random.default_rng(1000 + lo)
    m = 1 << 17
    # |dh| in [2^lo, 2^hi) as odd multiples of 2^(hi - 34): sums of pairs up and
    # down stay below 2^(hi + 18), 52 bits in all
    k = np.exp2(34 + rng.uniform(lo - hi, 0.0, m))
    dh = np.ldexp(2.0 * np.floor(k / 2) + 1.0, hi - 34) * rng.choice([-1.0, 1.0], m)
    h = np.concatenate([[0.0], np.cumsum(dh)])
    assert np.array_equal(np.diff(h), dh)
    line = np.repeat(h, 2)
    n = line.size
    g = Q.gradient(torch.as_tensor(line, device="cuda"), Q.Params(float(n), 1.0, 0.0, Q.Model.Arclength),
                   Q.ZeroNoise()).cpu().numpy()
    got = -g[1:-1:2]  # site 2k + 1: 0 - slope of the edge to site 2k + 2
    assert got.size == m
    x = dh.astype(np.longdouble)
    want = x / np.sqrt(1 + x * x)
    ideal = dh * (1 / np.sqrt(1 + x * x)).astype(np.float64)
    err = ((got.astype(np.longdouble) - want) / np.spacing(np.abs(got))).astype(np.float64) * np.sign(dh)
    bias = np.mean((np.abs(got) - np.abs(ideal)) / np.spacing(np.abs(got)))
    stat = "rms %.3f bias %.4f max %.3f" % (np.sqrt(np.mean(err ** 2)), bias, np.abs(err).max())
    assert abs(bias) <= 0.005, stat
    assert np.sqrt(np.mean(err ** 2)) <= 0.55, stat
    assert np.abs(err).max() <= 1.51, stat


def test_slope_with_a_spacing_whose_reciprocal_rounds_far(Q):
    """dx with 1 / dx almost half an ulp from a number: the slopes stay unbiased."""
    import torch
    rng = np.random.default_rng(4)
    m = 1 << 15
    n = 2 * (m + 1)
    cand = rng.uniform(1.0, 2.0, 20000)
    off = np.abs((1 / cand.astype(LD) - (1 / cand).astype(LD)) / np.spacing(1 / cand))
    dx = float(cand[np.argmax(off)])
    assert off.max() > 0.45
    k = rng.integers(1 << 20, 1 << 21, m).astype(np.float64) * rng.choice([-1.0, 1.0], m)
    dh = np.ldexp(2 * k + 1, -25)
    line = np.repeat(np.concatenate([[0.0], np.cumsum(dh)]), 2)
    length = float(n) * dx
    x = dh.astype(LD) / (length / n)  # the spacing as the model forms it
    got = -Q.gradient(torch.as_tensor(line, device="cuda"),
                      Q.Params(length, 1.0, 0.0, Q.Model.Arclength), Q.ZeroNoise()).cpu().numpy()[1:-1:2]
    want = x / np.sqrt(1 + x * x)
    err = ((got - want) / np.spacing(np.abs(got))).astype(np.float64) * np.sign(dh)
    # three roundings of at most a third of an ulp rms each, as seen in the
    # slope's ulps; the mean of 2^15 of them scatters by 0.003
    assert abs(err.mean()) <= 0.01 and np.sqrt(np.mean(err ** 2)) <= 0.6
