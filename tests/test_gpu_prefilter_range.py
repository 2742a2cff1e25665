"""The B-spline prefilter of fields with a few samples many orders above the
rest, against the exact periodic solve in extended precision, coefficient by
coefficient: chunks of 64 samples start their recursions from neighbours far
enough away that a large sample beyond them does not count.

Bar: along an axis c = g sum_j s_j z^|k - j|, g = sqrt 3, z = sqrt 3 - 2; every
partial sum of the two recursions rounds at most at the same sum of |s_j|
|z|^|k - j|, and an error made j samples away arrives with |z|^j: at most
1 / (1 - |z|) = 1.4 of the 4 roundings a step on either side, 12 half ulps an
axis with the products of the gain, 32 with the second axis on top."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
LD = np.longdouble


def kernel(n, absolute):
    z = np.sqrt(LD(3)) - 2
    k = np.arange(n)
    k = np.minimum(k, n - k)
    row = np.zeros(n, dtype=LD)
    zz = abs(z) if absolute else z
    for m in range(0, 700 // n + 2):          # the periodic images
        row = row + zz ** (np.arange(n) + m * n) + zz ** ((m + 1) * n - np.arange(n))
    i = np.arange(n)
    return np.sqrt(LD(3)) * row[(i[:, None] - i[None, :]) % n]


@pytest.mark.parametrize("shape", [(300, 3), (3, 300), (129, 130), (64, 64)])
@pytest.mark.parametrize("spike", [1.0, 1e8, 1e16])
def test_prefilter_beside_large_samples(Q, shape, spike):
    nx, ny = shape
    rng = np.random.default_rng(nx)
    s = rng.standard_normal((nx, ny))
    s[nx // 3, ny // 3] *= spike
    got = Q.FilteredNoise(s, float(nx), float(ny)).coefficients()
    want = kernel(nx, False) @ s.astype(LD) @ kernel(ny, False)
    bar = 32 * 2.0 ** -53 * (kernel(nx, True) @ np.abs(s).astype(LD) @ kernel(ny, True))
    err = np.abs(got - want) / bar
    assert np.all(err <= 1), (np.unravel_index(np.argmax(err), shape), float(err.max()))
