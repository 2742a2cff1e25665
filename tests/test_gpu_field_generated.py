"""The device field generator (fixed-point Box-Muller and Gaussian filter, the
two-pass moments, the one-pass prefilter) against its definition in FP64 on
the host, at the edges of its ranges: single rows and columns, lengths around
the prefilter's chunk of 64, no filter at all, a filter longer than the field.

Bar: the noise, the filter's sums and the scale each round at or below
2^-53 of their largest term, the prefilter amplifies by at most 9 (3 per
axis): 64 ulps of the largest coefficient."""
from __future__ import annotations

import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 5), (5, 1), (3, 7), (64, 65), (127, 33), (200, 130), (1000, 4)])
@pytest.mark.parametrize("xi", [(0.0, 0.0), (0.7, 3.0), (4.0, 4.0), (60.0, 2.0)])
def test_generated_field_matches_definition(Q, O, shape, xi):
    nx, ny = shape
    seed, amplitude = 12345678901234567, 0.7
    w = np.stack([np.asarray(O.philox_normals(seed, i, ny)) for i in range(nx)])
    for axis, x in ((1, xi[1]), (0, xi[0])):
        R = math.ceil(5 * x) if x > 0 else 0
        t = np.exp(-0.5 * np.arange(-R, R + 1) ** 2 / x ** 2) if x > 0 else np.ones(1)
        t /= np.sqrt(np.sum(t * t))
        w = sum(t[k + R] * np.roll(w, -k, axis=axis) for k in range(-R, R + 1))
    std = w.std()
    if std < 1e-6 * np.abs(w).max():
        pytest.skip("a constant field has no scale")
    want = O.prefilter(w * (amplitude / std))
    got = Q.FilteredNoise.generated(nx, ny, float(nx), float(ny), amplitude, xi[0], xi[1],
                                    seed).coefficients()
    # a filter that leaves a nearly constant field cancels in the deviation
    bar = 64 * 2.0 ** -53 * max(1.0, np.abs(w).max() / std)
    assert np.max(np.abs(got - want)) <= bar * np.max(np.abs(want))
    again = Q.FilteredNoise.generated(nx, ny, float(nx), float(ny), amplitude, xi[0], xi[1],
                                      seed).coefficients()
    assert np.array_equal(got, again)


def test_increments_tails(Q, O):
    """Philox increments of many steps: the fixed-point pair stays within
    4 ulps of its largest value (8.6) of the FP64 form, which rounds 2 pi u2
    (up to 4e-16 of the radius) besides."""
    n = 200001
    dyn = Q.LangevinDynamics(n, 99)
    z = dyn.peek_increments().cpu().numpy()
    assert np.max(np.abs(z - O.philox_normals(99, 0, n))) < 8.6 * 4 * 2.0 ** -52
