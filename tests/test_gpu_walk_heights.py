"""The linear gradient on the cell-polynomial store where a chunk's heights
differ by many orders of magnitude, or all lie within a fraction of a row of
zero: every site as exact as FP64 sums of its own three heights make it.

Bar: the neighbours' sum, the second difference and its product with tension
over spacing round at up to 2, 4 and 4 times the largest of a site's three
heights: 10 half ulps of it; an edge's dV/dy is within
32 ulps of its stencil's largest coefficient (tests/test_gpu_dynamic_range.py)
and carries its row coordinate's rounding, at most 4 ulps of the edge's larger
height, through the field's curvature (at most 4 coefficients a cell squared)."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -53
LD = np.longdouble


def line(kind, n, rng):
    u = rng.uniform(-1.0, 1.0, n)
    if kind == "zero":
        return 0.0 * u
    if kind == "tiny":
        return 1e-300 * u
    if kind == "eighth":
        return u / 8
    if kind == "jumps":                       # one site in 90 far above its neighbours
        h = 1e-6 * u
        h[::90] += 5000.0
        return h
    if kind == "orders":                      # runs of sites at every order of magnitude
        return u * np.exp2(10.0 * np.sin(np.arange(n) / 17.0))
    if kind == "crossing":                    # a smooth line through zero
        return 40.0 * np.sin(2 * np.pi * np.arange(n) / n * 3) + 1e-9 * u
    h = 1e-3 * u                              # small heights at both sides of chunk ends
    h[[0, 254, 255, 256, 509, 510, n - 1]] = 700.0
    return h


@pytest.mark.parametrize("kind", ["zero", "tiny", "eighth", "jumps", "orders", "crossing", "ends"])
@pytest.mark.parametrize("spacing", [1.0, 0.7])
@pytest.mark.parametrize("scale", [0.0, 1.0])
def test_small_heights_beside_large_ones(Q, kind, spacing, scale):
    import torch
    n, ny = 1100, 64
    rng = np.random.default_rng(8)
    f = Q.FilteredNoise(scale * rng.standard_normal((n, ny)), float(n), spacing * ny,
                        store=Q.QEW_STORE_FP64 | Q.QEW_STORE_FP64_POLY)
    h = line(kind, n, rng) * spacing
    tension = 1.3
    p = Q.Params(float(n), tension, 0.0, Q.Model.Linear)
    g = Q.gradient(torch.as_tensor(h, device="cuda"), p, f).cpu().numpy()
    hm, hp = np.roll(h, 1).astype(LD), np.roll(h, -1).astype(LD)
    want = -LD(tension) * (hm + hp - 2 * h.astype(LD))
    big = np.maximum(np.abs(h), np.maximum(np.abs(np.roll(h, 1)), np.abs(np.roll(h, -1))))
    bar = 10 * EPS * tension * big + 1e-320
    if scale:
        c = f.coefficients()
        i = np.arange(n)
        y = (h.astype(LD) + hp) / 2 / LD(f.dy)
        gx = (i + np.roll(i, -1)) * 0.5
        iy, ix = np.floor(y), np.floor(gx).astype(int)
        t = y - iy
        fx = gx - ix
        o = 1 - fx
        wx = [o ** 3 / 6, (4 - 6 * fx ** 2 + 3 * fx ** 3) / 6, (1 + 3 * fx + 3 * fx ** 2 - 3 * fx ** 3) / 6,
              fx ** 3 / 6]
        dw = [-(1 - t) ** 2 / 2, (-12 * t + 9 * t * t) / 6, (3 + 6 * t - 9 * t * t) / 6, t * t / 2]
        dv, cl = 0, np.zeros(n)
        for a in range(4):
            for b in range(4):
                k = c[(ix + a - 1) % n, (iy.astype(int) + b - 1) % ny]
                dv = dv + wx[a] * dw[b] * k.astype(LD)
                cl = np.maximum(cl, np.abs(k))
        dv = dv / LD(f.dy)
        rows = np.maximum(np.abs(h), np.abs(np.roll(h, -1))) / f.dy
        # a negative coordinate is folded into the period first, at the period's ulp
        edge = (32 + 16 * (rows + np.where(y < 0, ny, 0))) * EPS * cl / f.dy
        want = want + (np.roll(dv, 1) + dv) / 2
        bar = bar + (np.roll(edge, 1) + edge) / 2 + 8 * EPS * np.abs(want)
    err = np.abs(g - want) / bar
    assert np.all(err <= 1), (int(np.argmax(err)), float(err.max()))
