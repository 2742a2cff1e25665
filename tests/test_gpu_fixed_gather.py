"""The fixed-point 16-tap gather (the default FP64 gradient and energy on a
B-spline field) against the reference-order FP64 sums on the same field, at
the edges of its range: one- to four-cell fields, cell boundaries, heights of
other periods, and what it hands back to the FP64 sum (negative, huge,
subnormal and non-finite heights, a field that is zero or holds an infinity).

Bar, from the formats: a tap is cut at 2^-56 of the largest coefficient, the
weights add up to at most 1 along x and 2 along y, and the FP64 sum it is
compared with rounds some twenty times: 32 ulps of the largest coefficient
over dy per edge, and 16 ulps of the largest height for the elastic part."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -53


def t64(a):
    import torch
    return torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")


def bars(f, h, Lx, n, tension):
    c = np.max(np.abs(f.coefficients()))
    dx = Lx / n
    hm = np.max(np.abs(h[np.isfinite(h)])) if np.isfinite(h).any() else 1.0
    return dx * 32 * EPS * c / f.dy + 16 * EPS * tension * max(1.0, hm) / dx + 1e-300


@pytest.mark.parametrize("shape", [(1, 1), (2, 3), (3, 4), (4, 2), (5, 7), (96, 40), (300, 64)])
@pytest.mark.parametrize("geometry", ["unit", "pow2", "odd", "offgrid"])
def test_fixed_gather_matches_reference_order(Q, shape, geometry):
    import torch
    nx, ny = shape
    rng = np.random.default_rng(100 * nx + ny)
    Lx, Ly = {"unit": (float(nx), float(ny)), "pow2": (nx / 8.0, ny / 64.0),
              "odd": (0.37 * nx, 1.9 * ny / 7), "offgrid": (float(nx), float(ny))}[geometry]
    n = nx if geometry != "offgrid" else 3 * nx + 1
    f = Q.FilteredNoise(rng.standard_normal((nx, ny)) * 10.0 ** rng.integers(-3, 4), Lx, Ly)
    h = rng.uniform(0, 3 * Ly, n)
    h[::3] = np.round(h[::3] / f.dy) * f.dy               # cell boundaries
    h[1::5] = Ly * rng.integers(0, 4, h[1::5].size)       # whole periods
    h[2::7] = rng.uniform(-2 * Ly, 0, h[2::7].size)       # the fold's side
    for model in (0, 1):
        p = Q.Params(Lx, 0.8, 0.3, Q.Model(model))
        a = Q.gradient(t64(h), p, f).cpu().numpy()
        b = Q.gradient(t64(h), p, f, precision=Q.QEW_PREC_FP64_REFERENCE).cpu().numpy()
        assert np.max(np.abs(a - b)) <= bars(f, h, Lx, n, 0.8)
    # the energy: the value's sum has the same taps
    v, _, _ = f.sample(t64((np.arange(n) + np.roll(np.arange(n), -1)) * 0.5 * Lx / n),
                       t64(0.5 * (h + np.roll(h, -1))))
    e = Q.objective(t64(h), Q.Params(Lx, 0.0, 0.0), f)
    vs = v.cpu().numpy() * Lx / n
    c = np.max(np.abs(f.coefficients()))
    assert abs(e - vs.sum()) <= 32 * EPS * c * Lx + 64 * EPS * np.abs(vs).sum() + 1e-300
    assert torch.isfinite(v).all()


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf, 1e300, -1e300, 5e-324, 1e15])
def test_fixed_gather_special_heights(Q, bad):
    """Non-finite results exactly where the reference-order sum has them."""
    n, ny = 64, 16
    rng = np.random.default_rng(3)
    f = Q.FilteredNoise(rng.standard_normal((n, ny)), float(n), float(ny))
    h = rng.uniform(0, ny, n)
    h[10] = bad
    p = Q.Params(float(n), 1.0, 0.1)
    a = Q.gradient(t64(h), p, f).cpu().numpy()
    b = Q.gradient(t64(h), p, f, precision=Q.QEW_PREC_FP64_REFERENCE).cpu().numpy()
    assert np.array_equal(np.isfinite(a), np.isfinite(b))
    far = np.ones(n, bool)
    far[9:12] = False
    assert np.max(np.abs(a - b)[far]) <= bars(f, np.ones(1) * ny, float(n), n, 1.0)


@pytest.mark.parametrize("kind", ["zero", "inf", "tiny", "huge"])
def test_fixed_gather_field_scales(Q, kind):
    """Fields whose coefficients leave the fixed-point range take FP64 sums."""
    n, ny = 48, 12
    v = np.random.default_rng(8).standard_normal((n, ny))
    v = {"zero": 0 * v, "tiny": v * 1e-290, "huge": v * 1e290, "inf": v}[kind]
    if kind == "inf":
        v[5, 5] = np.inf
    f = Q.FilteredNoise(v, float(n), float(ny))
    h = np.random.default_rng(9).uniform(0, ny, n)
    p = Q.Params(float(n), 0.0 if kind != "zero" else 1.0, 0.0)
    a = Q.gradient(t64(h), p, f).cpu().numpy()
    b = Q.gradient(t64(h), p, f, precision=Q.QEW_PREC_FP64_REFERENCE).cpu().numpy()
    assert np.array_equal(np.isfinite(a), np.isfinite(b))
    ok = np.isfinite(b)
    if ok.any():
        c = np.max(np.abs(f.coefficients()))
        c = c if np.isfinite(c) else 0.0
        assert np.max(np.abs(a - b)[ok]) <= 32 * EPS * c + 16 * EPS * (ny if kind == "zero" else 0)
