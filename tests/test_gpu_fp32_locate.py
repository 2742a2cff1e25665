"""The FP32 gather's row cell and fraction from the bits of the two heights'
sum, through one noiseless Langevin step (h - a dV/dh with a = 1), against the
FP64 gradient: cell boundaries, other periods, negative heights, spacings that
are no power of two, and heights that the FP64 locate decides.

Bar: the fraction is the FP64 one rounded to FP32, so dV/dy moves by 2^-24 of
the second derivative (<= 4 c / dy); coefficients and weights in FP32, 16 taps
whose weights add up to at most 2: 20 roundings of 2^-24 of 2 c / dy. Together
less than 64 * 2^-24 c / dy an edge, two half edges a site."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def run_step(Q, f, h, p, precision):
    import torch
    d = torch.as_tensor(h, dtype=torch.float64, device="cuda").clone()
    Q.LangevinDynamics(d.numel(), 5).run(d, p, f, np.ones(1), np.zeros(1), precision=precision)
    return d.cpu().numpy()


@pytest.mark.parametrize("shape", [(1, 1), (2, 3), (5, 7), (64, 16), (300, 40)])
@pytest.mark.parametrize("spacing", [(1.0, 1.0), (0.5, 2.0 ** -6), (0.37, 1.9 / 7)])
def test_fp32_row_locate(Q, shape, spacing):
    nx, ny = shape
    rng = np.random.default_rng(nx + 10 * ny)
    Lx, Ly = nx * spacing[0], ny * spacing[1]
    f = Q.FilteredNoise(rng.standard_normal((nx, ny)), Lx, Ly,
                        store=Q.QEW_STORE_FP64 | Q.QEW_STORE_FP32)
    h = rng.uniform(0, 3 * Ly, nx)
    h[::3] = np.round(h[::3] / f.dy) * f.dy
    h[1::5] = Ly * rng.integers(0, 4, h[1::5].size)
    h[2::7] = rng.uniform(-2 * Ly, 0, h[2::7].size)
    c = np.max(np.abs(f.coefficients()))
    p = Q.Params(Lx, 0.0, 0.0)
    a, b = (run_step(Q, f, h, p, k) for k in (Q.QEW_PREC_FP32_SPLIT, Q.QEW_PREC_FP64))
    assert np.max(np.abs(a - b)) <= spacing[0] * 64 * 2.0 ** -24 * c / f.dy + 4e-16 * np.max(np.abs(h))


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf, 1e300, 5e-324, -5e-324, 1e15])
def test_fp32_row_locate_special_heights(Q, bad):
    n, ny = 64, 16
    rng = np.random.default_rng(3)
    f = Q.FilteredNoise(rng.standard_normal((n, ny)), float(n), float(ny),
                        store=Q.QEW_STORE_FP64 | Q.QEW_STORE_FP32)
    h = rng.uniform(0, ny, n)
    h[10] = bad
    p = Q.Params(float(n), 0.0, 0.0)
    a, b = (run_step(Q, f, h, p, k) for k in (Q.QEW_PREC_FP32_SPLIT, Q.QEW_PREC_FP64))
    assert np.array_equal(np.isfinite(a), np.isfinite(b))
    far = np.ones(n, bool)
    far[9:12] = False
    c = np.max(np.abs(f.coefficients()))
    assert np.max(np.abs(a - b)[far]) <= 64 * 2.0 ** -24 * c + 4e-16 * ny
