"""The cubic-cell forward-zero search where the field is steeper than the
line's elasticity: a site's two edges whose slopes nearly cancel, so that v
falls as slowly as the elastic part alone while each edge magnifies the
rounding of its height sum, at heights of hundreds to many millions of rows;
spacings that are no power of two and heights below zero. Line and verdict of
every search form are the plain form's bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def forms_agree(Q, f, h0, p, dstep, tol, sweeps, scale=1.0):
    import torch
    rp = Q.RkParams(dstep=dstep, max_advance=1000.0 * dstep, root_tol=tol, sweep_tol=1e-30 * scale,
                    runaway=1e9 * scale, max_sweeps=sweeps)
    want = h0.clone()
    rw = Q.rk_block(want, p, f, rp, form=Q.QEW_RK_PLAIN)
    assert bool((want != h0).any())
    try:
        for cand in (0, 1, 2):
            f.ctx.force_tune_candidate(Q.QEW_TUNE_RK_SEARCH, cand)
            got = h0.clone()
            rg = Q.rk_block(got, p, f, rp, form=Q.QEW_RK_RESIDENT)
            same = got.view(torch.int64) == want.view(torch.int64)
            assert bool(same.all()), (tol, cand, int((~same).sum()))
            assert (rg.blocked, rg.runaway, rg.sweeps) == (rw.blocked, rw.runaway, rw.sweeps)
    finally:
        f.ctx.force_tune_candidate(Q.QEW_TUNE_RK_SEARCH, -1)
    return want


@pytest.mark.parametrize("spacing,base", [(1.0, 600.25), (1.0, 3.0e7), (0.375, 3.0e7), (0.37, 2.0e7),
                                          (1.0, -3.0e6)])
@pytest.mark.parametrize("steep", [10.0, 100.0])
def test_cancelling_edges_bitwise(Q, steep, spacing, base):
    """Edge e of the line lies on a field column that holds (-1)^e A cos(2 pi y
    / 1024 rows): on a nearly flat line a site's two edges pull with opposite
    slopes of `steep` times half the elastic one, changing little along a cell."""
    import torch
    n, ny = 1024, 1024
    a = steep / (0.25 * (2 * np.pi / ny) ** 2) * spacing ** 2
    sign = 1.0 - 2.0 * (np.arange(n) % 2)
    v = np.zeros((2 * n, ny))
    v[1::2] = sign[:, None] * a * np.cos(2 * np.pi * np.arange(ny) / ny)[None, :]
    rng = np.random.default_rng(3)
    v += 0.05 * spacing ** 2 * rng.standard_normal(v.shape)
    f = Q.FilteredNoise(v, float(n), spacing * ny)
    h0 = torch.as_tensor((base + 0.05 / steep * rng.uniform(-1, 1, n)) * spacing, device="cuda")
    p = Q.Params(float(n), 1.0, 0.05 * spacing, Q.Model.Linear)
    for tol, sweeps in ((1e-10 * spacing, 6), (0.0, 4)):
        forms_agree(Q, f, h0, p, 0.5 * spacing, tol, sweeps)


@pytest.mark.parametrize("tension,xi,amplitude", [(0.01, 1.0, 1.0), (1.0, 1.0, 30.0), (2.0, 0.7, 0.3)])
@pytest.mark.parametrize("spacing,base,store", [(1.0, 40000.5, "fp64"), (0.37, -300.0, "poly")])
def test_steep_random_fields_bitwise(Q, tension, xi, amplitude, spacing, base, store):
    import torch
    n, ny = 2048, 1024
    flags = Q.QEW_STORE_FP64 | (Q.QEW_STORE_FP64_POLY if store == "poly" else 0)
    f = Q.FilteredNoise.generated(n, ny, float(n), spacing * ny, amplitude, xi, xi, 77, store=flags)
    h0 = torch.as_tensor((base + np.random.default_rng(5).uniform(0, 20.0, n)) * spacing, device="cuda")
    p = Q.Params(float(n), tension, 0.2 * amplitude, Q.Model.Linear)
    for tol, sweeps in ((1e-10 * spacing, 40), (0.0, 12)):
        forms_agree(Q, f, h0, p, 0.5 * spacing, tol, sweeps)


@pytest.mark.parametrize("height,force", [(2.0 ** -90, 2.0 ** -34), (2.0 ** -60, 2.0 ** -66), (2.0 ** 60, 2.0 ** 50)])
def test_scaled_units_bitwise(Q, height, force):
    """Heights and forces in units whose velocities leave the range of single
    precision, in which the search compares slopes: a power of two scales the
    plain form's line exactly, and every form follows it."""
    import torch
    n, ny = 1024, 256
    v = np.random.default_rng(4).standard_normal((n, ny))
    rng = np.random.default_rng(5)
    h = torch.as_tensor(100.0 + rng.uniform(0, 5.0, n), device="cuda")
    lines = []
    for a, b in ((1.0, 1.0), (height, force)):
        f = Q.FilteredNoise(v * (a * a * b), float(n), a * ny)
        p = Q.Params(float(n), 2.0 * b, 0.2 * a * b, Q.Model.Linear)
        h0 = h * a
        lines.append(forms_agree(Q, f, h0, p, 0.5 * a, 1e-10 * a, 20, a) / a)
    assert torch.equal(*lines)
