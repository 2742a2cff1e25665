"""FP64 gathers on fields whose coefficients differ by many orders of
magnitude: a few strong rows and a weak rest, where the lines lie. The
fixed-point sums take each stencil's own unit, so the weak region keeps the
accuracy of FP64 sums there, with and without the cell-polynomial store, in
the gradient, the energy and the solvers.

Bar, from the format: a tap is cut at 2^-56 of its stencil's largest
coefficient c, the weights add up to at most 1 along x and 2 along y, and the
results round a few times: 32 ulps of c over dy for an edge (16 for a sum of
values), the bar that the FP64 sums of some twenty roundings meet. The midpoint of an edge
is rounded to FP64 as the reference rounds it, but for the linear gradient on
the store, which forms it exactly save about the line's ends (there FP64's
rounding of the coordinate is allowed for). Where the row spacing is no power of two the
store's row coordinate is a product within an ulp of the quotient, which the
field's curvature (at most 4 c a cell squared) carries into the slope: 8 ulps
of the coordinate times c more."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -53
LD = np.longdouble


def t64(a):
    import torch
    return torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")


def weights(t, deriv):
    t = t.astype(LD)
    o = 1 - t
    if deriv:
        return [-o * o / 2, (-12 * t + 9 * t * t) / 6, (3 + 6 * t - 9 * t * t) / 6, t * t / 2]
    return [o ** 3 / 6, (4 - 6 * t * t + 3 * t ** 3) / 6, (1 + 3 * t + 3 * t * t - 3 * t ** 3) / 6,
            t ** 3 / 6]


def gather(c, dx, dy, x, y, deriv):
    """V or dV/dy at (x, y) in extended precision from the FP64 coordinates,
    and the largest |coefficient| of each stencil."""
    nx, ny = c.shape
    gx, gy = x / dx, y / dy
    ix, iy = np.floor(gx), np.floor(gy)
    wx, wy = weights(gx - ix, False), weights(gy - iy, deriv)
    out, big = 0, np.zeros(x.size)
    for a in range(4):
        for b in range(4):
            k = c[(ix.astype(int) + a - 1) % nx, (iy.astype(int) + b - 1) % ny]
            out = out + wx[a] * wy[b] * k.astype(LD)
            big = np.maximum(big, np.abs(k))
    return (out / dy if deriv else out), big


def strong_rows(nx, ny, ratio, seed):
    v = np.random.default_rng(seed).standard_normal((nx, ny))
    v[:, :3] *= ratio
    return v


@pytest.mark.parametrize("store", ["fp64", "poly"])
@pytest.mark.parametrize("geometry", ["unit", "odd", "offgrid"])
@pytest.mark.parametrize("ratio", [1.0, 4e3, 4e6, 4e10, 1e30])
def test_weak_region_keeps_its_accuracy(Q, store, geometry, ratio):
    nx, ny = 96, 512
    Lx, Ly = (0.37 * nx, 1.9 * ny) if geometry == "odd" else (float(nx), float(ny))
    n = 3 * nx + 1 if geometry == "offgrid" else nx
    f = Q.FilteredNoise(strong_rows(nx, ny, ratio, 5), Lx, Ly,
                        store=Q.QEW_STORE_FP64 | (Q.QEW_STORE_FP64_POLY if store == "poly" else 0))
    c = f.coefficients()
    h = np.random.default_rng(7).uniform(200.0, 310.0, n) * f.dy
    dx = Lx / n
    i = np.arange(n)
    x = (i + np.roll(i, -1)) * 0.5 * dx
    y = (np.roll(h, -1) + h) * 0.5
    exact_y = (np.roll(h, -1).astype(LD) + h) / 2
    walk = store == "poly" and geometry != "offgrid"
    loc = 8 * 310.0 if geometry == "odd" else 0.0
    ends = np.zeros(n)
    ends[[0, -1]] = 8 * 310.0 if walk else 0.0
    for model in (0, 1):
        dv, big = gather(c, f.dx, f.dy, x, exact_y if walk and model == 0 else y, True)
        assert big.max() < 40.0  # the strong rows' tails are far below the weak values here
        want = dx * (np.roll(dv, 1) + dv) / 2
        bar = dx * (32 + loc + ends) * EPS * np.maximum(np.roll(big, 1), big) / f.dy
        g = Q.gradient(t64(h), Q.Params(Lx, 0.0, 0.0, Q.Model(model)), f).cpu().numpy()
        assert np.all(np.abs(g - want) <= bar), float(np.max(np.abs(g - want) / bar))
    v, big = gather(c, f.dx, f.dy, x, y, False)
    e = Q.objective(t64(h), Q.Params(Lx, 0.0, 0.0), f)
    bar = dx * ((16 + loc) * EPS * big.sum() + 64 * EPS * np.abs(v).sum())
    assert abs(e - (dx * v).sum()) <= bar


@pytest.mark.parametrize("store", ["fp64", "poly"])
def test_solvers_do_not_see_a_strong_region_far_away(Q, store):
    """Rows 4e10 times stronger, 200 rows away, change no bit of a gradient, a
    solve, a Langevin run or a block of sweeps: the coefficients where the line
    lies are the same to the last bit."""
    n, ny = 512, 512
    flags = Q.QEW_STORE_FP64 | (Q.QEW_STORE_FP64_POLY if store == "poly" else 0)
    h0 = np.random.default_rng(2).uniform(250.0, 260.0, n)
    out = []
    for ratio in (1.0, 4e10):
        f = Q.FilteredNoise(strong_rows(n, ny, ratio, 11), float(n), float(ny), store=flags)
        c = f.coefficients()[:, 180:330]
        lines = [t64(h0) for _ in range(4)]
        lp = Q.LbfgsParams(m=10, ftol=1e-8, max_iter=60, precondition=True, precond_shift=0.1,
                           ls_fallback=True)
        Q.lbfgs_minimize(lines[0], Q.Params(float(n), 4.0, 0.0, Q.Model.Linear), f, lp)
        Q.LangevinDynamics(n, 3).run(lines[1], Q.Params(float(n), 1.0, 0.1, Q.Model.Arclength), f,
                                     np.full(50, 0.01), np.full(50, 0.05))
        rp = Q.RkParams(dstep=0.5, max_advance=64.0, root_tol=1e-10, sweep_tol=1e-8, runaway=60.0,
                        max_sweeps=25)
        p = Q.Params(float(n), 4.0, 0.2, Q.Model.Linear)
        for form, k in ((Q.QEW_RK_PLAIN, 2), (Q.QEW_RK_RESIDENT, 3)):
            Q.rk_block(lines[k], p, f, rp, form=form)
        g = Q.gradient(t64(h0), p, f)
        out.append([c] + [x.cpu().numpy() for x in lines + [g]])
        assert np.array_equal(out[-1][3].view(np.int64), out[-1][4].view(np.int64))
    for a, b in zip(*out):
        assert np.array_equal(a.view(np.int64), b.view(np.int64))
