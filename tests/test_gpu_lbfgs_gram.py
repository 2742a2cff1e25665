"""The device-resident L-BFGS (inner-product recursion, points owned by
threads, vectors in shared or global memory) against the plain host-driven
form at the edges of its partition: fewer points than threads, one point more
or less than a block or a cluster has threads, last threads with fewer points
than the others, the smallest and largest history, with and without the
preconditioner.

The potential is one convex well in h: -A cos(2 pi y / Ly + 0.3 sin(6 pi x / Lx)).
Near its minimum the Hessian is at least A (2 pi / Ly)^2 cos(0.6) dx > lam, so a
line with max |gradient| < ftol is within sqrt(n) ftol / lam of the minimum, two
such lines within twice that. (The preconditioner's shift is the well's
curvature and the slope test decides near ftol, where energies differ by their
rounding: without both the plain form leaves the well or stalls on this line.)
The recursion is the reference's term by term, so a wrong product shows as a
solve that takes many more iterations than the plain one."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
FTOL = 1e-9


@pytest.mark.parametrize("n", [1, 2, 3, 31, 255, 256, 257, 700, 2047, 2048, 2049, 4099, 8200])
@pytest.mark.parametrize("m,precondition", [(1, True), (10, True), (32, True), (10, False)])
def test_resident_solver_partitions(Q, n, m, precondition):
    import torch
    nx, ny, A = max(n, 4), 32, 2.0
    Lx = float(n)
    x = np.arange(nx)[:, None] / nx
    y = np.arange(ny)[None, :] / ny
    f = Q.FilteredNoise(-A * np.cos(2 * np.pi * y + 0.3 * np.sin(6 * np.pi * x)), Lx, float(ny))
    h0 = np.random.default_rng(n).uniform(-2.0, 2.0, n)
    lam = 0.8 * A * (2 * np.pi / ny) ** 2
    for model in (0, 1):
        p = Q.Params(Lx, 1.3, 0.01, Q.Model(model))
        lp = Q.LbfgsParams(m=m, ftol=FTOL, max_iter=5000, precondition=precondition,
                            precond_shift=lam, ls_fallback=True)
        out = []
        for form in (Q.QEW_LBFGS_PLAIN, Q.QEW_LBFGS_RESIDENT):
            h = torch.as_tensor(h0, dtype=torch.float64, device="cuda").clone()
            r = Q.lbfgs_minimize(h, p, f, lp, form=form)
            assert r.converged
            g = Q.gradient(h, p, f)
            # the gradient of the accepted line and of the stored one differ by roundings
            assert float(g.abs().max()) < FTOL + 1e-13
            out.append((h.cpu().numpy(), r))
        assert np.max(np.abs(out[0][0] - out[1][0])) <= 2 * np.sqrt(n) * FTOL / lam
        assert out[1][1].iterations <= 1.5 * out[0][1].iterations + 3
