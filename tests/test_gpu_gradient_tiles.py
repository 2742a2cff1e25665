"""gradient() and gradient_batch() on the FP64 gathers at the edges of their
tiles (127 sites a block): lines of one site to one more than three tiles, one
to three lines in a launch, against the oracle on the same coefficients, and
every row of a batch bit for bit what the line alone gives.

Bar, as for the fixed-point gather: 32 ulps of the largest coefficient over dy
per edge and 16 ulps of the elastic terms."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -53


@pytest.mark.parametrize("n", [1, 2, 3, 126, 127, 128, 253, 254, 255, 382])
@pytest.mark.parametrize("model", [0, 1])
def test_gradient_tile_edges(Q, O, n, model):
    import torch
    rng = np.random.default_rng(n + 1000 * model)
    nx, ny, Lx, Ly = 60, 24, 0.5 * n, 3.0
    fld = rng.standard_normal((nx, ny))
    f = Q.FilteredNoise(fld, Lx, Ly)
    coef = f.coefficients()
    of = O.BSplineField(fld, Lx, Ly, coef=coef)
    h = rng.uniform(0, 2 * Ly, (3, n))
    p = Q.Params(Lx, 0.8, 0.3, Q.Model(model))
    bar = 0.5 * 32 * EPS * np.max(np.abs(coef)) / f.dy + 16 * EPS * 0.8 * 2 * Ly / 0.5
    ht = torch.as_tensor(h, device="cuda")
    rows = Q.gradient_batch(ht, p, f).cpu().numpy()
    two = Q.gradient_batch(ht[:2].contiguous(), p, f).cpu().numpy()
    ref = Q.gradient_batch(ht, p, f, precision=Q.QEW_PREC_FP64_REFERENCE).cpu().numpy()
    assert np.array_equal(two, rows[:2])
    for k in range(3):
        one = Q.gradient(ht[k].contiguous(), p, f).cpu().numpy()
        assert np.array_equal(one, rows[k])
        o = O.gradient(h[k], O.params(Lx, 0.8, 0.3, model), of)
        assert np.max(np.abs(one - o)) <= bar
        assert np.array_equal(ref[k], o)
