"""The store's gradient where spacings and coefficients are at the ends of
FP64's range: what the integer forms cannot hold goes to FP64 sums, with the
linear model's result. Strong columns far away; where the line is compared the
field is exactly zero, so the reference-order kernel's result is finite and
its elastic part the whole of it (a few roundings: 1e-14)."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model", [0, 1])
@pytest.mark.parametrize("amplitude,dx,dy", [(2.0 ** 590, 2.0 ** 500, 1.0), (2.0 ** 700, 1.0, 2.0 ** -400),
                                             (2.0 ** -690, 2.0 ** -200, 1.0), (1.0, 1.0, 1.0)])
def test_spacings_and_coefficients_at_the_ends(Q, model, amplitude, dx, dy):
    import torch
    nx, ny = 1024, 16
    v = np.zeros((nx, ny))
    v[:3] = amplitude * np.random.default_rng(1).standard_normal((3, ny))
    f = Q.FilteredNoise(v, nx * dx, ny * dy, store=Q.QEW_STORE_FP64 | Q.QEW_STORE_FP64_POLY)
    assert not np.any(f.coefficients()[200:-200])
    h = dx * np.random.default_rng(2).uniform(-1.0, 1.0, nx)
    p = Q.Params(nx * dx, 1.5, 0.0, Q.Model(model))
    t = torch.as_tensor(h, device="cuda")
    got = Q.gradient(t, p, f).cpu().numpy()[250:-250]
    want = Q.gradient(t, p, f, precision=Q.QEW_PREC_FP64_REFERENCE).cpu().numpy()[250:-250]
    assert np.all(np.isfinite(want)) and np.any(want)
    assert np.max(np.abs(got - want)) <= 1e-14 * np.max(np.abs(want))
