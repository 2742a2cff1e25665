"""Gradients of pinned host lines on the cell-polynomial store (runs of 2040
sites staged in shared memory) at the edges of their runs: lines shorter than a
run, one site about a run and its halo, lines that start at every alignment
(odd n), negative and non-finite heights. The device batch's bits."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 254, 255, 2039, 2040, 2041, 2042, 2295, 2297, 4337, 9001])
@pytest.mark.parametrize("spacing", [1.0, 0.7])
def test_host_lines_bitwise(Q, n, spacing):
    import torch
    rng = np.random.default_rng(n)
    ny = 20
    f = Q.FilteredNoise(rng.standard_normal((n, ny)), float(n), spacing * ny,
                        store=Q.QEW_STORE_FP64 | Q.QEW_STORE_FP64_POLY)
    h = rng.uniform(-ny, 2 * ny, (3, n))
    if n > 300:
        h[1, 290] = np.nan
    p = Q.Params(float(n), 1.1, 0.2, Q.Model.Linear)
    hh = torch.as_tensor(h).pin_memory().numpy()
    out = torch.empty((3, n), dtype=torch.float64).pin_memory().numpy()
    Q.gradient_host_batch(hh, p, f, out)
    want = Q.gradient_batch(torch.as_tensor(h, device="cuda"), p, f).cpu().numpy()
    assert np.array_equal(out.view(np.int64), want.view(np.int64))
