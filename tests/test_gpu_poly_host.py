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


@pytest.mark.parametrize("n,count", [(1785, 1), (1786, 3), (3571, 2), (20001, 40)])
@pytest.mark.parametrize("offset_in,offset_out", [(0, 0), (1, 0), (5, 11), (15, 1)])
def test_host_lines_at_any_offset_bitwise(Q, n, count, offset_in, offset_out):
    """Buffers that start anywhere in a 128-byte line, stretches of several
    runs a block, small and zero heights in some of the chunks; the words about
    the output stay as they were."""
    import torch
    rng = np.random.default_rng(n + offset_in)
    ny = 16
    f = Q.FilteredNoise(rng.standard_normal((n, ny)), float(n), float(ny),
                        store=Q.QEW_STORE_FP64 | Q.QEW_STORE_FP64_POLY)
    h = rng.uniform(-ny, 2 * ny, (count, n))
    h[:, 300:900] *= 1e-5
    h[-1, 1000:1500] = 0.0
    p = Q.Params(float(n), 1.1, 0.2, Q.Model.Linear)
    buf = torch.zeros(count * n + 16, dtype=torch.float64).pin_memory().numpy()
    out = torch.full((count * n + 32,), 7.5, dtype=torch.float64).pin_memory().numpy()
    hh = buf[offset_in:offset_in + count * n].reshape(count, n)
    hh[:] = h
    og = out[offset_out:offset_out + count * n].reshape(count, n)
    Q.gradient_host_batch(hh, p, f, og)
    want = Q.gradient_batch(torch.as_tensor(h, device="cuda"), p, f).cpu().numpy()
    assert np.array_equal(og.view(np.int64), want.view(np.int64))
    assert np.all(out[:offset_out] == 7.5) and np.all(out[offset_out + count * n:] == 7.5)
