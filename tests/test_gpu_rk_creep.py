"""The cubic-cell forward-zero search on lines that have nearly come to rest:
sites whose velocity at the start of their search is rounding, zeros within an
ulp or a tolerance of either end of the bracket. Line and verdict of every
search form are the plain form's bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,ny,store", [(64, 96, "fp64"), (258, 128, "fp64"), (258, 128, "poly"),
                                        (1024, 1100, "fp64")])
def test_resting_lines_bitwise(Q, n, ny, store):
    import torch
    flags = Q.QEW_STORE_FP64 | (Q.QEW_STORE_FP64_POLY if store == "poly" else 0)
    f = Q.FilteredNoise.generated(n, ny, float(n), float(ny), 1.0, 4.0, 4.0, 17 + n, store=flags)
    ctx = f.ctx

    def rp(sweeps, root_tol=1e-10, sweep_tol=1e-30):
        return Q.RkParams(dstep=0.5, max_advance=float(ny), root_tol=root_tol, sweep_tol=sweep_tol,
                          runaway=2.0 * ny, max_sweeps=sweeps)

    rest = torch.full((n,), ny / 2 + 0.25, dtype=torch.float64, device="cuda")
    p0 = Q.Params(float(n), 1.0, 0.05, Q.Model.Linear)
    Q.rk_block(rest, p0, f, rp(600))
    for df, tol in ((0.0, 1e-10), (1e-13, 1e-10), (1e-11, 1e-10), (1e-9, 1e-12), (-1e-12, 1e-10),
                    (0.0, 0.0)):
        p = Q.Params(float(n), 1.0, 0.05 + df, Q.Model.Linear)
        want = rest.clone()
        rw = Q.rk_block(want, p, f, rp(6, tol), form=Q.QEW_RK_PLAIN)
        try:
            for cand in (-1, 0, 1, 2):
                ctx.force_tune_candidate(Q.QEW_TUNE_RK_SEARCH, cand)
                got = rest.clone()
                rg = Q.rk_block(got, p, f, rp(6, tol), form=Q.QEW_RK_RESIDENT)
                assert torch.equal(got.view(torch.int64), want.view(torch.int64)), (df, tol, cand)
                assert (rg.blocked, rg.runaway, rg.sweeps) == (rw.blocked, rw.runaway, rw.sweeps)
        finally:
            ctx.force_tune_candidate(Q.QEW_TUNE_RK_SEARCH, -1)
