"""The FP32 split gradient on the x-filtered store (chunks of a warp: 63, 95 or
127 sites) at the edges of its chunks, bit for bit against the one-tile-a-block
kernel, which the FP64-heights form of the same field runs on the same split:
lines of one site to several chunks, one to three lines in a launch, cells of
other periods on both sides and stencils that wrap the rows."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 3, 62, 63, 64, 65, 95, 96, 97, 126, 127, 128, 129, 191, 255, 256, 700])
@pytest.mark.parametrize("ny", [1, 3, 40])
def test_split_chunk_edges(Q, n, ny):
    import torch
    rng = np.random.default_rng(n + 1000 * ny)
    f = Q.FilteredNoise(rng.standard_normal((n, ny)), 0.25 * n, 0.7 * ny,
                        store=Q.QEW_STORE_FP64 | Q.QEW_STORE_FP32 | Q.QEW_STORE_FP32_EDGE)
    h = torch.as_tensor(rng.uniform(-2.0, 3.0, (3, n)) * f.dy * ny, device="cuda")
    ctx = f.ctx
    for model in (0, 1):
        p = Q.Params(0.25 * n, 0.9, 0.2, Q.Model(model))
        want = torch.stack([Q.gradient(h[k].contiguous(), p, f, precision=Q.QEW_PREC_FP32_SPLIT)
                            for k in range(3)]).to(torch.float32)
        ps = [Q.split_heights(h[k].contiguous(), f) for k in range(3)]
        c, fr = torch.stack([a for a, _ in ps]), torch.stack([b for _, b in ps])
        try:
            for cand in range(6):
                ctx.force_tune_candidate(Q.QEW_TUNE_GRADIENT_SPLIT, cand)
                got = Q.gradient_split_batch(c, fr, p, f)
                assert torch.equal(got.view(torch.int32), want.view(torch.int32)), cand
                one = Q.gradient_split(c[1].contiguous(), fr[1].contiguous(), p, f)
                assert torch.equal(one.view(torch.int32), want[1].view(torch.int32)), cand
        finally:
            ctx.force_tune_candidate(Q.QEW_TUNE_GRADIENT_SPLIT, -1)
