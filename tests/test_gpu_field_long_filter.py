"""The device field generator with filters of tens of thousands of taps: the
field's values against extended-precision sums of the same noise, itself in
extended precision (an offset of 3e-17 in the noise, as the rounding of 2 pi in
an FP64 Box-Muller gives it, is 120 times that in a field of xi = 4096).

Bar, root mean square in units of the field's deviation: the noise rounds at
2^-56 and its transform is good to 2^-57, the taps round at 2^-59 (41000 of them
on unit noise: 2e-16), the samples between the passes at 2^-54 and the value read
back through the interpolation at some 20 roundings (2e-16): 4e-16 together,
doubled. FP64 sums of that length wander by 8e-15; a sum whose terms are all
rounded down is off by more still, the same way everywhere."""
from __future__ import annotations

import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
LD = np.longdouble


def normals(seed, i, ny):
    """Philox4x32-10 of counter (pair, 0, i, 0) under key seed, Box-Muller."""
    M = np.uint64(0xFFFFFFFF)
    pairs = np.arange((ny + 1) // 2, dtype=np.uint64)
    c = [pairs[None, :] + np.zeros((len(i), 1), np.uint64), np.zeros((len(i), pairs.size), np.uint64),
         i.astype(np.uint64)[:, None] + 0 * pairs[None, :], np.zeros((len(i), pairs.size), np.uint64)]
    k0, k1 = seed & 0xFFFFFFFF, seed >> 32
    for r in range(10):
        if r:
            k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
        p0, p1 = np.uint64(0xD2511F53) * c[0], np.uint64(0xCD9E8D57) * c[2]
        c = [(p1 >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), p1 & M,
             (p0 >> np.uint64(32)) ^ c[3] ^ np.uint64(k1), p0 & M]
    u = [((a << np.uint64(32)) | b) >> np.uint64(11) for a, b in ((c[0], c[1]), (c[2], c[3]))]
    radius = np.sqrt(-2 * np.log((u[0].astype(LD) + 1) * LD(2.0 ** -53)))
    angle = u[1].astype(LD) * LD(2.0 ** -53) * (8 * np.arctan(LD(1)))
    z = np.stack([radius * np.cos(angle), radius * np.sin(angle)], axis=-1)
    return z.reshape(len(i), -1)[:, :ny]


@pytest.mark.parametrize("along", ["x", "y"])
@pytest.mark.parametrize("xi", [300.0, 4096.0])
def test_long_filters(Q, O, along, xi):
    import torch
    n, other, seed = 50000, 4, 31
    nx, ny = (n, other) if along == "x" else (other, n)
    w = normals(seed, np.arange(nx), ny)
    assert np.max(np.abs(w[3].astype(float) - np.asarray(O.philox_normals(seed, 3, ny)))) < 1e-14
    R = math.ceil(5 * xi)
    k = np.arange(-R, R + 1)
    t = np.exp(-LD(k * k) / (2 * LD(xi) * LD(xi)))
    t = t / np.sqrt((t * t).sum())
    lines = w.T if along == "x" else w
    full = np.stack([np.fft.irfft(np.fft.rfft(v.astype(float)) * np.fft.rfft(np.roll(np.pad(
        t.astype(float), (0, n - t.size)), -R)), n) for v in lines])
    at = np.random.default_rng(1).integers(0, n, 60)
    want = np.stack([[(t * v[(p + k) % n]).sum() for p in at] for v in lines])
    assert np.max(np.abs(want - full[:, at])) < 1e-12   # the sums and the transform agree
    want = want / LD(full.std())
    xi2 = (xi, 0.0) if along == "x" else (0.0, xi)
    f = Q.FilteredNoise.generated(nx, ny, float(nx), float(ny), 1.0, xi2[0], xi2[1], seed)
    j = np.repeat(np.arange(other), at.size).astype(float)
    p = np.tile(at, other).astype(float)
    x, y = (p, j) if along == "x" else (j, p)
    got = f.sample(torch.as_tensor(x, device="cuda"), torch.as_tensor(y, device="cuda"))[0]
    err = (got.cpu().numpy().reshape(other, -1) - want).astype(float)
    rms = float(np.sqrt(np.mean(err ** 2)))
    assert rms <= 8e-16, (rms, float(err.mean()))
