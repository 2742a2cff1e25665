"""The integer row cell and fraction (fx_cell64) against the reference's FP64
fold on the host, over every kind of coordinate it accepts: all magnitudes and
signs, whole cells and periods, and the FP64 numbers either side of them. It
may decline what the reference's rounding decides, but only that."""
from __future__ import annotations

import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    out = str(tmp_path_factory.mktemp("cell") / "cell_probe")
    subprocess.run([nvcc, "-O2", "-std=c++17", "-Xcompiler", "-ffp-contract=off",
                    "-gencode", "arch=compute_103a,code=sm_103a",
                    os.path.join(HERE, "native", "cell_probe.cu"), "-o", out], check=True)
    return out


def run(probe, g, n):
    text = "\n".join("%x %d" % (b, k) for b, k in zip(g.view(np.uint64), n))
    r = subprocess.run([probe], input=text, capture_output=True, text=True)
    assert r.returncode == 0, r.stdout[:2000]
    last = r.stdout.split()
    return int(last[1]), int(last[3])


def neighbours(g, steps=3):
    out = [g]
    up = dn = g
    for _ in range(steps):
        up, dn = np.nextafter(up, np.inf), np.nextafter(dn, -np.inf)
        out += [up, dn]
    return np.concatenate(out)


def test_fold_is_the_reference_s(probe):
    rng = np.random.default_rng(1)
    g, n = [], []
    for period in (1, 2, 3, 5, 7, 64, 77, 1000, 1024, 65535, 1 << 20, (1 << 21) - 1):
        m = 4000
        r = np.exp2(rng.uniform(-70, 49.5, m)) * rng.choice([-1.0, 1.0], m)
        k = rng.integers(-1000, 1000, m).astype(float)
        far = np.floor(np.exp2(rng.uniform(0, 48.0 - np.log2(period), m))) * rng.choice([-1.0, 1.0], m)
        near = neighbours(np.concatenate([k * period, far * period, k * period + 0.5,
                                          far * period - rng.integers(0, period, m),
                                          rng.integers(-3 * period, 3 * period, m).astype(float)]))
        small = np.exp2(rng.uniform(-60, 0, m)) * rng.choice([-1.0, 1.0], m)
        near = near[np.abs(near) < 2.0 ** 50]
        a = np.concatenate([r, near, small, k * period - np.abs(small)])
        g.append(a)
        n.append(np.full(a.size, period))
    g, n = np.concatenate(g), np.concatenate(n)
    accepted, declined = run(probe, g, n)
    assert accepted + declined == g.size
    # declined: negative coordinates of a one-cell period, and the last two
    # numbers of later periods
    one = np.count_nonzero((n == 1) & np.signbit(g))
    with np.errstate(invalid="ignore"):
        left = n - np.mod(g, n)
    late = np.count_nonzero((n > 1) & ((g >= n) | (g < -n)) & (left <= 4 * np.spacing(np.abs(g))))
    zero = np.count_nonzero((n == 1) & (g == 0.0) & np.signbit(g))
    assert declined <= one + late + zero + np.count_nonzero((n == 1) & (g >= 1)), (declined, one, late)


def test_ordinary_coordinates_are_not_declined(probe):
    rng = np.random.default_rng(2)
    for period in (64, 77, 1024):
        k = rng.integers(-5000, 5000, 20000).astype(float)
        g = (k + rng.uniform(0.0, 1.0, k.size)) * period      # every cell of every period
        _, declined = run(probe, g, np.full(g.size, period))
        assert declined == 0


def test_non_finite_and_huge_coordinates_are_declined(probe):
    g = np.array([np.nan, np.inf, -np.inf, 2.0 ** 50, -2.0 ** 60, 1e300, 5e-324, -1e-310])
    accepted, declined = run(probe, g, np.full(g.size, 64))
    assert (accepted, declined) == (0, g.size)
