"""The work that users of qew_gb300 have it do, as cases that can be timed.

A case is a dict of plain values; ``op`` names the kind of call:

gradient   gradients of one line or a batch of lines on one pinning field, in
           FP64 (``store`` fp64: 16 taps per edge, any geometry; poly: the
           cell-polynomial store) or on FP32 split heights (store edge)
energy     what a minimiser outside the library asks for at each step: the
           energy, a trial energy along a direction, and the gradient
lbfgs      one line relaxed by the preconditioned L-BFGS solver
ensemble   many lines of uneven length relaxed in one call, in FP64 as static_sweep
           does (an FP32 first phase ends in another minimum when a last bit
           changes, so its lines cannot be compared from build to build)
langevin   an annealed Langevin schedule run on the device, FP64 or FP32
depinning  a block of Rosso-Krauth no-passing sweeps at a fixed force
field      a pinning field generated on the device (as for each served
           request), or built from real-space values, and the first gradients
           of lines on it

Fields are white noise filtered to a correlation length of ``xi`` cells, unit
variance; ``length`` and ``height`` are the field's physical extents (0: one
unit per column / per row).
"""
import math

import numpy as np
import torch

import qew_gb300 as Q

STORES = {"fp64": Q.QEW_STORE_FP64,
          "poly": Q.QEW_STORE_FP64 | Q.QEW_STORE_FP64_POLY,
          "edge": Q.QEW_STORE_FP64 | Q.QEW_STORE_FP32 | Q.QEW_STORE_FP32_EDGE,
          "both": Q.QEW_STORE_FP64 | Q.QEW_STORE_FP32}


def listed():
    return [
        # The smallest call: one gradient of a 1024-point line on a field as
        # FilteredNoise makes it by default (a user's own relaxation loop).
        dict(name="gradient_small", op="gradient", n=1024, columns=1024, rows=1024, lines=1,
             store="fp64", length=0.0, height=0.0, model=0, force=0.0, xi=4.0),
        # The reference's own benchmark shape (n = 262144 on 262144 x 64,
        # Lx = 256, Ly = 1, arclength, f = 0.1), default store.
        dict(name="gradient_reference_shape", op="gradient", n=262144, columns=262144, rows=64,
             lines=1, store="fp64", length=256.0, height=1.0, model=1, force=0.1, xi=4.0),
        # Odd sizes: lines that do not share the field's columns, spacings that
        # are no powers of two, three lines in one call.
        dict(name="gradient_ragged", op="gradient", n=100003, columns=65537, rows=77, lines=3,
             store="fp64", length=250.0, height=1.0, model=0, force=0.3, xi=4.0),
        # The largest gather: 8 lines of 2^20 points, FP64 on the
        # cell-polynomial store (the benchmark's headline call).
        dict(name="gradient_store_batch", op="gradient", n=1 << 20, columns=1 << 20, rows=64,
             lines=8, store="poly", length=0.0, height=0.0, model=0, force=0.0, xi=4.0),
        # The same lines on FP32 split heights and the x-filtered store.
        dict(name="gradient_split_batch", op="gradient", n=1 << 20, columns=1 << 20, rows=64,
             lines=8, store="edge", length=0.0, height=0.0, model=0, force=0.0, xi=4.0),
        # One step of a minimiser outside the library on a depinning-sized line.
        dict(name="energy_step", op="energy", n=16384, columns=16384, rows=1024, store="fp64",
             length=0.0, height=0.0, model=0, force=0.05, xi=4.0),
        # qew_static: one 4096-point line to max|g| < 1e-8.
        dict(name="lbfgs_line", op="lbfgs", n=4096, rows=512, store="fp64", model=0, xi=4.0,
             tension=1.0, m=10),
        # Ensemble statics: 768 lines of 256 to 4096 points, both models.
        dict(name="ensemble", op="ensemble", fields=192, per_field=4, n_min=256, n_max=4096,
             rows=256, store="fp64", m=10),
        # qew_dynamic: annealed Langevin, L = 65536, arclength, f = 0.5.
        dict(name="langevin_fp64", op="langevin", n=65536, rows=512, store="fp64", precision=0,
             model=1, force=0.5, steps=500, t_start=0.5, dt=0.01, xi=4.0),
        # The same on FP32 coefficients.
        dict(name="langevin_fp32", op="langevin", n=65536, rows=512, store="both", precision=1,
             model=1, force=0.5, steps=1000, t_start=0.5, dt=0.01, xi=4.0),
        # qew_depinning: sweeps of a 2048-point line below its depinning force.
        dict(name="depinning_block", op="depinning", n=2048, rows=2048, store="fp64", force=0.1,
             sweeps=200, xi=4.0),
        # A served request's field, generated on the device, and first gradients.
        dict(name="field_generated", op="field", source="generated", n=4096, rows=1024, lines=4,
             store="both", xi=4.0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed kinds and ranges."""
    op = rng.choice(["gradient", "gradient", "gradient", "energy", "lbfgs", "ensemble",
                     "langevin", "langevin", "depinning", "field"])
    xi = rng.choice([2.0, 3.0, 4.0, 6.0, 8.0])
    if op == "gradient":
        store = rng.choice(["fp64", "fp64", "poly", "edge"])
        n = _log(rng, 1024, 1 << 20)
        if rng.random() < 0.5:
            n = max(1024, n & ~63)
        rows = rng.choice([64, 77, 128, 256])
        if n * rows > 1 << 26:
            rows = 64
        unit = rng.random() < 0.5
        columns = n
        if store == "fp64" and rng.random() < 0.3:
            columns = max(512, int(n * rng.uniform(0.5, 1.0)))
        return dict(op="gradient", n=n, columns=columns, rows=rows,
                    lines=rng.choice([1, 1, 2, 3, 8]), store=store,
                    length=0.0 if unit else round(n * rng.uniform(0.001, 0.1), 3),
                    height=0.0 if unit else rng.choice([1.0, 2.5]),
                    model=rng.randint(0, 1), force=rng.choice([0.0, 0.1, 0.25]), xi=xi)
    if op == "energy":
        n = _log(rng, 1024, 262144)
        unit = rng.random() < 0.5
        return dict(op="energy", n=n, columns=n, rows=rng.choice([64, 77, 256]),
                    store=rng.choice(["fp64", "poly"]),
                    length=0.0 if unit else round(n * rng.uniform(0.001, 0.1), 3),
                    height=0.0 if unit else 1.0, model=rng.randint(0, 1),
                    force=rng.choice([0.0, 0.05]), xi=xi)
    if op == "lbfgs":
        model = rng.randint(0, 1)
        return dict(op="lbfgs", n=2 * _log(rng, 256, 4096), rows=rng.choice([256, 512]),
                    store=rng.choice(["fp64", "poly"]), model=model, xi=rng.choice([2.0, 3.0, 4.0]),
                    tension=4.0 if model else rng.choice([1.0, 2.0, 4.0]), m=rng.choice([8, 10]))
    if op == "ensemble":
        return dict(op="ensemble", fields=rng.randint(24, 192), per_field=rng.randint(1, 4),
                    n_min=256, n_max=_log(rng, 512, 4096), rows=256,
                    store=rng.choice(["fp64", "poly"]), m=rng.choice([8, 10]))
    if op == "langevin":
        precision = rng.randint(0, 1)
        n = _log(rng, 1024, 65536)
        return dict(op="langevin", n=n, rows=rng.choice([256, 512]),
                    store="both" if precision else rng.choice(["fp64", "poly"]),
                    precision=precision, model=rng.randint(0, 1), force=rng.choice([0.0, 0.5]),
                    steps=rng.randint(100, 1000), t_start=round(rng.uniform(0.0, 0.5), 3),
                    dt=0.01, xi=xi)
    if op == "depinning":
        return dict(op="depinning", n=2 * _log(rng, 256, 4096), rows=rng.choice([512, 1024]),
                    store=rng.choice(["fp64", "poly"]), force=round(rng.uniform(0.02, 0.1), 3),
                    sweeps=rng.randint(50, 200), xi=rng.choice([3.0, 4.0, 6.0]))
    return dict(op="field", source=rng.choice(["generated", "values"]), n=_log(rng, 512, 16384),
                rows=rng.choice([256, 1000, 1024]), lines=rng.choice([1, 4]),
                store=rng.choice(["both", "poly", "fp64"]), xi=xi)


# ------------------------------------------------------------------ inputs
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _values(nx, ny, xi, seed):
    """White noise of `seed`, Gaussian-filtered along both axes, unit variance."""
    w = torch.randn((nx, ny), dtype=torch.float64, device="cuda", generator=_gen(seed))
    for dim, m in ((1, ny), (0, nx)):
        k = torch.fft.rfftfreq(m, device="cuda", dtype=torch.float64)
        s = torch.exp(-0.5 * (2 * math.pi * xi * k) ** 2)
        w = torch.fft.irfft(torch.fft.rfft(w, dim=dim) * (s if dim else s[:, None]), n=m, dim=dim)
    w -= w.mean()
    return (w / w.std(unbiased=False)).contiguous()


def _lines(count, n, height, rows, seed, std_cells=3.0):
    """Rough periodic lines, each about its own mean height inside the field."""
    w = torch.randn((count, n), dtype=torch.float64, device="cuda", generator=_gen(seed + 7919))
    k = torch.fft.rfftfreq(n, device="cuda", dtype=torch.float64)
    w = torch.fft.irfft(torch.fft.rfft(w) * torch.exp(-0.5 * (2 * math.pi * 48.0 * k) ** 2), n=n)
    w *= std_cells / w.std(dim=1, unbiased=False, keepdim=True)
    at = (torch.arange(count, dtype=torch.float64, device="cuda") + 0.5)[:, None] * (rows / count)
    return ((w + at) * (height / rows)).contiguous()


def _extents(case):
    return case["length"] or float(case["columns"]), case["height"] or float(case["rows"])


def _split(h, dy):
    g = h / dy
    cell = torch.floor(g)
    return cell.to(torch.int32), (g - cell).to(torch.float32)


def prepare(case, seed):
    seed, op = int(seed), case["op"]
    if op in ("gradient", "energy"):
        Lx, Ly = _extents(case)
        v = _values(case["columns"], case["rows"], case["xi"], seed)
        s = {"op": op, "field": Q.FilteredNoise(v, Lx, Ly, store=STORES[case["store"]]),
             "p": Q.Params(Lx, 1.0, case["force"], Q.Model(case["model"]))}
        h = _lines(case.get("lines", 1), case["n"], Ly, case["rows"], seed)
        if op == "energy":
            s["h"] = h[0].contiguous()
            s["d"] = 0.01 * Ly / case["rows"] * torch.randn(
                case["n"], dtype=torch.float64, device="cuda", generator=_gen(seed + 5))
        elif case["store"] == "edge":
            s["cells"], s["fracs"] = _split(h, Ly / case["rows"])
        else:
            s["h"] = h if case["lines"] > 1 else h[0].contiguous()
        return s
    if op == "ensemble":
        work = []
        for k in range(case["fields"]):  # lengths, xi and models spread over their ranges
            u, v = (0.5 + 0.6180339887 * k) % 1.0, (0.25 + 0.7548776662 * k) % 1.0
            n = 2 * int(round(0.5 * case["n_min"] * (case["n_max"] / case["n_min"]) ** u))
            xi = 2.0 + 2.0 * v
            f = Q.FilteredNoise.generated(n, case["rows"], float(n), float(case["rows"]), 1.0, xi,
                                          xi, 30000 + 1000 * (seed % 1000000) + k,
                                          store=STORES[case["store"]])
            p = Q.Params(float(n), 4.0 if k % 2 else 1.0, 0.0, Q.Model(k % 2))
            for j in range(case["per_field"]):
                h0 = torch.full((n,), case["rows"] * (j + 0.5) / case["per_field"],
                                dtype=torch.float64, device="cuda")
                work.append((h0, p, f, 0.5 / xi ** 2))
        return {"op": op, "work": work,
                "lp": Q.LbfgsParams(m=case["m"], ftol=1e-8, max_iter=20000, precondition=True,
                                    ls_fallback=True)}
    n, rows, xi = case["n"], case["rows"], case["xi"]
    if op == "field":
        s = {"op": op, "case": dict(case), "seed": seed,
             "h": _lines(case["lines"], n, float(rows), rows, seed),
             "p": Q.Params(float(n), 1.0, 0.0, Q.Model.Linear)}
        if case["source"] == "values":
            s["values"] = _values(n, rows, xi, seed)
        return s
    s = {"op": op, "case": dict(case), "seed": seed,
         "field": Q.FilteredNoise(_values(n, rows, xi, seed), float(n), float(rows),
                                  store=STORES[case["store"]]),
         "h0": torch.full((n,), 0.5 * rows, dtype=torch.float64, device="cuda")}
    if op == "lbfgs":
        s["p"] = Q.Params(float(n), case["tension"], 0.0, Q.Model(case["model"]))
        s["lp"] = Q.LbfgsParams(m=case["m"], ftol=1e-8, max_iter=20000, precondition=True,
                                precond_shift=0.5 / xi ** 2, ls_fallback=True)
    elif op == "langevin":
        s["p"] = Q.Params(float(n), 1.0, case["force"], Q.Model(case["model"]))
        s["drift"], s["diff"] = _schedule(case)
    else:
        s["p"] = Q.Params(float(n), 1.0, case["force"], Q.Model.Linear)
        s["rp"] = Q.RkParams(dstep=0.5, max_advance=float(rows), root_tol=1e-10, sweep_tol=1e-8,
                             runaway=2.0 * rows, max_sweeps=case["sweeps"])
    return s


def _schedule(case):
    k, dt = case["steps"], case["dt"]
    t = case["t_start"] * (1.0 - np.arange(k) / k)
    return np.full(k, dt), np.sqrt(2.0 * t * dt)


# -------------------------------------------------------------------- calls
def run(s):
    op = s["op"]
    if op == "gradient":
        if "cells" in s:
            return Q.gradient_split_batch(s["cells"], s["fracs"], s["p"], s["field"])
        if s["h"].dim() == 2:
            return Q.gradient_batch(s["h"], s["p"], s["field"])
        return Q.gradient(s["h"], s["p"], s["field"])
    if op == "energy":
        e = Q.objective(s["h"], s["p"], s["field"])
        t = Q.objective_trial(s["h"], s["d"], 0.5, s["p"], s["field"])
        return e, t, Q.gradient(s["h"], s["p"], s["field"])
    if op == "ensemble":
        lines = [(h0.clone(), p, f, shift) for h0, p, f, shift in s["work"]]
        r = Q.ensemble_minimize(lines, s["lp"])
        return torch.cat([h for h, _, _, _ in lines]), sum(int(x.converged) for x in r)
    if op == "field":
        c = s["case"]
        n, rows = c["n"], c["rows"]
        if c["source"] == "generated":
            f = Q.FilteredNoise.generated(n, rows, float(n), float(rows), 1.0, c["xi"], c["xi"],
                                          s["seed"], store=STORES[c["store"]])
        else:
            f = Q.FilteredNoise(s["values"], float(n), float(rows), store=STORES[c["store"]])
        return Q.gradient_batch(s["h"], s["p"], f)
    h = s["h0"].clone()
    if op == "lbfgs":
        r = Q.lbfgs_minimize(h, s["p"], s["field"], s["lp"])
        return h, int(r.converged)
    if op == "langevin":
        dyn = Q.LangevinDynamics(h.numel(), s["seed"])
        dyn.run(h, s["p"], s["field"], s["drift"], s["diff"], precision=s["case"]["precision"])
        return h
    r = Q.rk_block(h, s["p"], s["field"], s["rp"])
    return h, r.mean_h


# --------------------------------------------------------------------- work
def work(case):
    """Per line point: the height in, the gradient out, the four field values
    of its edge's column that the gather cannot do without, and the sums of
    that gather (20 multiply-adds) and of the site."""
    op = case["op"]
    if op == "gradient":
        pts = case["n"] * case["lines"]
        return {"bytes": pts * (28 if case["store"] == "edge" else 48), "flops": pts * 56}
    if op == "energy":
        return {"bytes": case["n"] * (40 + 56 + 48), "flops": case["n"] * 3 * 56}
    if op == "lbfgs":
        # about 60 iterations of a gather, an energy and 4 m vector products
        return {"bytes": 60 * case["n"] * (88 + 16 * case["m"]),
                "flops": 60 * case["n"] * (112 + 8 * case["m"])}
    if op == "ensemble":
        mean = (case["n_max"] - case["n_min"]) / math.log(case["n_max"] / case["n_min"])
        pts = case["fields"] * case["per_field"] * mean
        return {"bytes": 80 * pts * (44 + 8 * case["m"]), "flops": 80 * pts * (112 + 8 * case["m"])}
    if op == "langevin":
        return {"bytes": case["steps"] * case["n"] * (32 if case["precision"] else 48),
                "flops": case["steps"] * case["n"] * 100}
    if op == "depinning":
        return {"bytes": case["sweeps"] * case["n"] * 80, "flops": case["sweeps"] * case["n"] * 120}
    cells, taps = case["n"] * case["rows"], 2 * math.ceil(5 * case["xi"]) + 1
    generated = case["source"] == "generated"
    per = {"both": 12, "poly": 40, "fp64": 8}[case["store"]] + (0 if generated else 8)
    return {"bytes": cells * per, "flops": cells * (20 + (4 * taps if generated else 0))}


# ------------------------------------------------------- the same in 64 bits
def _coefficients(v):
    nx, ny = v.shape
    kx = 2 / 3 + torch.cos(2 * math.pi * torch.arange(nx, device="cuda", dtype=torch.float64) / nx) / 3
    ky = 2 / 3 + torch.cos(2 * math.pi * torch.arange(ny // 2 + 1, device="cuda",
                                                      dtype=torch.float64) / ny) / 3
    return torch.fft.irfft2(torch.fft.rfft2(v) / (kx[:, None] * ky[None, :]), s=(nx, ny))


def _weights(t, deriv):
    o = 1 - t
    if deriv:
        return (-0.5 * o * o, -2 * t + 1.5 * t * t, 0.5 + t - 1.5 * t * t, 0.5 * t * t)
    return (o ** 3 / 6, (4 - 6 * t * t + 3 * t ** 3) / 6, (1 + 3 * t + 3 * t * t - 3 * t ** 3) / 6,
            t ** 3 / 6)


def _gather(coef, Lx, Ly, x, y, deriv):
    """V (or dV/dy) of the periodic bicubic B-spline at the points (x, y)."""
    nx, ny = coef.shape
    gx, gy = x / (Lx / nx), y / (Ly / ny)
    ix, iy = torch.floor(gx), torch.floor(gy)
    wx, wy = _weights(gx - ix, False), _weights(gy - iy, deriv)
    ix, iy = ix.long(), iy.long()
    flat, out = coef.reshape(-1), 0.0
    for a in range(4):
        col = torch.remainder(ix + a - 1, nx) * ny
        out = out + wx[a] * sum(wy[b] * flat[col + torch.remainder(iy + b - 1, ny)]
                                for b in range(4))
    return out / (Ly / ny) if deriv else out


def _edge_x(n, dx):
    i = torch.arange(n, device="cuda", dtype=torch.float64)
    ip = torch.roll(i, -1)  # the last edge's right end is site 0
    return (i + ip) * 0.5 * dx


def _gradient(coef, Lx, Ly, h, tension, force, model):
    n = h.numel()
    dx = Lx / n
    hp, hm = torch.roll(h, -1), torch.roll(h, 1)
    dv = _gather(coef, Lx, Ly, _edge_x(n, dx), 0.5 * (h + hp), True)
    if model:
        s = (hp - h) / dx
        s = s / torch.sqrt(1 + s * s)
        el = tension * (torch.roll(s, 1) - s) / dx
    else:
        el = -tension * ((hm - h) + (hp - h)) / (dx * dx)
    return dx * (el + 0.5 * (torch.roll(dv, 1) + dv) - force)


def _energy(coef, Lx, Ly, h, tension, force, model):
    n = h.numel()
    dx = Lx / n
    hp = torch.roll(h, -1)
    s = (hp - h) / dx
    el = tension * (torch.sqrt(1 + s * s) - 1) if model else 0.5 * tension * s * s
    v = _gather(coef, Lx, Ly, _edge_x(n, dx), 0.5 * (h + hp), False)
    return float((dx * (el + v - force * h)).sum())


def _mulhilo(m, c):
    """High and low 32 bits of m * c for a constant m < 2^32 and c < 2^32."""
    lo, hi = c * (m & 0xFFFF), c * (m >> 16)
    total = (lo >> 16) + hi  # bits 16 and up
    return total >> 16, ((total & 0xFFFF) << 16) | (lo & 0xFFFF)


def _normals(seed, step, pairs):
    """The library's counter stream: Philox4x32-10 of (pair, 0, step), key seed, Box-Muller.
    step and pairs broadcast; the last axis holds the two normals of a pair."""
    mask = 0xFFFFFFFF
    step, pairs = torch.broadcast_tensors(step, pairs)
    c = [pairs, torch.zeros_like(pairs), step & mask, step >> 32]
    k0, k1 = seed & mask, (seed >> 32) & mask
    for r in range(10):
        if r:
            k0, k1 = (k0 + 0x9E3779B9) & mask, (k1 + 0xBB67AE85) & mask
        h0, l0 = _mulhilo(0xD2511F53, c[0])
        h1, l1 = _mulhilo(0xCD9E8D57, c[2])
        c = [h1 ^ c[1] ^ k0, l1, h0 ^ c[3] ^ k1, l0]
    u1 = (((c[0] << 21) | (c[1] >> 11)).double() + 1.0) * 2.0 ** -53
    u2 = ((c[2] << 21) | (c[3] >> 11)).double() * 2.0 ** -53
    r = torch.sqrt(-2.0 * torch.log(u1))
    return torch.stack((r * torch.cos(2 * math.pi * u2), r * torch.sin(2 * math.pi * u2)), dim=-1)


def _generated(nx, ny, xi, seed):
    i = torch.arange(nx, device="cuda")[:, None]
    j = torch.arange((ny + 1) // 2, device="cuda")[None, :]
    w = _normals(seed, i, j).reshape(nx, -1)[:, :ny].contiguous()
    R = math.ceil(5 * xi)
    k = torch.arange(-R, R + 1, dtype=torch.float64)
    t = torch.exp(-0.5 * k * k / (xi * xi))
    t = (t / torch.sqrt((t * t).sum())).tolist()
    for dim in (1, 0):
        w = sum(t[m + R] * torch.roll(w, -m, dims=dim) for m in range(-R, R + 1))
    return w / w.std(unbiased=False)


def exact(case, seed):
    seed, op = int(seed), case["op"]
    if op in ("gradient", "energy"):
        Lx, Ly = _extents(case)
        coef = _coefficients(_values(case["columns"], case["rows"], case["xi"], seed))
        h = _lines(case.get("lines", 1), case["n"], Ly, case["rows"], seed)
        a = (1.0, case["force"], case["model"])
        if op == "energy":
            d = 0.01 * Ly / case["rows"] * torch.randn(
                case["n"], dtype=torch.float64, device="cuda", generator=_gen(seed + 5))
            return (_energy(coef, Lx, Ly, h[0], *a), _energy(coef, Lx, Ly, h[0] + 0.5 * d, *a),
                    _gradient(coef, Lx, Ly, h[0], *a))
        if case["store"] == "edge":
            cell, frac = _split(h, Ly / case["rows"])
            h = (cell.double() + frac.double()) * (Ly / case["rows"])
        g = torch.stack([_gradient(coef, Lx, Ly, x, *a) for x in h])
        return g if case["lines"] > 1 or case["store"] == "edge" else g[0]
    if op == "langevin":
        n, rows = case["n"], case["rows"]
        coef = _coefficients(_values(n, rows, case["xi"], seed))
        h = torch.full((n,), 0.5 * rows, dtype=torch.float64, device="cuda")
        j, step = torch.arange((n + 1) // 2, device="cuda"), 0
        for a, b in zip(*_schedule(case)):
            g = _gradient(coef, float(n), float(rows), h, 1.0, case["force"], case["model"])
            h = h - a * g
            if b > 0:
                at = torch.full((1,), step, dtype=torch.int64, device="cuda")
                h += b * _normals(seed, at, j).reshape(-1)[:n]
                step += 1
        return h
    if op == "field":
        n, rows = case["n"], case["rows"]
        v = _generated(n, rows, case["xi"], seed) if case["source"] == "generated" else \
            _values(n, rows, case["xi"], seed)
        coef = _coefficients(v)
        return torch.stack([_gradient(coef, float(n), float(rows), h, 1.0, 0.0, 0)
                            for h in _lines(case["lines"], n, float(rows), rows, seed)])
    return None  # a relaxed or swept line: no closed form
