"""Work that users of the engine have it do, through its public Python entry points.

Two families. The plain simulator turns an initial fluorescence histogram and a set of cell
types into the output histogram: one call with host data in and out (Engine.simulate), a
prepared plan run again (Engine.plan), many uneven inputs in one call
(Engine.simulate_batch) and a prepared batch whose types change between runs (Engine.batch,
the inner step of a parameter search). The smoothed form gives expected counts and their
derivatives for many candidate parameter sets at once (procell.smooth), the inner step of a
calibration.

Inputs are seeded and synthetic, with the value distributions of procell/configs.py and
procell/calibrate.py: fluorescence log-uniform, cells spread over the bins by a Poisson or
multinomial law, division times of tens of hours with a spread of 10 to 40%.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cuda-pro-cell_gb300"))
from procell import Engine  # noqa: E402
from procell.smooth import Smooth, expected_counts  # noqa: E402

_ENGINE = []


def engine():
    """The process's one engine (a program keeps it for its lifetime)."""
    if not _ENGINE:
        _ENGINE.append(Engine(0))
    return _ENGINE[0]


# ---------------------------------------------------------------------------- cases --

def _sim(name, path, bins, cells, top, types, quiescent, mean, t_max, phi):
    """Plain simulator: `cells` initial cells in `bins` bins of fluorescence log-uniform on
    [1, top], `types` proliferating types of mean division time U[0.85, 1.15] x mean (and a
    quiescent one), simulated to t_max; phi 0 is the automatic threshold."""
    c = {"path": path, "bins": bins, "cells": cells, "top": float(top), "types": types, "quiescent": quiescent,
         "mean": float(mean), "t_max": float(t_max), "phi": float(phi)}
    return dict(c, name=name) if name else c


def _smo(name, path, bins, cells, top, types, candidates, paths, t_max):
    """Smoothed form: `candidates` parameter sets on one histogram, `paths` sampled lineages
    per initial cell."""
    c = {"path": path, "bins": bins, "cells": cells, "top": float(top), "types": types, "candidates": candidates,
         "paths": paths, "t_max": float(t_max)}
    return dict(c, name=name) if name else c


def listed():
    return [
        # one small measurement (1e4 events, two types, a week): an interactive call, where the
        # fixed cost of a call counts
        _sim("small_simulate", "simulate", 64, 9600, 1e4, 2, False, 67.0, 168.0, 0.0),
        # an ordinary measurement: 1e6 events, two weeks, a quiescent fraction, a stated phi
        _sim("medium_simulate", "simulate", 1024, 1024000, 1e5, 3, True, 63.0, 336.0, 4.0),
        # the largest: 1e7 events followed for two weeks, billions of divisions
        _sim("large_simulate", "simulate", 4096, 10240000, 1e6, 5, False, 37.0, 336.0, 1.0),
        # a few sorted bright cells followed for three weeks: few initial cells, deep trees
        _sim("few_deep_cells", "simulate", 23, 611, 1e6, 2, False, 40.0, 504.0, 1.0),
        # an unbinned export, nearly every event its own row, prepared once and run again (as
        # under several thresholds of a viewer): many ragged bins of one to a few cells
        _sim("unbinned_rerun", "rerun", 20011, 50003, 1e4, 4, True, 55.0, 240.0, 0.0),
        # a plate of uneven samples in one call, host data in and out
        {"name": "uneven_batch", "path": "batch", "instances": 160, "cells_lo": 1000, "cells_hi": 300000, "bins_hi": 1024,
         "top": 1e4, "t_lo": 48.0, "t_hi": 336.0},
        # one iteration of a gradient-free search: 256 candidate type sets on one histogram, as a
        # prepared batch with its types replaced, run, and all totals read
        {"name": "search_step", "path": "search", "candidates": 256, "bins": 256, "cells": 100000, "top": 1e4, "types": 3,
         "t_max": 168.0},
        # scoring a swarm on the smoothed form (forward only)
        _smo("smooth_forward", "smooth_forward", 256, 100000, 1e4, 3, 256, 2, 168.0),
        # one gradient-descent step of a calibration: expected counts, log loss, adjoint
        _smo("smooth_step", "smooth_step", 256, 100000, 1e4, 3, 256, 2, 168.0),
        # the same for a handful of candidates on a smaller histogram
        _smo("smooth_step_few", "smooth_step", 101, 20011, 1e4, 2, 5, 1, 168.0),
        # sensitivities of the expected counts for a report: odd sizes
        _smo("smooth_jacobian", "smooth_jacobian", 97, 30011, 1e4, 2, 37, 2, 192.0),
        # one Levenberg-Marquardt iteration's system for every candidate
        _smo("gauss_newton", "gauss_newton", 256, 100000, 1e4, 3, 256, 2, 168.0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["simulate", "simulate", "simulate", "rerun", "batch", "search", "smooth_forward", "smooth_step",
                       "smooth_jacobian", "gauss_newton"])
    if kind in ("simulate", "rerun"):
        while True:
            cells = _log(rng, 300, 1e7)
            bins = _log(rng, 8, min(20000, max(9, cells // 2)))
            c = _sim(None, kind, bins, cells, 10.0 ** rng.uniform(3.5, 6.0), rng.randint(1, 6), rng.random() < 0.3,
                     rng.uniform(35.0, 80.0), rng.uniform(72.0, 504.0), rng.choice([0.0, 1.0, 4.0]))
            if _divisions(c) <= 2e9:
                return c
    if kind == "batch":
        return {"path": "batch", "instances": _log(rng, 8, 400), "cells_lo": 1000, "cells_hi": _log(rng, 5000, 300000),
                "bins_hi": rng.randint(48, 1024), "top": 1e4, "t_lo": 48.0, "t_hi": rng.uniform(120.0, 336.0)}
    if kind == "search":
        return {"path": "search", "candidates": _log(rng, 16, 300), "bins": _log(rng, 32, 512), "cells": _log(rng, 5000, 100000),
                "top": 1e4, "types": rng.randint(1, 4), "t_max": rng.uniform(96.0, 200.0)}
    return _smo(None, kind, _log(rng, 32, 300), _log(rng, 5000, 100000), 10.0 ** rng.uniform(3.5, 4.5), rng.randint(1, 4),
                _log(rng, 3, 256), rng.randint(1, 2), rng.uniform(96.0, 240.0))


# --------------------------------------------------------------------------- inputs --

def _channels(bins, top, which=0):
    """Fluorescence of an instrument's channels: the same for every measurement made on it."""
    return np.exp(np.random.default_rng([bins, which]).uniform(0.0, math.log(top), bins))


def _histogram(rng, bins, cells, top):
    """A measurement: every channel listed has at least one cell."""
    freq = 1 + rng.multinomial(max(0, cells - bins), np.full(bins, 1.0 / bins))
    return _channels(bins, top), freq.astype(np.uint64)


def _ratios(rng, n):
    r = rng.dirichlet(np.ones(n))
    return r / r.sum()


def _types(rng, n, quiescent, mean, cv=(0.1, 0.4)):
    r = _ratios(rng, n + int(quiescent))
    rows = []
    for i in range(n):
        m = float(rng.uniform(0.85, 1.15) * mean)
        rows.append((float(r[i]), m, float(rng.uniform(*cv) * m)))
    if quiescent:
        rows.append((float(r[n]), -1.0, -1.0))
    return rows


def _candidates(rng, n, types):
    """Candidate (ratio, mean, sd) sets, uniform in the search box of a calibration."""
    ratio = np.stack([_ratios(rng, types) for _ in range(n)])
    mean = rng.uniform(25.0, 110.0, (n, types))
    return np.stack([ratio, mean, mean * rng.uniform(0.08, 0.45, (n, types))], axis=-1)


def _instances(case, rng):
    """A plate: the layout (channels, sizes, number of types, durations) is the case's, the
    cells and the types' parameters the seed's."""
    plate, out = np.random.default_rng(case["instances"]), []
    for i in range(case["instances"]):
        bins = int(plate.integers(32, case["bins_hi"] + 1))
        cells = int(round(math.exp(plate.uniform(math.log(case["cells_lo"]), math.log(case["cells_hi"])))))
        n, quiescent, t_max = int(plate.integers(1, 5)), bool(plate.random() < 0.2), float(plate.uniform(case["t_lo"], case["t_hi"]))
        freq = 1 + rng.multinomial(max(0, cells - bins), rng.dirichlet(np.ones(bins)))
        types = _types(rng, n, quiescent, float(plate.uniform(50.0, 90.0)))
        out.append(((_channels(bins, case["top"], i), freq.astype(np.uint64)), types, t_max, None, int(rng.integers(1 << 40))))
    return out


def _smooth_inputs(case, seed):
    rng = np.random.default_rng(seed)
    values, freq = _histogram(rng, case["bins"], case["cells"], case["top"])
    phi = float(values[freq > 0].min())
    params = _candidates(rng, case["candidates"], case["types"])
    target = rng.lognormal(4.0, 1.5, 65536)  # as many of these counts as there are output values
    return values, freq, phi, params, target, int(rng.integers(1 << 40))


def prepare(case, seed):
    path, rng = case["path"], np.random.default_rng(seed)
    s = {"path": path, "engine": engine()}
    if path in ("simulate", "rerun"):
        hist = _histogram(rng, case["bins"], case["cells"], case["top"])
        types = _types(rng, case["types"], case["quiescent"], case["mean"])
        s["input"] = (hist, types, case["t_max"], case["phi"] or None, int(rng.integers(1 << 40)))
        if path == "rerun":
            s["plan"] = s["engine"].plan(*s["input"])
    elif path == "batch":
        s["instances"] = _instances(case, rng)
    elif path == "search":
        hist = _histogram(rng, case["bins"], case["cells"], case["top"])
        first = [(1.0 / case["types"], 60.0, 12.0)] * case["types"]
        key = int(rng.integers(1 << 40))
        rows = _candidates(rng, case["candidates"], case["types"]).reshape(-1, 3)
        s["batch"] = s["engine"].batch([(hist, first, case["t_max"], None, key)] * case["candidates"])
        s["types"] = np.empty(case["candidates"] * case["types"], [("ratio", "<f8"), ("mean", "<f8"), ("sd", "<f8")])
        for i, field in enumerate(("ratio", "mean", "sd")):
            s["types"][field] = rows[:, i]
    else:
        values, freq, phi, params, target, key = _smooth_inputs(case, seed)
        s["smooth"] = Smooth(s["engine"], (values, freq), case["types"], case["t_max"], phi, h=0.5, paths=case["paths"], seed=key)
        s["params"] = torch.tensor(params, device="cuda")
        s["target"] = torch.tensor(np.sort(target[:s["smooth"].n_values]), device="cuda")
    return s


def run(state):
    path = state["path"]
    if path == "simulate":
        r = state["engine"].simulate(*state["input"])
        return {"values": r.values, "totals": r.totals, "per_type": r.per_type}
    if path == "rerun":
        state["plan"].run()
        r = state["plan"].result()
        return {"values": r.values, "totals": r.totals, "per_type": r.per_type}
    if path == "batch":
        rs = state["engine"].simulate_batch(state["instances"])
        return {"values": np.concatenate([r.values for r in rs]), "totals": np.concatenate([r.totals for r in rs]),
                "per_type": np.concatenate([r.per_type.ravel() for r in rs])}
    if path == "search":
        state["batch"].set_types(state["types"])
        state["batch"].run()
        offsets, totals = state["batch"].totals()
        return {"offsets": offsets, "totals": totals}
    sm, p = state["smooth"], state["params"]
    if path == "smooth_forward":
        return {"expected": sm.forward(p)}
    if path == "smooth_step":
        q = p.clone().requires_grad_(True)
        e = expected_counts(sm, q)
        loss = ((torch.log1p(e) - torch.log1p(state["target"])) ** 2).sum(dim=1)
        loss.sum().backward()
        return {"expected": e.detach(), "loss": loss.detach(), "grad": q.grad}
    if path == "smooth_jacobian":
        e, j = sm.jacobian(p)
        return {"expected": e, "jacobian": j}
    loss, jtj, jtr = sm.gauss_newton(p, state["target"])
    return {"loss": loss, "jtj": jtj, "jtr": jtr}


# ----------------------------------------------------------------------------- work --

def _phi_generations(top, phi):
    """Mean number of generations the threshold allows for values log-uniform on [1, top]."""
    lo = max(phi, 1.0)
    return np.maximum(np.log2(np.geomspace(1.0, top, 64) / lo), 0.0)


def _divisions_per_cell(mean, cv, t_max, caps):
    """Expected divisions of one initial cell (normal division times, age U x the first)."""
    u = (np.arange(16) + 0.5) / 16
    total, reach = np.zeros(len(caps)), int(min(40, caps.max() if len(caps) else 0)) + 1
    for g in range(reach):
        z = (t_max - (1.0 + u + g) * mean) / (cv * mean * np.sqrt((1.0 + u) ** 2 + g))
        total += (caps > g) * 2.0 ** g * np.mean([0.5 * math.erfc(-x / math.sqrt(2.0)) for x in z])
    return float(total.mean())


def _divisions(case):
    if case["path"] in ("simulate", "rerun"):
        caps = _phi_generations(case["top"], case["phi"])
        share = case["types"] / (case["types"] + case["quiescent"])
        return case["cells"] * share * np.mean([_divisions_per_cell(case["mean"] * f, 0.25, case["t_max"], caps)
                                                for f in (0.87, 0.95, 1.0, 1.05, 1.13)])
    caps = _phi_generations(case["top"], 1.0)
    if case["path"] == "batch":
        lo, hi = case["cells_lo"], case["cells_hi"]
        cells = case["instances"] * ((hi - lo) / math.log(hi / lo) if hi > lo else lo)
        times = np.linspace(case["t_lo"], case["t_hi"], 5)
        return cells * np.mean([_divisions_per_cell(70.0 * f, 0.25, t, caps) for t in times for f in (0.8, 1.0, 1.2)])
    return case["candidates"] * case["cells"] * np.mean([_divisions_per_cell(m, 0.26, case["t_max"], caps)
                                                         for m in (35.0, 60.0, 90.0)])


def work(case):
    """Plain form: the histogram and types in, the output histogram out; a division is two
    daughters, each with a counter-based random word (half of a ten-round Philox block, about
    30 operations), a normal draw and a due time (about 15). Smoothed form: parameters in,
    results out; a lineage step is a remaining time, a sigmoid pair, a leaf weight (about 25
    operations) and for derivatives their tangents (about 12)."""
    if "candidates" in case and case["path"] != "search":
        chain = float(np.mean(np.floor(_phi_generations(case["top"], 1.0)) + 1.0))
        values, c, k = case["bins"] * chain, case["candidates"], case["types"]
        reached = min(chain, 1.0 + case["t_max"] / 60.0)
        steps = case["cells"] * case["paths"] * c * k * reached
        out = {"smooth_forward": c * values, "smooth_step": c * (2 * values + 3 * k), "smooth_jacobian": c * values * (1 + 3 * k),
               "gauss_newton": c * (1 + 9 * k * k + 3 * k)}[case["path"]]
        per = {"smooth_forward": 25, "smooth_step": 62, "smooth_jacobian": 37, "gauss_newton": 37}[case["path"]]
        more = values * c * (3 * k) ** 2 if case["path"] == "gauss_newton" else 0.0
        return {"bytes": 16.0 * case["bins"] + 8.0 * (3 * k * c + out), "flops": steps * per + more}
    if case["path"] == "batch":
        bins, types, n = 0.5 * (32 + case["bins_hi"]), 2.7, case["instances"]
        chain = float(np.mean(np.floor(_phi_generations(case["top"], 1.0)) + 1.0))
        moved = n * (16.0 * bins + 24.0 * types + bins * chain * 8.0 * (2 + types))
    elif case["path"] == "search":
        chain = float(np.mean(np.floor(_phi_generations(case["top"], 1.0)) + 1.0))
        moved = case["candidates"] * (24.0 * case["types"] + 8.0 * case["bins"] * chain) + 16.0 * case["bins"]
    else:
        chain = float(np.mean(np.floor(_phi_generations(case["top"], case["phi"])) + 1.0))
        k = case["types"] + case["quiescent"]
        moved = 16.0 * case["bins"] + 24.0 * k + 8.0 * case["bins"] * chain * (2 + k)
    return {"bytes": float(moved), "flops": 90.0 * float(_divisions(case))}


# ---------------------------------------------------------------------------- exact --

def _value_set(values, freq, phi):
    out = []
    cur = np.asarray(values, np.float64)[np.asarray(freq) > 0]
    phi = float(cur.min()) if phi is None else phi
    while (cur := cur[cur >= phi]).size:
        out.append(cur)
        cur = cur / 2
    return np.unique(np.concatenate(out)) if out else np.zeros(0)


M32 = 0xFFFFFFFF


def _philox(c0, c1, c2, c3, k0, k1):
    """Philox4x32-10 (Salmon et al. 2011) on int64 tensors of 32-bit words (or on ints)."""
    def mul(a, b):  # 32 x 32 -> (high, low) without leaving 63 bits
        lo, mid = (a & 0xFFFF) * b, (a >> 16) * b
        mid = mid + (lo >> 16)
        return (mid >> 16) & M32, ((mid << 16) | (lo & 0xFFFF)) & M32
    for _ in range(10):
        h0, l0 = mul(0xD2511F53, c0)
        h1, l1 = mul(0xCD9E8D57, c2)
        c0, c1, c2, c3 = h1 ^ c1 ^ k0, l1, h0 ^ c3 ^ k1, l0
        k0, k1 = (k0 + 0x9E3779B9) & M32, (k1 + 0xBB67AE85) & M32
    return c0, c1, c2, c3


def _ziggurat():
    """1024-layer normal ziggurat (Marsaglia & Tsang 2000): r closes the construction, v is
    the area of a layer."""
    n, r, v = 1024, 4.0388498461095045227, 1.2263246463530880729e-3
    x = [0.0, r]
    for _ in range(n - 2):
        x.append(math.sqrt(-2.0 * math.log(v / x[-1] + math.exp(-0.5 * x[-1] ** 2))))
    x.append(0.0)
    base = v / math.exp(-0.5 * r * r)
    k = [math.floor(r / base * 2.0 ** 31)] + [math.floor(x[i + 1] / x[i] * 2.0 ** 31) for i in range(1, n)]
    w = np.array([base] + x[1:n]) / 2.0 ** 31
    f = [0.0] + [math.exp(-0.5 * x[i] ** 2) for i in range(1, n)] + [1.0]
    return k, w.astype(np.float32), f, r


def _rejected(j, layer, wedge, node, root, k0, k1, tab):
    """The rare draws that the strip test does not settle, one at a time."""
    k, w, f, r = tab
    words, block = [], 0

    def word():
        nonlocal block
        if not words:
            words.extend(_philox(node & M32, node >> 32, root, 0x20000000 | block, k0, k1))
            block += 1
        return words.pop(0)
    first = True
    while True:
        mag, sign = j & 0x7FFFFFFF, -1.0 if j >> 31 else 1.0
        x = float(np.float32(mag) * w[layer])
        if mag < k[layer]:
            return sign * x
        if layer == 0:
            while True:
                a = -math.log(((word() >> 8) + 1) / 2.0 ** 24) / r
                b = -math.log(((word() >> 8) + 1) / 2.0 ** 24)
                if 2 * b > a * a:
                    return sign * (r + a)
        u = ((wedge if first else word()) >> 8) / 2.0 ** 24
        if f[layer] + u * (f[layer + 1] - f[layer]) < math.exp(-0.5 * x * x):
            return sign * x
        first = False
        j, layer = word(), word() & 1023


def _lineages(root, steps, seed):
    """Initial age U [L] and normals z [L, steps] of one sampled lineage per root index."""
    dev = root.device
    k0, k1 = seed & M32, seed >> 32
    zero = torch.zeros_like(root)
    R = _philox(zero, zero, root, zero + 0x30000000, k0, k1)
    u = (((R[2] << 21) | (R[3] >> 11)) + 1).double() * 2.0 ** -53
    B = _philox(zero, zero, root, zero + 0x40000000, k0, k1)
    bits = B[0] | (B[1] << 32)
    tab = _ziggurat()
    k, w = torch.tensor(tab[0], device=dev), torch.tensor(tab[1], device=dev)
    node, z = torch.ones_like(root), torch.zeros(len(root), steps, dtype=torch.float64, device=dev)
    for g in range(steps):
        parent, c = node >> 1, node & 1
        P = _philox(parent & M32, parent >> 32, root, zero + 0x10000000, k0, k1)
        j = torch.where(c == 1, P[1], P[0])
        layer = (P[2] >> (10 * c)) & 1023
        wedge = torch.where(c == 1, ((P[3] >> 22) << 22) | (((P[2] >> 20) << 10) & M32), (P[3] << 10) & M32)
        mag = j & 0x7FFFFFFF
        x = (mag.float() * w[layer]).double()  # the draw itself is an FP32 number
        z[:, g] = torch.where((j >> 31) == 1, -x, x)
        bad = torch.nonzero(mag >= k[layer])[:, 0]
        rows = torch.stack([j[bad], layer[bad], wedge[bad], node[bad], root[bad]], 1).tolist()
        if rows:
            z[bad, g] = torch.tensor([_rejected(*r, k0, k1, tab) for r in rows], dtype=torch.float64, device=dev)
        node = 2 * node + ((bits >> g) & 1)
    return u, z


def _smooth_exact(case, seed):
    """Expected counts E [C, V] and their Jacobian [C, V, K, 3] in FP64: along each sampled
    lineage s_j = sigmoid((T - S_j) / h), a generation-g leaf weighs s_1 ... s_g (1 - s_{g+1})
    and stands for 2^g cells."""
    values, freq, phi, params, _, key = _smooth_inputs(case, seed)
    T, h, paths, C, K = case["t_max"], 0.5, case["paths"], case["candidates"], case["types"]
    keep = freq > 0
    v, f = values[keep], freq[keep].astype(np.int64)
    ncells, out = int(f.sum()), _value_set(values, freq, phi)
    chain = np.zeros(len(v), np.int64)  # divisions the threshold allows
    cur = v.copy()
    while (ok := cur / 2 > phi).any():
        chain[ok] += 1
        cur = np.where(ok, cur / 2, 0.0)
    rows = int(chain.max()) + 1
    # (bin, generation) -> output value, and the value set's own length for none
    vidx = np.full((len(v), rows), len(out))
    for b in range(len(v)):
        for g in range(int(chain[b]) + 1):
            x = v[b] / 2.0 ** g
            if x >= phi:
                vidx[b, g] = int(np.searchsorted(out, x))
    dev = torch.device("cuda")
    cell_bin = torch.tensor(np.repeat(np.arange(len(v)), f), device=dev)
    lin_bin = cell_bin.repeat_interleave(paths)
    lin = torch.arange(ncells * paths, device=dev)
    u, z = _lineages(lin // paths + (lin % paths) * ncells, rows, key)
    cap = torch.tensor(chain, device=dev)[lin_bin]
    vmap = torch.tensor(vidx, device=dev)
    P = torch.tensor(params, device=dev)
    acc = torch.zeros(K, 3, len(out) + 1, C, dtype=torch.float64, device=dev)
    step = max(1, (1 << 23) // C)
    for kk in range(K):
        ratio, mean, sd = P[:, kk, 0], P[:, kk, 1], P[:, kk, 2]
        for a in range(0, len(lin), step):
            b, uu, zz = lin_bin[a:a + step], u[a:a + step, None], z[a:a + step]
            dm, ds = 1.0 + uu, zz[:, :1] * (1.0 + uu)
            w = torch.ones(len(b), C, dtype=torch.float64, device=dev)
            Dm, Ds = torch.zeros_like(w), torch.zeros_like(w)
            alive = cap[a:a + step]
            for g in range(rows):
                x = (T - (dm * mean + ds * sd)) / h
                s, n = torch.sigmoid(x), torch.sigmoid(-x)
                leaf = w * n * (alive >= g)[:, None] * (2.0 ** g / paths)
                at = vmap[b, g]
                acc[kk, 0].index_add_(0, at, leaf)
                acc[kk, 1].index_add_(0, at, leaf * (Dm + s * dm / h) * ratio)
                acc[kk, 2].index_add_(0, at, leaf * (Ds + s * ds / h) * ratio)
                Dm, Ds, w = Dm - n * dm / h, Ds - n * ds / h, w * s
                if g + 1 < rows:
                    dm, ds = dm + 1.0, ds + zz[:, g + 1:g + 2]
    J = acc[:, :, :len(out)].permute(3, 2, 0, 1).contiguous()
    return (J[..., 0] * P[:, None, :, 0]).sum(-1), J


def exact(case, seed):
    path = case["path"]
    if path in ("simulate", "rerun"):  # counts are whole numbers
        values, freq = _histogram(np.random.default_rng(seed), case["bins"], case["cells"], case["top"])
        return {"values": _value_set(values, freq, case["phi"] or None), "totals": None, "per_type": None}
    if path == "batch":
        inst = _instances(case, np.random.default_rng(seed))
        return {"values": np.concatenate([_value_set(*x[0], x[3]) for x in inst]), "totals": None, "per_type": None}
    if path == "search":
        return None
    E, J = _smooth_exact(case, seed)
    if path == "smooth_forward":
        return {"expected": E}
    if path == "smooth_jacobian":
        return {"expected": E, "jacobian": J}
    target = torch.tensor(np.sort(_smooth_inputs(case, seed)[4][:E.shape[1]]), device=E.device)
    r = torch.log1p(E) - torch.log1p(target)
    if path == "smooth_step":
        return {"expected": E, "loss": (r ** 2).sum(1), "grad": torch.einsum("cv,cvkp->ckp", 2.0 * r / (1.0 + E), J)}
    Js = (J / (1.0 + E)[:, :, None, None]).reshape(len(E), E.shape[1], -1)
    return {"loss": (r ** 2).sum(1), "jtj": torch.einsum("cvp,cvq->cpq", Js, Js), "jtr": torch.einsum("cvp,cv->cp", Js, r)}
