"""Workloads for timing the package: what PyCPET users have the GPU do.

Every case goes through a public entry point: the calculator methods that the
PyCPET dispatcher calls (``drop_in.Calculator``, host arrays in and out) and
the array-level API on device tensors (``field_grid`` / ``GridBatch`` /
``topo_lines`` / ``TopoBatch`` / ``topo_dipole_lines`` / ``topo_hist2d`` /
``chi2_distance_matrix``).  Frames are the seeded synthetic ones of
``pycpet_gb300.synth``: 0.04 charges per cubic Angstrom, at least 1 A apart,
none within 2 A of the box centre.

Sizes: frames of 2,000-100,000 charges, volumes of 11-51 points per side at
0.1 A, streamline sets of a few lines up to 100,000, batches of uneven frames.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from pycpet_gb300 import (GridBatch, TopoBatch, chi2_distance_matrix, topo_dipole_lines, topo_hist2d, topo_lines)
from pycpet_gb300.drop_in import Calculator
from pycpet_gb300.synth import make_dipole_frame, make_frame, random_start_points

COULOMB = 14.3996451   # V*A/e
DEV = "cuda"


def listed():
    return [
        # the smallest call: the field at the active-site centre of one frame
        {"name": "point_field", "kind": "point_field", "n": 8000, "precision": "fp32c"},
        # method "volume" on one frame: a 21^3 grid, default precision and the plain FP64 form
        {"name": "volume_21", "kind": "volume", "n": 5000, "hx": 1.0, "hy": 1.0, "hz": 1.0, "precision": "fp32c"},
        {"name": "volume_21_fp64", "kind": "volume", "n": 5000, "hx": 1.0, "hy": 1.0, "hz": 1.0,
         "precision": "fp64"},
        # method "volume_ESP" on a larger frame: a 31^3 grid
        {"name": "esp_31", "kind": "esp", "n": 20000, "hx": 1.5, "hy": 1.5, "hz": 1.5, "precision": "fp32c"},
        # a trajectory's volumes in one prepared launch, replayed as frames arrive
        {"name": "volume_batch", "kind": "batch", "what": "field", "frames": 24, "n_lo": 3000, "n_hi": 40000,
         "graph": True, "precision": "fp32c"},
        # a few potentials in one unprepared launch, as a serving loop issues them
        {"name": "esp_batch", "kind": "batch", "what": "esp", "frames": 7, "n_lo": 3000, "n_hi": 40000,
         "graph": False, "precision": "fp32c"},
        # method "topo": 1,000 samples with random step caps, host arrays in and out
        {"name": "topo_1k", "kind": "topo", "n": 8000, "lines": 1000, "half": 1.5, "step": 0.001,
         "precision": "fp32c"},
        # the headline topology: 100,000 lines of one frame and their histogram
        {"name": "topo_100k", "kind": "topo_device", "n": 8000, "lines": 100000, "half": 1.5, "step": 0.001,
         "cap": 6000, "precision": "fp32c"},
        # the plain FP64 form of a small topology
        {"name": "topo_fp64", "kind": "topo_device", "n": 4000, "lines": 1000, "half": 1.5, "step": 0.002,
         "cap": 6000, "precision": "fp64"},
        # topologies of several frames in one prepared launch; the larger frames exceed shared memory
        {"name": "topo_batch", "kind": "topo_batch", "frames": 6, "n_lo": 5000, "n_hi": 20000, "lines": 3000,
         "step": 0.001, "cap": 6000, "precision": "fp32c"},
        # point-dipole streamlines
        {"name": "topo_dipole", "kind": "dipole", "n": 8000, "lines": 5000, "half": 1.5, "step": 0.001, "cap": 6000,
         "precision": "fp32c"},
        # the distance matrix of a trajectory's topology histograms, ahead of clustering
        {"name": "chi2", "kind": "chi2", "n": 1024, "bins": 400, "precision": "fp32c"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["point_field", "volume", "volume", "esp", "batch", "topo", "topo", "topo_device", "topo_batch",
                       "dipole", "chi2"])
    prec = rng.choice(["fp32c", "fp32c", "fp64"])
    if kind == "point_field":
        return {"kind": kind, "n": _log(rng, 2000, 100000), "precision": prec}
    if kind in ("volume", "esp"):
        half = [rng.randint(5, 25) / 10 for _ in range(3)]
        return {"kind": kind, "n": _log(rng, 2000, 40000), "hx": half[0], "hy": half[1], "hz": half[2],
                "precision": prec}
    if kind == "batch":
        return {"kind": kind, "what": rng.choice(["field", "esp"]), "frames": rng.randint(2, 24),
                "n_lo": _log(rng, 1000, 5000), "n_hi": _log(rng, 6000, 40000), "graph": rng.random() < 0.5,
                "precision": "fp32c"}
    if kind in ("topo", "topo_device", "dipole"):
        n = _log(rng, 2000, 100000 if prec == "fp32c" else 20000)
        most = (2.0e8 if kind == "topo_device" else 2.0e7) if prec == "fp32c" else 4.0e6
        half, step = rng.choice([1.0, 1.5, 2.0]), rng.choice([0.001, 0.002, 0.005, 0.01])
        if prec == "fp64":  # the plain form is kept to passes of about a second
            step = next(h for h in (0.002, 0.005, 0.01, 0.02) if half * n / h <= 3.0e6)
        case = {"kind": kind, "n": n, "lines": _log(rng, 10, max(20, min(60000, most * step * 1000 / n))),
                "half": half, "step": step, "precision": prec}
        if kind != "topo":
            case["cap"] = rng.choice([2000, 6000])
        return case
    if kind == "topo_batch":
        n_lo = _log(rng, 2000, 10000)
        return {"kind": kind, "frames": rng.randint(2, 12), "n_lo": n_lo, "n_hi": n_lo * rng.randint(2, 6),
                "lines": _log(rng, 50, 3000), "step": rng.choice([0.001, 0.002, 0.005]), "cap": 6000,
                "precision": "fp32c"}
    return {"kind": kind, "n": _log(rng, 100, 3000), "bins": rng.randint(50, 900), "precision": prec}


# ---- inputs -------------------------------------------------------------------

def _calculator(case, seed):
    """A calculator in the reference's option keys, as a program keeps one per frame."""
    fr = make_frame(case["n"], seed)
    opts = {"CPET_method": {"volume": "volume", "esp": "volume_ESP", "topo": "topo"}.get(case["kind"], "point_field"),
            "center": [0.0, 0.0, 0.0], "x": [1.0, 0.0, 0.0], "y": [0.0, 1.0, 0.0], "precision": case["precision"]}
    if case["kind"] in ("volume", "esp"):
        opts.update(dimensions=[case["hx"], case["hy"], case["hz"]], step_size=0.1)
    if case["kind"] == "topo":
        opts.update(dimensions=[case["half"]] * 3, step_size=case["step"], n_samples=case["lines"],
                    initializer="random")
    np.random.seed(seed % (1 << 32))
    return Calculator(opts, fr["x"], fr["q"])


def _batch_specs(case, seed):
    """(charges, half-width, frame seed) per frame: a trajectory batch of uneven frames."""
    rng = np.random.default_rng(seed)
    return [(int(rng.integers(case["n_lo"], case["n_hi"] + 1)), (0.5, 1.0, 1.5)[(f + 1) % 3], seed + 17 * f)
            for f in range(case["frames"])]


def _cube(half, step=0.1):
    g = np.linspace(-half, half, int(round(2 * half / step)) + 1)
    return np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)


def _grid_frames(case, seed):
    out = []
    for n, half, s in _batch_specs(case, seed):
        fr = make_frame(n, s)
        out.append((_cube(half), fr["x"], fr["q"]))
    return out


def _topo_frames(case, seed):
    F = case["frames"]
    out = []
    for f in range(F):
        n = case["n_lo"] + (case["n_hi"] - case["n_lo"]) * f // max(F - 1, 1)
        fr = make_frame(n, seed + 31 * f)
        half = [1.5, 1.5, 1.5]
        out.append({"x": fr["x"], "q": fr["q"], "starts": random_start_points(case["lines"], half, seed + 31 * f + 1),
                    "n_iter": case["cap"], "step": case["step"], "half_dims": half})
    return out


def _lines(case, seed):
    """Start points, caps, positions and charges (or moments) as device tensors."""
    fr = make_dipole_frame(case["n"], seed) if case["kind"] == "dipole" else make_frame(case["n"], seed)
    starts = random_start_points(case["lines"], [case["half"]] * 3, seed + 1)
    caps = np.full(case["lines"], case["cap"], np.int32)
    src = fr["mu"] if case["kind"] == "dipole" else fr["q"]
    return [torch.from_numpy(np.ascontiguousarray(a)).to(DEV) for a in (starts, caps, fr["x"], src)]


def _hists(case, seed):
    rng = np.random.default_rng(seed)
    centre = rng.gamma(0.5, 1.0, (8, case["bins"]))
    h = rng.poisson(40.0 * centre[rng.integers(0, 8, case["n"])]).astype(np.float64) + (rng.random(case["bins"]) < 0.5)
    return torch.from_numpy(h / h.sum(axis=1, keepdims=True)).to(DEV)


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("point_field", "volume", "esp", "topo"):
        return kind, case, _calculator(case, seed)
    if kind == "batch":
        return kind, case, GridBatch(_grid_frames(case, seed), kind=case["what"], precision=case["precision"],
                                     device=True, graph=case["graph"])
    if kind == "topo_batch":
        return kind, case, TopoBatch(_topo_frames(case, seed), precision=case["precision"], device=True, graph=True)
    if kind == "chi2":
        return kind, case, _hists(case, seed)
    return kind, case, _lines(case, seed)


def run(state):
    kind, case, s = state
    if kind == "point_field":
        return s.compute_point_field()
    if kind == "volume":
        return s.compute_box()
    if kind == "esp":
        return s.compute_box_ESP()
    if kind == "topo":
        return s.compute_topo_complete_c_shared()
    if kind == "batch":
        return s.run()
    if kind == "topo_batch":
        return s.run(return_steps=True)
    if kind == "chi2":
        return chi2_distance_matrix(s, precision=case["precision"])
    starts, caps, x, src = s
    half = [case["half"]] * 3
    if kind == "dipole":
        return topo_dipole_lines(starts, caps, x, src, case["step"], half, precision=case["precision"],
                                 return_steps=True)
    res, steps = topo_lines(starts, caps, x, src, case["step"], half, precision=case["precision"], return_steps=True)
    return res, steps, topo_hist2d(res, bins=(20, 20), range=((0.0, 5.2), (0.0, 4.0)))


# ---- work of one pass ----------------------------------------------------------
# flops per term: field 17, potential 9, dipole 29, chi-square 6 (the reciprocal
# square root or reciprocal not counted)

def _mean_steps(case):
    """Euler steps of a line on average: about 0.98 half-widths of arc until it leaves the box."""
    full = 0.98 * case.get("half", 1.5) / case["step"]
    return (0.75 * full if "cap" not in case else min(full, 0.8 * case["cap"])) + 2


def work(case):
    kind, n = case["kind"], case.get("n", 0)
    if kind == "point_field":
        return {"bytes": 16 * n + 24, "flops": 17 * n}
    if kind in ("volume", "esp"):
        pts = 1
        for h in (case["hx"], case["hy"], case["hz"]):
            pts *= int(2 * h / 0.1) + 1
        return {"bytes": 16 * n + pts * (36 if kind == "volume" else 20),
                "flops": pts * n * (17 if kind == "volume" else 9)}
    if kind == "batch":
        specs = _batch_specs(case, 1)
        pts = [(int(round(20 * h)) + 1) ** 3 for _, h, _ in specs]
        pairs = sum(p * m for p, (m, _, _) in zip(pts, specs))
        field = case["what"] == "field"
        return {"bytes": sum(32 * m for m, _, _ in specs) + sum(pts) * (48 if field else 32),
                "flops": pairs * (17 if field else 9)}
    if kind == "chi2":
        return {"bytes": 8 * n * case["bins"] + 8 * n * n, "flops": 6 * case["bins"] * n * (n - 1) // 2}
    steps = _mean_steps(case)
    if kind == "topo_batch":
        F = case["frames"]
        ns = [case["n_lo"] + (case["n_hi"] - case["n_lo"]) * f // max(F - 1, 1) for f in range(F)]
        return {"bytes": sum(32 * m for m in ns) + F * case["lines"] * 48,
                "flops": 17 * steps * case["lines"] * sum(ns)}
    per = 29 if kind == "dipole" else 17
    return {"bytes": n * (48 if kind == "dipole" else 32) + case["lines"] * 48, "flops": per * steps * case["lines"] * n}


# ---- the same in plain 64-bit torch ---------------------------------------------

def _t(a):
    return (a if isinstance(a, torch.Tensor) else torch.from_numpy(np.ascontiguousarray(a))).to(DEV, torch.float64)


def _sum64(pts, x, q, clamp, esp):
    pts, x, q = _t(pts), _t(x), _t(q).reshape(-1)
    per = max(1, 20_000_000 // max(len(q), 1))
    out = []
    for p in pts.split(per):
        d = p[:, None, :] - x[None, :, :]
        r2 = (d * d).sum(-1)
        if esp:
            out.append(COULOMB * (q / r2.sqrt()).sum(1))
        else:
            r2 = r2.clamp(min=1e-6) if clamp else r2
            out.append(COULOMB * ((q / (r2 * r2.sqrt()))[..., None] * d).sum(1))
    return torch.cat(out)


def _direction(p, x, src, dipole):
    out = []
    for c in p.split(max(1, 20_000_000 // len(x))):
        d = c[:, None, :] - x[None, :, :]
        r2 = (d * d).sum(-1)
        if dipole:
            w = (3 * src[:, 0] * d[..., 0] + src[:, 1] * d[..., 1] + src[:, 2] * d[..., 2]) / r2.pow(2.5)
            e = (w[..., None] * d).sum(1) - (1 / (r2 * r2.sqrt())) @ src
        else:
            e = ((src / (r2 * r2.sqrt()))[..., None] * d).sum(1)
        out.append(e / e.norm(dim=1, keepdim=True))
    return torch.cat(out)


def _curve(a, b):
    return torch.linalg.cross(a, b).norm(dim=1) / a.norm(dim=1) ** 3


def _streamlines64(starts, caps, x, src, step, half, dipole=False):
    starts, x, src, half = _t(starts), _t(x), _t(src), _t(half)
    src = src if dipole else src.reshape(-1)
    caps = _t(caps)

    def ahead(p):
        return p + step * _direction(p, x, src, dipole)

    pos, live = starts.clone(), torch.nonzero(caps > 0).reshape(-1)
    k = 0
    while len(live):
        k += 1
        nx = ahead(pos[live])
        pos[live] = nx
        live = live[(nx.abs() <= half).all(1) & (caps[live] > k)]
    x1 = ahead(starts)
    x2 = ahead(x1)
    e1 = ahead(pos)
    e2 = ahead(e1)
    curv = 0.5 * (_curve(x1 - starts, x2 - 2 * x1 + starts) + _curve(e1 - pos, e2 - 2 * e1 + pos))
    return torch.stack([(starts - pos).norm(dim=1), curv], 1)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("point_field", "volume", "esp"):
        c = _calculator(case, seed)
        if kind == "point_field":
            return _sum64(np.zeros((1, 3)), c.x, c.Q, False, False)[0]
        p = c.mesh.reshape(-1, 3)
        v = _sum64(p, c.x, c.Q, True, kind == "esp")
        return torch.cat([_t(p), v.reshape(len(p), -1)], 1), tuple(c.mesh.shape)
    if kind == "batch":
        v = [_sum64(p, x, q, True, case["what"] == "esp") for p, x, q in _grid_frames(case, seed)]
        return torch.cat([t.reshape(len(t), -1) for t in v])
    if kind == "chi2":
        h = _hists(case, seed)
        rows = []
        for a in h.split(max(1, 20_000_000 // h.numel())):
            s = a[:, None] + h[None]
            d = (a[:, None] - h[None]) ** 2
            rows.append(torch.where(s != 0, d / torch.where(s != 0, s, 1.0), 0.0).sum(-1) / 2)
        return torch.cat(rows).fill_diagonal_(0.0)
    if work(case)["flops"] > 1.2e12:
        return None
    if kind == "topo":
        c = _calculator(case, seed)
        return _streamlines64(c.random_start_points, c.random_max_samples, c.x, c.Q, float(c.step_size), c.dimensions)
    if kind == "topo_batch":
        return torch.cat([_streamlines64(f["starts"], np.full(len(f["starts"]), f["n_iter"]), f["x"], f["q"],
                                         f["step"], np.array(f["half_dims"])) for f in _topo_frames(case, seed)]), None
    starts, caps, x, src = _lines(case, seed)
    res = _streamlines64(starts, caps, x, src, case["step"], np.array([case["half"]] * 3), kind == "dipole")
    return (res, None) if kind == "dipole" else (res, None, None)
