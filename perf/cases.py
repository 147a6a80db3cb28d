"""The work whose speed is followed: calls of the Ewald operator as host programs make them.

Every case goes through the public Python interface over the C ABI.  Inputs are seeded and synthetic
(Bohr, one lattice vector per row): rigid water boxes at 1 g/cm^3, jittered rock salt, random charges in
cubic and triclinic cells, the families of the benchmark and the tests.  `call` names the entry point:

  device   Context.potential_force_device on device arrays (a program that keeps its state on the GPU)
  host     Context.potential_force on host arrays
  scf      TCoulomb on host arrays: one geometry, several charge updates with a shift each, then the
           gradients and the stress of the fast engine (one step of DFTB+'s SCC loop and forces)
  shifts   Context.shift_batch on a resident geometry
  stress   Context.potential_force_stress on host arrays
  points   Context.potential_at and potential_gradient_at: field of the charges at other points
  batch    PackedCells.evaluate: many independent cells in one call

`exact` is a plain Ewald sum in 64 bits with torch, converged far below the tolerances asked for.
"""

import gc
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(_ROOT, "dftb_fast-ewald_3d_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import ewald_b200 as eb  # noqa: E402

BOHR = 1.8897261254578281  # per Angstrom


def listed():
    return [
        # The smallest call: one shift+force evaluation of a small cell; latency and launches.
        {"name": "host_64", "call": "host", "system": "cubic", "n": 64, "form": "fp64", "scheme": "ik",
         "tol": 1e-10},
        # One DFTB+ step on a molecular cell of ordinary size at the adapter's default tolerance.
        {"name": "scf_999", "call": "scf", "system": "water", "n": 999, "form": "fp64", "scheme": "ik",
         "tol": 1e-9, "updates": 6},
        # A few thousand charges, the size at which the reference's own benchmark starts.
        {"name": "device_4096", "call": "device", "system": "cubic", "n": 4096, "form": "fp64",
         "scheme": "ik", "tol": 1e-10, "force": True},
        # The headline workload of the benchmark, plain form.
        {"name": "device_32769", "call": "device", "system": "water", "n": 32769, "form": "fp64",
         "scheme": "ik", "tol": 1e-10, "force": True},
        # The same with the mixed form at the parameters its tuner returns for this density.
        {"name": "device_32769_mixed", "call": "device", "system": "water", "n": 32769, "form": "mixed",
         "scheme": "ad", "tol": 1e-7, "force": True, "alpha": 0.26581903, "r_cut": 14.0326168,
         "k_cut": 1.85530234, "window": 6},
        # Forces by window differentiation, an odd size in a skew cell.
        {"name": "device_10007_skew_ad", "call": "device", "system": "skew", "n": 10007, "form": "fp64",
         "scheme": "ad", "tol": 1e-10, "force": True},
        # A large ionic crystal.
        {"name": "device_216000", "call": "device", "system": "salt", "n": 216000, "form": "fp64",
         "scheme": "ik", "tol": 1e-10, "force": True},
        # SCC charge updates on one geometry.
        {"name": "shifts_12000x8", "call": "shifts", "system": "water", "n": 12000, "form": "fp64",
         "scheme": "ik", "tol": 1e-9, "updates": 8},
        # Cell relaxation: potential, force and stress in one evaluation.
        {"name": "stress_5001_skew", "call": "stress", "system": "skew", "n": 5001, "form": "fp64",
         "scheme": "ik", "tol": 1e-10},
        # Electrostatic potential and field of a molecular cell at the points of an output grid.
        {"name": "points_20011", "call": "points", "system": "water", "n": 6000, "targets": 20011,
         "form": "fp64", "scheme": "ik", "tol": 1e-9},
        # A data set of small triclinic crystals, plain and mixed form.
        {"name": "batch_128", "call": "batch", "system": "cells", "n": 64000, "cells": 128, "form": "fp64",
         "scheme": "ik", "tol": 1e-10},
        {"name": "batch_96_mixed", "call": "batch", "system": "cells", "n": 48000, "cells": 96,
         "form": "mixed", "scheme": "ik", "tol": 1e-7},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    call = rng.choice(["device"] * 4 + ["host", "host", "scf", "shifts", "stress", "points", "batch", "batch"])
    c = {"call": call, "system": rng.choice(["cubic", "water", "skew", "salt"]), "form": "fp64",
         "scheme": rng.choice(["ik", "ik", "ad"]), "tol": rng.choice([1e-10, 1e-10, 1e-9])}
    if call == "device":
        c.update(n=_log(rng, 60, 120000), force=rng.random() < 0.75)
        if rng.random() < 0.25:
            c.update(form="mixed", tol=1e-7)
    elif call == "host":
        c.update(n=_log(rng, 50, 30000))
    elif call == "scf":
        c.update(n=_log(rng, 50, 12000), updates=rng.randint(3, 9))
    elif call == "shifts":
        c.update(n=_log(rng, 300, 30000), updates=rng.randint(3, 12))
    elif call == "stress":
        c.update(n=_log(rng, 60, 20000))
    elif call == "points":
        c.update(n=_log(rng, 1100, 12000), targets=_log(rng, 1100, 40000))
    else:
        k = _log(rng, 4, 128)
        c.update(system="cells", cells=k, n=k * rng.randint(150, 500))
        if rng.random() < 0.25:
            c.update(form="mixed", tol=1e-7)
    if c["system"] == "water":
        c["n"] = max(48, c["n"] // 3 * 3)
    if c["system"] == "salt":  # whole crystals: an even number of sites per axis
        c["n"] = max(4, 2 * round(0.5 * c["n"] ** (1.0 / 3.0))) ** 3
    return c


# ---- inputs -------------------------------------------------------------------------------------------


def _neutral(q):
    return q - q.mean()


def _lattice(a, b, c, al, be, ga):
    al, be, ga = (math.radians(x) for x in (al, be, ga))
    cx = c * math.cos(be)
    cy = c * (math.cos(al) - math.cos(be) * math.cos(ga)) / math.sin(ga)
    return np.array([[a, 0.0, 0.0], [b * math.cos(ga), b * math.sin(ga), 0.0],
                     [cx, cy, math.sqrt(c * c - cx * cx - cy * cy)]])


def _spaced(rng, n):
    """n fractional points, one in each of n cells of a grid, so that no two charges nearly coincide."""
    k = math.ceil(n ** (1.0 / 3.0) - 1e-9)
    site = np.sort(rng.choice(k ** 3, n, replace=False))
    ijk = np.stack([site // (k * k), site // k % k, site % k], axis=1)
    return (ijk + 0.5 + rng.uniform(-0.45, 0.45, size=(n, 3))) / k


def _system(kind, n, rng):
    """positions (n, 3), charges (n), lattice rows."""
    if kind == "water":
        m = n // 3
        edge = (m * 18.015 / 0.602214076) ** (1.0 / 3.0)  # Angstrom, 1 g/cm^3
        k = math.ceil(m ** (1.0 / 3.0) - 1e-9)
        gap = edge / k
        site = np.sort(rng.choice(k ** 3, m, replace=False))
        ijk = np.stack([site // (k * k), site // k % k, site % k], axis=1)
        o = (ijk + 0.5) * gap + rng.uniform(-1, 1, size=(m, 3)) * max(0.0, 0.5 * (gap - 2.5))
        half = math.radians(104.5) / 2
        h = 0.96 * np.array([[math.sin(half), math.cos(half), 0], [-math.sin(half), math.cos(half), 0]])
        r, _ = np.linalg.qr(rng.normal(size=(m, 3, 3)))
        pos = np.concatenate([o[:, None], o[:, None] + np.einsum("nij,hj->nhi", r, h)], axis=1).reshape(-1, 3)
        q = np.tile([-0.82, 0.41, 0.41], m) * (1 + rng.normal(0, 0.03, size=3 * m))
        return pos * BOHR, _neutral(q), np.eye(3) * edge * BOHR
    if kind == "salt":
        k = round(n ** (1.0 / 3.0))
        ijk = np.stack(np.meshgrid(*(np.arange(k),) * 3, indexing="ij"), -1).reshape(-1, 3)
        q = 0.8 * np.where(ijk.sum(axis=1) % 2 == 0, 1.0, -1.0) + rng.normal(0, 0.05, size=k ** 3)
        pos = ijk * 2.82 + rng.normal(0, 0.05, size=(k ** 3, 3))
        return pos * BOHR, _neutral(q), np.eye(3) * k * 2.82 * BOHR
    edge = (n * 10.5) ** (1.0 / 3.0) * BOHR  # about 10.5 cubic Angstrom per charge
    if kind == "cubic":
        lat = np.eye(3) * edge
    else:
        lat = _lattice(*(edge * rng.uniform(0.75, 1.3, size=3)), *rng.uniform(72, 108, size=3))
    return _spaced(rng, n) @ lat, _neutral(rng.normal(0, 0.35, size=n)), lat


def _cells(case, rng):
    """cells of 30 to some thousand charges whose sizes add up to about case["n"]; 10 to 30 Angstrom wide."""
    w = np.exp(rng.uniform(math.log(50), math.log(2000), size=case["cells"]))
    sizes = np.clip(np.round(w * case["n"] / w.sum()), 30, 4000).astype(int)
    out = []
    for n in sizes:
        while True:
            lat = _lattice(*rng.uniform(10, 30, size=3), *rng.uniform(70, 110, size=3)) * BOHR
            if np.isfinite(lat).all() and lat[2, 2] > 0.3 * np.linalg.norm(lat[2]):
                break
        out.append((_spaced(rng, n) @ lat, _neutral(rng.normal(0, 0.4, size=n)), lat))
    return out


def _inputs(case, seed):
    # Cell shapes and the sizes of a batch belong to the case: the same work for every seed.
    shape = np.random.default_rng([17, case["n"]])
    rng = np.random.default_rng([seed, case["n"]])
    d = {}
    if case["call"] == "batch":
        d["cells"] = [(_spaced(rng, len(q)) @ lat, _neutral(rng.normal(0, 0.4, size=len(q))), lat)
                      for _, q, lat in _cells(case, shape)]
        return d
    if case["system"] == "skew":
        lat = _system("skew", 8, shape)[2] * (case["n"] / 8.0) ** (1.0 / 3.0)
        d["pos"], d["q"], d["lat"] = _spaced(rng, case["n"]) @ lat, _neutral(rng.normal(0, 0.35, case["n"])), lat
    else:
        d["pos"], d["q"], d["lat"] = _system(case["system"], case["n"], rng)
    n = len(d["q"])
    if "updates" in case:
        d["updates"] = np.stack([_neutral(d["q"] * (1 + rng.normal(0, 0.05, size=n)))
                                 for _ in range(case["updates"])])
    if "targets" in case:
        d["targets"] = rng.uniform(size=(case["targets"], 3)) @ d["lat"]
    return d


# ---- the calls ----------------------------------------------------------------------------------------


def prepare(case, seed):
    d = _inputs(case, seed)
    form = eb.MIXED if case["form"] == "mixed" else eb.FP64
    scheme = eb.FORCE_AD if case["scheme"] == "ad" else eb.FORCE_IK
    s = {"case": case, "d": d}
    if case["call"] == "scf":
        s["coulomb"] = eb.TCoulomb(len(d["q"]), tolEwald=case["tol"], precision=form, fastStress=True)
        s["coulomb"].ctx.set_force_scheme(scheme)
        return s
    s["ctx"] = ctx = eb.Context(0, form)
    ctx.set_force_scheme(scheme)
    if case["call"] == "device":
        n = len(d["q"])
        s["x"] = torch.tensor(d["pos"], dtype=torch.float64, device="cuda")
        s["q"] = torch.tensor(d["q"], dtype=torch.float64, device="cuda")
        s["pot"] = torch.zeros(n, dtype=torch.float64, device="cuda")
        s["force"] = torch.zeros((n, 3), dtype=torch.float64, device="cuda") if case["force"] else None
        names = {"alpha": "alpha_in", "r_cut": "r_cut_in", "k_cut": "k_cut_in", "window": "windowCutoff_in"}
        s["ov"] = {names[k]: case[k] for k in names if k in case}
        torch.cuda.synchronize()  # the context works on a stream of its own
    elif case["call"] == "shifts":
        ctx.set_lattice(d["lat"].T)
        ctx.set_coords(d["pos"])
        ctx.set_charges(d["q"])
        s["out"] = np.zeros_like(d["updates"])
    elif case["call"] == "batch":
        s["packed"] = eb.PackedCells(d["cells"], alloc=lambda shape: torch.zeros(
            shape, dtype=torch.float64, pin_memory=True).numpy())
    return s


def run(s):
    case, d, call = s["case"], s["d"], s["case"]["call"]
    if call == "device":
        s["ctx"].potential_force_device(s["x"], s["q"], d["lat"], case["tol"], s["pot"], s["force"], **s["ov"])
        return [s["pot"], s["force"]] if case["force"] else [s["pot"]]
    if call == "host":
        return list(s["ctx"].potential_force(d["pos"], d["q"], d["lat"], case["tol"]))
    if call == "stress":
        return list(s["ctx"].potential_force_stress(d["pos"], d["q"], d["lat"], case["tol"]))
    if call == "shifts":
        return [s["ctx"].shift_batch(case["tol"], d["updates"], out=s["out"])]
    if call == "points":
        return [s["ctx"].potential_at(d["targets"], d["pos"], d["q"], d["lat"].T, case["tol"]),
                s["ctx"].potential_gradient_at(d["targets"], d["pos"], d["q"], d["lat"].T, case["tol"])]
    if call == "batch":
        s["packed"].evaluate(s["ctx"], case["tol"])
        return [s["packed"].pot, s["packed"].force]
    c = s["coulomb"]
    c.updateLatVecs(d["lat"].T)
    c.updateCoords(d["pos"].T)
    shifts = []
    for q in d["updates"]:
        c.updateCharges(q)
        shifts.append(c.updateShifts())
    gradient = c.addGradients(np.zeros((3, c.nAtom)))
    stress = c.addStress(np.zeros((3, 3)))
    return [np.stack(shifts), gradient, stress]


def work(case):
    """Inputs read and outputs written once; pair terms within three mean spacings (113 pairs per charge,
    about 30 operations each) and, per evaluation, one transform of the retained modes there and one back
    (about 85 modes per charge at these tolerances)."""
    n = case["n"]
    if case["call"] == "scf":
        evals, values = case["updates"] + 2, n * (3 + 2 * case["updates"] + 3)
    elif case["call"] == "shifts":
        evals, values = case["updates"], 2 * n * case["updates"]
    elif case["call"] == "points":
        evals, values = 2, 8 * n + 10 * case["targets"]
    else:
        evals, values = 1, 8 * n if case.get("force", True) else 5 * n
    modes = 85 * n / case.get("cells", 1)
    flops = evals * (113 * 30 * n + case.get("cells", 1) * 10 * modes * math.log2(modes))
    return {"bytes": 8 * values, "flops": flops}


# ---- plain Ewald sums in 64 bits ----------------------------------------------------------------------


def _ewald(lat, src, q, tgt=None, force=False, stress=False):
    """Potential at the targets (the sources themselves by default) of the sources and their images, and on
    request its negative gradient times the target's charge (the gradient itself for other targets) and
    the stress (2/V) dE/d(strain).  Real space within r_c, minimum images; all modes of a box beyond."""
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    f64 = dict(dtype=torch.float64, device=dev)
    self_sum = tgt is None
    lat = torch.tensor(np.asarray(lat), **f64)
    rec = torch.linalg.inv(lat).T.contiguous()  # rows b_i, b_i . a_j = delta_ij
    vol = float(torch.linalg.det(lat).abs())
    src, q = torch.tensor(np.asarray(src), **f64), torch.tensor(np.asarray(q), **f64)
    s = src @ rec.T
    t = s if self_sum else torch.tensor(np.asarray(tgt), **f64) @ rec.T
    nt, ns = len(t), len(s)
    width = 1.0 / float(rec.norm(dim=1).max())
    # The cutoff falls as the cell grows, so that pairs and modes share the work.
    rc = width * min(0.45, max(0.1, 1.2 * ns ** -0.2))
    x = 6.0
    alpha = x / rc
    kmax = 2.0 * alpha * x
    pot = torch.zeros(nt, **f64)
    grad = torch.zeros(nt, 3, **f64)
    vir = torch.zeros(3, 3, **f64)
    rows = max(1, int(3e7) // ns)
    for i in range(0, nt, rows):
        f = t[i:i + rows, None, :] - s[None]
        f -= f.round()
        r = torch.stack([f[..., 0] * lat[0, c] + f[..., 1] * lat[1, c] + f[..., 2] * lat[2, c] for c in range(3)])
        r2 = (r * r).sum(0)
        if self_sum:
            k = torch.arange(i, i + r2.shape[0], device=dev)
            r2[k - i, k] = 4 * rc * rc
        a, b = (r2 < rc * rc).nonzero(as_tuple=True)
        r, r2 = r[:, a, b].T, r2[a, b]
        d = r2.sqrt()
        e = torch.erfc(alpha * d) / d
        pot.index_add_(0, a + i, q[b] * e)
        if force or stress:
            g = -(e + 2 * alpha / math.sqrt(math.pi) * torch.exp(-alpha * alpha * r2)) / r2  # phi'(r) / r
            grad.index_add_(0, a + i, (q[b] * g)[:, None] * r)
            if stress:
                vir += 0.5 * ((q[a + i] * q[b] * g)[:, None] * r).T @ r
        del f, r, r2, d, e, a, b
    # Modes: exp(2 pi i k.s) factorised along the three axes, the sum over sources as products of matrices.
    h = [int(math.ceil(kmax * float(lat[d].norm()) / (2 * math.pi))) for d in range(3)]
    k1 = torch.arange(-h[0], h[0] + 1, **f64)
    k2 = torch.arange(-h[1], h[1] + 1, **f64)

    def phase(frac, k):
        a = 2 * math.pi * frac[:, None] * k[None]
        return torch.complex(torch.cos(a), torch.sin(a))

    es1, es2 = phase(s[:, 0], k1), phase(s[:, 1], k2)
    et1, et2 = (es1, es2) if self_sum else (phase(t[:, 0], k1), phase(t[:, 1], k2))
    for k3 in range(h[2] + 1):
        kk = torch.tensor([float(k3)], **f64)
        z = phase(s[:, 2], kk)
        sk = (es1 * (q[:, None] * z)).conj().T @ es2.conj()  # sum_j q exp(-2 pi i k.s_j)
        kv = 2 * math.pi * (k1[:, None, None] * rec[0] + k2[None, :, None] * rec[1] + k3 * rec[2])
        g2 = (kv * kv).sum(-1)
        if k3 == 0:
            g2[h[0], h[1]] = 1.0
        w = 4 * math.pi / vol * torch.exp(-g2 / (4 * alpha * alpha)) / g2 * (2.0 if k3 else 1.0)
        if k3 == 0:
            w[h[0], h[1]] = 0.0
        if stress:
            e = 0.5 * w * (sk.real ** 2 + sk.imag ** 2)
            m = e * 2 * (1 / (4 * alpha * alpha) + 1 / g2)
            vir += torch.einsum("ab,abc,abd->cd", m, kv, kv) - e.sum() * torch.eye(3, **f64)
        zt = z if self_sum else phase(t[:, 2], kk)
        c = w * sk
        row = (et1 @ c) * et2 * zt
        pot += row.real.sum(1)
        if force:
            d1 = -(((et1 * k1) @ c) * et2 * zt).imag.sum(1)
            d2 = -(row * k2).imag.sum(1)
            d3 = -k3 * row.imag.sum(1)
            grad += 2 * math.pi * torch.stack([d1, d2, d3], 1) @ rec
    out = [pot - 2 * alpha / math.sqrt(math.pi) * q if self_sum else pot]
    if force:
        out.append(-q[:, None] * grad if self_sum else grad)
    if stress:
        out.append(2.0 / vol * vir)
    out = [v.cpu().numpy() for v in out]
    return out


def exact(case, seed):
    d, call = _inputs(case, seed), case["call"]
    if call == "batch":
        each = [_ewald(lat, p, q, force=True) for p, q, lat in d["cells"]]
        out = [np.concatenate([e[k] for e in each]) for k in (0, 1)]
    elif call == "points":
        out = _ewald(d["lat"], d["pos"], d["q"], tgt=d["targets"], force=True)
    elif call == "shifts":
        out = [np.stack([_ewald(d["lat"], d["pos"], q)[0] for q in d["updates"]])]
    elif call == "scf":
        each = [_ewald(d["lat"], d["pos"], q, force=True, stress=True) for q in d["updates"]]
        out = [np.stack([e[0] for e in each]), -each[-1][1].T, -0.5 * each[-1][2]]
    else:
        out = _ewald(d["lat"], d["pos"], d["q"], force=case.get("force", True), stress=call == "stress")
    gc.collect()
    return out
