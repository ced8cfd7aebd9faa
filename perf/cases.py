"""The work users of this framework have it do, as cases that can be timed and compared.

Every case goes through the public entry points of `dda_fft_b200`:

  convolution   `Context.convolution_dev`: G * p (or its conjugate) for device-resident fields
  plain         `Context.dda_fft` of both polarisations and `Context.mueller`: the drop-in
                path of the sample loop
  orientations  `Context.orientation_solves`: one target, many orientations
  realisations  `Context.realization_solves`: a target of its own for every sample
  agglomerates  `Group.agglomerate_solves`: lattices of different sizes, one graph launch
  linear        `Context.solve_linear`: mixed-precision CG for a given right-hand side
  fp64          `Context.solve_fp64`: the whole solve in double

Lattices have power-of-two edges (2..128 per axis), cubic or not.  Sizes, materials and
solver settings are those of the benchmark and the tests: spheres, ellipsoids, porous cubes
and agglomerates at size parameters 1.5..11, Error_max 1e-3 and below.  The batched solves hand
back doubles that were computed from single-precision fields (and are stored as floats in a
state file), so `run` gives them as float32.

`exact` computes the same outputs in double with torch alone: a dense FFT convolution, the
solvers' recurrences, the sums of the far field and the cross sections, and the Mueller
matrices.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import dda_fft_b200 as D

PI = math.pi
CM, CMRR, LDR = 1, 2, 5
CG, AA, BICGSTAB, SIMPLE = 0, 1, 2, 3


# ------------------------------------------------------------------------------- the cases
def listed():
    return [
        {"name": "convolution 16 x1", "kind": "convolution", "grid": "16,16,16", "nrhs": 1,
         "conj": False, "tune": False},
        {"name": "convolution 8x64x32 x4", "kind": "convolution", "grid": "8,64,32", "nrhs": 4,
         "conj": False, "tune": False},
        {"name": "convolution 32x128x64 x6 conj", "kind": "convolution", "grid": "32,128,64", "nrhs": 6,
         "conj": True, "tune": False},
        {"name": "convolution 64 x24", "kind": "convolution", "grid": "64,64,64", "nrhs": 24,
         "conj": False, "tune": False},
        {"name": "convolution 128 x16 tuned", "kind": "convolution", "grid": "128,128,128", "nrhs": 16,
         "conj": False, "tune": True},
        {"name": "plain 32", "kind": "plain", "grid": "32,32,32", "x": 2.0, "m_re": 1.5, "m_im": 0.01,
         "b_a": 1.0, "c_a": 1.0, "model": CM, "solver": CG, "err_max": 1e-3, "max_step": 20,
         "nplanes": 1, "theta_step": 10.0},
        {"name": "orientation 64 planes 12", "kind": "orientations", "grid": "64,64,64", "count": 1,
         "mc": False, "x": 6.0, "m_re": 1.5, "m_im": 0.01, "b_a": 1.0, "c_a": 1.0, "model": LDR,
         "solver": BICGSTAB, "err_max": 1e-3, "max_step": 100, "nplanes": 12, "theta_step": 1.0,
         "tune": False},
        {"name": "orientations 64 x64", "kind": "orientations", "grid": "64,64,64", "count": 64,
         "mc": True, "x": 6.0, "m_re": 1.55, "m_im": 0.005, "b_a": 0.7, "c_a": 0.5, "model": CM,
         "solver": CG, "err_max": 1e-3, "max_step": 20, "nplanes": 1, "theta_step": 10.0,
         "tune": True},
        {"name": "realisations 32 x24", "kind": "realisations", "grid": "32,32,32", "count": 24,
         "x": 3.0, "packing": 0.3, "model": CMRR, "solver": BICGSTAB, "err_max": 1e-6, "max_step": 20,
         "nplanes": 2, "theta_step": 5.0},
        {"name": "agglomerates 32 64 128", "kind": "agglomerates", "sizes": "32,64,128",
         "counts": "8,8,7", "x": 6.0, "m_re": 1.55, "m_im": 0.005, "packing": 0.25,
         "err_max": 1e-3, "max_step": 20, "nplanes": 1, "theta_step": 10.0},
        {"name": "linear 64", "kind": "linear", "grid": "64,64,64", "x": 5.0, "packing": 0.3,
         "err_max": 1e-9},
        {"name": "fp64 64", "kind": "fp64", "grid": "64,64,64", "x": 5.0, "m_re": 1.5, "m_im": 0.01,
         "b_a": 1.0, "c_a": 1.0, "solver": CG, "err_max": 1e-14, "max_step": 100, "theta_step": 2.0},
    ]


def _log_int(rng, lo, hi):
    """An integer spread over the logarithm of lo..hi."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _box(rng, lo, hi, cells):
    """Edges that are powers of two, at most `cells` lattice cells."""
    while True:
        e = [rng.choice([n for n in (2, 4, 8, 16, 32, 64, 128) if lo <= n <= hi]) for _ in range(3)]
        if rng.random() < 0.5:
            e = [e[0]] * 3
        if e[0] * e[1] * e[2] <= cells:
            return e


def _text(edges):
    return ",".join(str(n) for n in edges)


def draw(rng):
    kind = rng.choice(["convolution", "convolution", "convolution", "plain", "orientations",
                       "orientations", "realisations", "agglomerates", "linear", "fp64"])
    if kind == "convolution":
        e = _box(rng, 4, 128, 128 ** 3)
        n = e[0] * e[1] * e[2]
        most = max(1, min(64, 16 * 128 ** 3 // n))
        return {"kind": kind, "grid": _text(e), "nrhs": _log_int(rng, 1, most), "conj": rng.random() < 0.3,
                "tune": rng.random() < 0.2}
    m_re, m_im = round(rng.uniform(1.3, 1.65), 3), round(math.exp(rng.uniform(math.log(0.002), math.log(0.05))), 5)
    if kind == "plain":
        n = rng.choice((16, 32, 64))
        return {"kind": kind, "grid": _text((n, n, n)), "x": round(rng.uniform(1.5, 0.08 * n + 1), 2),
                "m_re": m_re, "m_im": m_im, "b_a": round(rng.uniform(0.5, 1.0), 2),
                "c_a": round(rng.uniform(0.5, 1.0), 2), "model": rng.choice((CM, CMRR, LDR)),
                "solver": rng.choice((CG, BICGSTAB)), "err_max": 1e-3, "max_step": 20,
                "nplanes": rng.choice((1, 1, 2, 4)), "theta_step": rng.choice((1.0, 2.0, 5.0, 10.0))}
    if kind == "orientations":
        n = rng.choice((16, 32, 64, 64, 128))
        most = {16: 128, 32: 96, 64: 56, 128: 6}[n]
        mc = rng.random() < 0.75
        return {"kind": kind, "grid": _text((n, n, n)), "count": _log_int(rng, 1, most) if mc else 1, "mc": mc,
                "x": round(rng.uniform(2.0, 0.08 * n + 1), 2), "m_re": m_re, "m_im": m_im,
                "b_a": round(rng.uniform(0.4, 1.0), 2), "c_a": round(rng.uniform(0.4, 1.0), 2),
                "model": rng.choice((CM, CM, CMRR, LDR)), "solver": rng.choice((CG, BICGSTAB)),
                "err_max": 1e-3, "max_step": 20, "nplanes": rng.choice((1, 1, 2) if mc else (2, 6, 12)),
                "theta_step": rng.choice((5.0, 10.0) if mc else (1.0, 2.0)), "tune": rng.random() < 0.2}
    if kind == "realisations":
        n = rng.choice((16, 32, 64))
        return {"kind": kind, "grid": _text((n, n, n)), "count": _log_int(rng, 1, {16: 64, 32: 32, 64: 6}[n]),
                "x": round(rng.uniform(1.5, 0.06 * n + 1.5), 2), "packing": round(rng.uniform(0.1, 0.4), 2),
                "model": rng.choice((CM, CMRR)), "solver": rng.choice((CG, BICGSTAB)),
                "err_max": rng.choice((1e-3, 1e-6)), "max_step": 20, "nplanes": rng.choice((1, 2)),
                "theta_step": rng.choice((5.0, 10.0))}
    if kind == "agglomerates":
        sizes = rng.choice(((16, 32), (32, 64), (32, 64, 128), (64, 128)))
        most = {16: 16, 32: 12, 64: 8, 128: 4}
        return {"kind": kind, "sizes": _text(sizes), "counts": _text(_log_int(rng, 1, most[n]) for n in sizes),
                "x": round(rng.uniform(3.0, 7.0), 2), "m_re": m_re, "m_im": m_im,
                "packing": round(rng.uniform(0.1, 0.25), 3), "err_max": 1e-3, "max_step": 20,
                "nplanes": 1, "theta_step": rng.choice((5.0, 10.0))}
    if kind == "linear":
        n = rng.choice((16, 32, 64))
        return {"kind": kind, "grid": _text((n, n, n)), "x": round(rng.uniform(1.5, 0.05 * n + 1.5), 2),
                "packing": round(rng.uniform(0.1, 0.4), 2), "err_max": rng.choice((1e-9, 3e-10))}
    e = _box(rng, 8, 64, 64 ** 3)
    return {"kind": kind, "grid": _text(e), "x": round(rng.uniform(1.5, 4.0), 2), "m_re": m_re, "m_im": m_im,
            "b_a": round(min(1.0, e[1] / e[0]) * 0.9, 3), "c_a": round(min(1.0, e[2] / e[0]) * 0.9, 3),
            "solver": rng.choice((CG, CG, BICGSTAB)), "err_max": 1e-14, "max_step": 100,
            "theta_step": rng.choice((5.0, 10.0))}


# ------------------------------------------------------------------------------ the inputs
def _ints(text):
    return tuple(int(v) for v in str(text).split(","))


def _grid(case):
    return _ints(case["grid"])


def _spacing(case):
    """k d of a target whose first axis spans the size parameter x."""
    return 2.0 * case["x"] / _grid(case)[0]


def _ellipsoid(grid, b_a, c_a):
    """Cell centres inside an ellipsoid whose first axis fills the lattice."""
    a = grid[0] / 2.0
    ax = [(np.arange(n) - (n / 2.0 - 0.5)) / r for n, r in zip(grid, (a, a * b_a, a * c_a))]
    r2 = ax[0][:, None, None] ** 2 + ax[1][None, :, None] ** 2 + ax[2][None, None, :] ** 2
    return (r2 <= 1.0).astype(np.int8)


def _index(case, seed):
    """The sample's refractive index: the case's, within a per cent (the next sample of a
    wavelength scan)."""
    rng = np.random.default_rng([seed, 1])
    f = np.float32
    return complex(f(case["m_re"] * (1 + 0.01 * rng.uniform(-1, 1))), f(case["m_im"] * (1 + 0.01 * rng.uniform(-1, 1))))


def _alpha(model, kd, m, kinc, einc):
    """Polarisability of one cell: CM, CMRR or LDR."""
    eps = m * m
    a = kd ** 3 * (0.75 / PI) * (eps - 1) / (eps + 2)
    if model == CMRR:
        return a / (1 - (2.0 / 3.0) * 1j * a)
    if model == LDR:
        s = float(np.sum((np.asarray(kinc) * np.asarray(einc)) ** 2))
        return a / (1 + (a / kd) * (-1.8915316 + 0.1648469 * eps - 1.7700004 * s * eps - (2.0 / 3.0) * kd * 1j))
    return a


def _rotations(count, mc, seed):
    """Rotation matrices uniform on SO(3), or the identity."""
    if not mc:
        return np.repeat(np.eye(3)[None], count, axis=0)
    q = np.random.default_rng([seed, 2]).standard_normal((count, 4))
    w, x, y, z = (q / np.linalg.norm(q, axis=1, keepdims=True)).T
    return np.stack([1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y),
                     2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x),
                     2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)], 1).reshape(-1, 3, 3)


def _planes(nplanes, theta_step):
    """Normals (planes, 3) and scattering directions (planes, angles, 3) before rotation."""
    na = D.num_angles(0.0, 180.0, theta_step)
    th = np.deg2rad(np.float32(theta_step) * np.arange(na, dtype=np.float64))
    ang = np.arange(nplanes) * (PI / nplanes)
    c, s = np.cos(ang)[:, None], np.sin(ang)[:, None]
    k = np.stack([c * np.sin(th), -s * np.sin(th), np.broadcast_to(np.cos(th), (nplanes, na))], -1)
    return np.stack([np.sin(ang), np.cos(ang), np.zeros(nplanes)], -1), k


def _porous(grid, packing, seed):
    """Cells filled at random, material 1 or 2 at 0.7 / 0.3."""
    rng = np.random.default_rng([seed, 3])
    filled = rng.random(grid, np.float32) < packing
    return np.where(filled, np.where(rng.random(grid, np.float32) < 0.7, 1, 2), 0).astype(np.int8)


_POROUS = (1.5 + 0.01j, 1.7 + 0.1j)


def _monomers(n, packing, seed):
    """Spherical monomers of radius 3 cells on a jittered grid that keeps them apart, inside
    the lattice's inscribed sphere: [count][13] = r, l, begin, end, axis, 0, 0."""
    r = 3.0
    step = max((4.0 / 3.0 * PI * r ** 3 / packing) ** (1.0 / 3.0), 2 * r + 0.1)
    rng = np.random.default_rng([seed, 4])
    k = max(1, int((n - 1) / step))
    g = (np.arange(k) - (k - 1) / 2.0) * step
    c = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    c = c + rng.uniform(-0.5, 0.5, c.shape) * (step - 2 * r)
    near = np.linalg.norm(c, axis=1) <= n / 2.0 - r
    c = c[near] if near.any() else c[:1]
    axis = rng.standard_normal(c.shape)
    axis /= np.linalg.norm(axis, axis=1, keepdims=True)
    out = np.zeros((len(c), 13), np.float32)
    out[:, 0] = r
    out[:, 2:5] = out[:, 5:8] = c
    out[:, 8:11] = axis
    return out


def _fields(case, seed):
    """Random device-resident dipole fields (nrhs, 3, ni, nj, nl)."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    shape = (case["nrhs"], 3) + _grid(case)
    return torch.randn(shape, dtype=torch.complex64, device="cuda", generator=g)


def _linear_rhs(case, seed):
    """An adjoint-like source on the active cells of a porous cube."""
    grid = _grid(case)
    occ = _porous(grid, case["packing"], seed)
    kd = _spacing(case)
    alpha = np.array([0, *(_alpha(CMRR, kd, m, (0, 0, 1), (1, 0, 0)) for m in _POROUS)], np.complex64)
    rng = np.random.default_rng([seed, 5])
    g = rng.standard_normal(grid + (3, 2), np.float32) + 1.0
    rhs = (g[..., 0] + 1j * g[..., 1]).astype(np.complex64) * alpha[occ][..., None]
    return occ, alpha, rhs.astype(np.complex64)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "convolution":
        grid, n = _grid(case), case["nrhs"]
        ctx = D.Context(grid, 2 * 6.0 / max(grid), max_rhs=n)
        if case["tune"]:
            ctx.autotune(n)
        x = _fields(case, seed)
        return {"kind": kind, "ctx": ctx, "x": x, "y": torch.empty_like(x), "nrhs": n, "conj": case["conj"]}
    if kind == "agglomerates":
        sizes, counts = _ints(case["sizes"]), _ints(case["counts"])
        m = _index(case, seed)
        ctxs = [D.Context(n, 2.0 * case["x"] / n, max_rhs=2 * c) for n, c in zip(sizes, counts)]
        mons = [[_monomers(n, case["packing"], seed + 1000 * n + k) for k in range(c)]
                for n, c in zip(sizes, counts)]
        cfg = D.BatchConfig(occ=None, materials=[(m.real, m.imag)], max_step=case["max_step"],
                            err_max=case["err_max"], nplanes=case["nplanes"], theta_step=case["theta_step"])
        return {"kind": kind, "ctxs": ctxs, "group": D.Group(ctxs), "cfg": cfg, "mons": mons}
    grid, kd = _grid(case), _spacing(case)
    if kind == "plain":
        m = _index(case, seed)
        normals, ksc = _planes(case["nplanes"], case["theta_step"])
        alpha = [np.array([0, _alpha(case["model"], kd, m, (0, 0, 1), e)], np.complex64) for e in ((1, 0, 0), (0, 1, 0))]
        return {"kind": kind, "ctx": D.Context(grid, kd, max_rhs=2), "kd": kd, "alpha": alpha,
                "occ": _ellipsoid(grid, case["b_a"], case["c_a"]), "ksc": ksc.astype(np.float32),
                "normals": normals.astype(np.float32), "solver": case["solver"],
                "err_max": case["err_max"], "max_step": case["max_step"]}
    if kind == "orientations":
        m, n = _index(case, seed), case["count"]
        ctx = D.Context(grid, kd, max_rhs=2 * n)
        if case["tune"]:
            ctx.autotune(2 * n)
        cfg = D.BatchConfig(occ=_ellipsoid(grid, case["b_a"], case["c_a"]), materials=[(m.real, m.imag)],
                            solver=case["solver"], max_step=case["max_step"], err_max=case["err_max"],
                            polarizability=case["model"], nplanes=case["nplanes"], theta_step=case["theta_step"])
        return {"kind": kind, "ctx": ctx, "cfg": cfg, "rot": _rotations(n, case["mc"], seed)}
    if kind == "realisations":
        n = case["count"]
        cfg = D.BatchConfig(occ=None, materials=[(m.real, m.imag) for m in _POROUS], solver=case["solver"],
                            max_step=case["max_step"], err_max=case["err_max"], polarizability=case["model"],
                            nplanes=case["nplanes"], theta_step=case["theta_step"])
        occ = np.stack([_porous(grid, case["packing"], seed + 1000 * (k + 1)) for k in range(n)])
        return {"kind": kind, "ctx": D.Context(grid, kd, max_rhs=2 * n), "cfg": cfg, "occ": occ,
                "rot": _rotations(n, True, seed)}
    if kind == "linear":
        occ, alpha, rhs = _linear_rhs(case, seed)
        return {"kind": kind, "ctx": D.Context(grid, kd), "occ": occ, "alpha": alpha, "rhs": rhs,
                "err_max": case["err_max"]}
    m = _index(case, seed)
    _, ksc = _planes(1, case["theta_step"])
    return {"kind": kind, "ctx": D.Context(grid, kd), "occ": _ellipsoid(grid, case["b_a"], case["c_a"]), "kd": kd,
            "alpha": np.array([0, _alpha(CMRR, kd, m, (0, 0, 1), (1, 0, 0))]), "ksc": ksc[0],
            "solver": case["solver"], "err_max": case["err_max"], "max_step": case["max_step"]}


# -------------------------------------------------------------------------------- the pass
def _batch(r):
    """A batched call's results in the precision of the fields they were computed from."""
    return {k: r[k].astype(np.float32) for k in ("cabs", "cext", "mueller")}


def run(state):
    s, kind = state, state["kind"]
    if kind == "convolution":
        s["ctx"].convolution_dev(s["x"], s["y"], s["nrhs"], s["conj"])
        return s["y"]
    if kind == "plain":
        k, E = (0, 0, 1), ((1, 0, 0), (0, 1, 0))
        r = [s["ctx"].dda_fft(s["occ"], s["alpha"][q], [0, 1], s["kd"], k, E[q], s["ksc"], solver=s["solver"],
                              max_step=s["max_step"], err_max=s["err_max"], trace=False) for q in range(2)]
        M = s["ctx"].mueller(k, E[0], E[1], s["ksc"], s["normals"], r[0]["esc"], r[1]["esc"])
        return {"esc": [q["esc"] for q in r], "cabs": [q["cabs"] for q in r], "cext": [q["cext"] for q in r],
                "mueller": M}
    if kind == "orientations":
        return _batch(s["ctx"].orientation_solves(s["cfg"], s["rot"]))
    if kind == "realisations":
        return _batch(s["ctx"].realization_solves(s["cfg"], s["occ"], s["rot"]))
    if kind == "agglomerates":
        return [{**_batch(r), "ndip": r["ndip"]} for r in s["group"].agglomerate_solves(s["cfg"], s["mons"])]
    if kind == "linear":
        return s["ctx"].solve_linear(s["occ"], s["alpha"], [0, 1, 1], s["rhs"], err_max=s["err_max"])[0]
    r = s["ctx"].solve_fp64(s["occ"], s["alpha"], [0, 1], s["kd"], (0, 0, 1), (1, 0, 0), s["ksc"],
                            solver=s["solver"], max_step=s["max_step"], err_max=s["err_max"], want_p=True,
                            trace=False)
    return {"esc": r["esc"], "cabs": r["cabs"], "cext": r["cext"], "p": r["p"]}


# -------------------------------------------------------------------------------- its work
def _fft_flops(edges):
    """Real operations of one zero-padded convolution of a 3-component field: six padded
    transforms and the symmetric product."""
    M = 8.0 * edges[0] * edges[1] * edges[2]
    return 6 * 5.0 * M * math.log2(M) + M * 66.0


def work(case):
    """Bytes and operations of one pass: every input read and every output written once
    (octants of the Green tensor; one read of the fields by each of an iteration's matvec),
    transforms and sums as far as the given solver must do them at least once."""
    kind = case["kind"]
    if kind == "agglomerates":
        b = f = 0.0
        for n, c in zip(_ints(case["sizes"]), _ints(case["counts"])):
            na = round(180.0 / case["theta_step"]) + 1
            b += 48.0 * (n + 1) ** 3 + 2 * c * (48.0 + 1) * n ** 3
            f += 2 * c * (_fft_flops((n, n, n)) + 24.0 * na * case["nplanes"] * 0.2 * n ** 3)
        return {"bytes": b, "flops": f}
    e = _grid(case)
    N = float(e[0] * e[1] * e[2])
    octant = 48.0 * (e[0] + 1) * (e[1] + 1) * (e[2] + 1)
    if kind == "convolution":
        return {"bytes": octant + 48.0 * N * case["nrhs"], "flops": case["nrhs"] * _fft_flops(e)}
    if kind == "linear":
        return {"bytes": octant + 10 * 144.0 * N, "flops": 10 * (_fft_flops(e) + 100 * N)}
    na = round(180.0 / case["theta_step"]) + 1
    if kind == "fp64":
        its = 20 if case["solver"] == CG else 16
        return {"bytes": 2 * octant + its * 288.0 * N, "flops": its * (_fft_flops(e) + 100 * N)}
    nrhs = 2.0 if kind == "plain" else 2.0 * case["count"]
    matvecs = 1.0 if case["err_max"] > 5e-4 and case["solver"] == CG else 3.0
    return {"bytes": octant + nrhs * matvecs * 49.0 * N,
            "flops": nrhs * (matvecs * _fft_flops(e) + 24.0 * na * case["nplanes"] * 0.3 * N)}


# ------------------------------------------------------------------- the outputs in double
_DEV = "cuda" if torch.cuda.is_available() else "cpu"


def _t(a, dtype=torch.complex128):
    return torch.as_tensor(np.asarray(a), device=_DEV).to(dtype)


class _Lattice:
    """G * p by dense FFTs on the doubled lattice, in double; the six components of the
    transformed Green tensor are e00, e01, e02, e11, e12, e22."""

    def __init__(self, grid, kd):
        self.grid, self.kd = grid, kd
        x = []
        for n in grid:
            i = torch.arange(2 * n, device=_DEV, dtype=torch.float64)
            x.append(torch.where(i < n, i, i - 2 * n) * kd)
        X = torch.meshgrid(*x, indexing="ij")
        r2 = X[0] ** 2 + X[1] ** 2 + X[2] ** 2
        zero = r2 < 1e-10
        r2 = torch.where(zero, torch.ones_like(r2), r2)
        r = r2.sqrt()
        c2 = torch.polar(1 / (r * r2), r)
        c2[zero] = 0
        off = c2 * torch.complex(3 - r2, -3 * r) / r2
        diag = c2 * torch.complex(r2 - 1, r)
        self.hat = []
        for a, b in ((0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2)):
            g = off * (X[a] * X[b])
            self.hat.append(torch.fft.fftn(g + diag if a == b else g))

    def convolve(self, p, conj=False):
        """p: (3, ni, nj, nl); the conjugate operator uses conj(G)."""
        n = self.grid
        if conj:
            return self.convolve(p.conj()).conj()
        f = torch.fft.fftn(p, s=tuple(2 * v for v in n), dim=(1, 2, 3))
        h = self.hat
        out = []
        for row in ((0, 1, 2), (1, 3, 4), (2, 4, 5)):
            v = h[row[0]] * f[0]
            v += h[row[1]] * f[1]
            v += h[row[2]] * f[2]
            out.append(torch.fft.ifftn(v)[: n[0], : n[1], : n[2]])
        return torch.stack(out)

    def phase(self, k, centre):
        """exp(i k_a (x_a - c_a)) per axis; centre n - 1 or n half spacings."""
        out = []
        for a, n in enumerate(self.grid):
            x = torch.arange(n, device=_DEV, dtype=torch.float64) * self.kd - (n - centre) * self.kd / 2
            out.append(torch.polar(torch.ones_like(x), x * float(k[a])))
        return out

    def plane_wave(self, k, centre=1):
        ex, ey, ez = self.phase(k, centre)
        return ex[:, None, None] * ey[None, :, None] * ez[None, None, :]

    def farfield(self, p, ksc):
        """(ndir, 3): the field of the dipoles p in every direction."""
        k = _t(ksc, torch.float64)
        ph = []
        for a, n in enumerate(self.grid):
            x = torch.arange(n, device=_DEV, dtype=torch.float64) * self.kd - (n - 1) * self.kd / 2
            ph.append(torch.polar(torch.ones((k.shape[0], n), device=_DEV, dtype=torch.float64), k[:, a, None] * x))
        out = []
        for d in range(0, k.shape[0], 128):
            s = slice(d, d + 128)
            t = torch.einsum("cijl,dl->dcij", p, ph[2][s])
            t = torch.einsum("dcij,dj->dci", t, ph[1][s])
            out.append(torch.einsum("dci,di->dc", t, ph[0][s]))
        S = torch.cat(out)
        kc = k.to(torch.complex128)
        return S - kc * (kc * S).sum(1, keepdim=True)

    def sections(self, p, alpha, k, e):
        """Cabs and Cext of the dipoles p; alpha: (ni, nj, nl), 0 off the target."""
        on = alpha != 0
        E = _t(e)
        w = self.plane_wave(-np.asarray(k, float), centre=0)
        pe = (p * E.conj()[:, None, None, None]).sum(0)
        pp = (p.abs() ** 2).sum(0)
        inv = torch.where(on, 1 / torch.where(on, alpha, torch.ones_like(alpha)).conj(), torch.zeros_like(alpha))
        r0 = 4 * PI / float((E.abs() ** 2).sum())
        cext = r0 * float((w * pe)[on].imag.sum())
        cabs = r0 * float((pp * inv.imag - (2.0 / 3.0) * pp)[on].sum())
        return cabs, cext

    def solve(self, alpha, b, solver, err_max, max_step):
        """The solvers' recurrences from p = b, to the mean residual norm err_max, with the
        best iterate kept."""
        on = alpha != 0
        nact = int(on.sum())

        def A(v):
            return torch.where(on, v - alpha * self.convolve(v), torch.zeros_like(v))

        def dot(x, y):
            return (x * y).sum()

        def err(r):
            return float((r.abs() ** 2).sum(0).sqrt().sum()) / nact

        p = b
        r = torch.where(on, -alpha * self.convolve(p), torch.zeros_like(p))
        s = r
        if solver == BICGSTAB:
            g, rho1 = r, dot(r, r)
            h = A(s)
            la = rho1 / dot(g, h)
            r = r - la * h
            w = A(r)
            lw = dot(w, r) / dot(w, w)
            p = p - la * s - lw * r
            r = r - lw * w
        e = err(r)
        best, e_min = p, e
        for step in range(1, max_step + 1):
            if e <= err_max:
                break
            if e < e_min:
                best, e_min = p, e
            if solver == BICGSTAB:
                rho = dot(r, g)
                lb = (rho * la) / (rho1 * lw)
                s = r + lb * s - lb * lw * h
                rho1 = rho
                h = A(s)
                la = rho / dot(g, h)
                r = r - la * h
                w = A(r)
                lw = dot(w, r) / dot(w, w)
                p = p - la * s - lw * r
                r = r - lw * w
            else:
                w = A(s)
                den = dot(s, w)
                a = dot(r, s) / den
                p = p - a * s
                r = r - a * w
                s = r - (dot(r, w) / den) * s
            e = err(r)
        return best if e > e_min else p

    def sample(self, occ, alpha, k, e, solver, err_max, max_step):
        """Dipoles of one incident wave; alpha per material, occ the materials."""
        al = _t(alpha)[_t(occ, torch.int64)]
        b = al * self.plane_wave(k) * _t(e)[:, None, None, None]
        return self.solve(al, b, solver, err_max, max_step), al


def _mueller(k, ksc, normals, e, s):
    """Mueller matrices (angles, 4, 4) averaged over the planes; ksc (planes, angles, 3),
    s the scattered fields of both polarisations (planes, angles, 3)."""
    k, e = np.asarray(k, float), [np.asarray(v, complex) for v in e]
    nv = normals[:, None, :]
    pin = np.cross(k, nv)
    pin = pin / np.linalg.norm(pin, axis=-1, keepdims=True)
    psc = np.cross(ksc, np.broadcast_to(nv, ksc.shape))
    psc = -psc / np.linalg.norm(psc, axis=-1, keepdims=True)
    i0n, i1n, i0p, i1p = (nv * e[0]).sum(-1), (nv * e[1]).sum(-1), (pin * e[0]).sum(-1), (pin * e[1]).sum(-1)
    den = 1j * (i0n * i1p - i1n * i0p)
    s0n, s1n, s0p, s1p = (nv * s[0]).sum(-1), (nv * s[1]).sum(-1), (psc * s[0]).sum(-1), (psc * s[1]).sum(-1)
    A, B = (s1p * i0n - s0p * i1n) / den, (s0p * i1p - s1p * i0p) / den
    C, E = (s1n * i0n - s0n * i1n) / den, (s0n * i1p - s1n * i0p) / den
    aa, bb, cc, dd = (np.abs(v) ** 2 for v in (A, B, C, E))
    c = np.conj
    M = [0.5 * (aa + bb + cc + dd), 0.5 * (aa - bb + cc - dd), (A * c(B) + E * c(C)).real, (A * c(B) - E * c(C)).imag,
         0.5 * (aa + bb - cc - dd), 0.5 * (aa - bb - cc + dd), (A * c(B) - E * c(C)).real, (A * c(B) + E * c(C)).imag,
         (A * c(C) + E * c(B)).real, (A * c(C) - E * c(B)).real, (E * c(A) + B * c(C)).real, (A * c(E) + C * c(B)).imag,
         (C * c(A) + E * c(B)).imag, (C * c(A) - E * c(B)).imag, (E * c(A) - B * c(C)).imag, (E * c(A) - B * c(C)).real]
    return np.stack(M, -1).mean(0).reshape(-1, 4, 4)


def _exact_samples(L, samples, case, solver, model, indices):
    """Cabs, Cext and Mueller matrices of samples (occ, rotation)."""
    normals, ksc = _planes(case["nplanes"], case["theta_step"])
    ca, ce, mm = [], [], []
    for occ, R in samples:
        k, nv, ks = R @ np.array([0.0, 0, 1]), normals @ R.T, ksc @ R.T
        E = [R @ np.array([1.0, 0, 0]), R @ np.array([0, 1.0, 0])]
        esc, c = [], []
        for e in E:
            alpha = np.array([0, *(_alpha(model, L.kd, m, k, e) for m in indices)], np.complex64)
            p, al = L.sample(occ, alpha, k, e, solver, case["err_max"], case["max_step"])
            esc.append(L.farfield(p, ks.reshape(-1, 3)).cpu().numpy().reshape(ks.shape))
            c.append(L.sections(p, al, k, e))
        ca.append(0.5 * (c[0][0] + c[1][0]))
        ce.append(0.5 * (c[0][1] + c[1][1]))
        mm.append(_mueller(k, ks, nv, E, esc))
    return {"cabs": np.array(ca), "cext": np.array(ce), "mueller": np.stack(mm)}


def exact(case, seed):
    kind = case["kind"]
    if kind == "convolution":
        grid = _grid(case)
        L = _Lattice(grid, 2 * 6.0 / max(grid))
        x = _fields(case, seed)
        y = torch.empty(x.shape, dtype=torch.complex128, device=x.device)
        for r in range(case["nrhs"]):
            y[r] = L.convolve(x[r].to(torch.complex128), case["conj"])
        return y
    if kind == "agglomerates":
        m, out = _index(case, seed), []
        for n, c in zip(_ints(case["sizes"]), _ints(case["counts"])):
            L = _Lattice((n, n, n), 2.0 * case["x"] / n)
            g = np.arange(n, dtype=np.float32) - np.float32(n / 2.0 - 0.5)
            samples = []
            for k in range(c):
                occ = np.zeros((n, n, n), np.int8)
                for q in _monomers(n, case["packing"], seed + 1000 * n + k):
                    lo = np.clip(np.floor(q[2:5] - g[0] - 4).astype(int), 0, n)
                    hi = np.clip(lo + 10, 0, n)
                    d = [(g[a:b] - v) ** 2 for a, b, v in zip(lo, hi, q[2:5])]
                    near = d[0][:, None, None] + d[1][None, :, None] + d[2][None, None, :] <= q[0] ** 2
                    occ[lo[0]:hi[0], lo[1]:hi[1], lo[2]:hi[2]] |= near.astype(np.int8)
                r2 = g[:, None, None] ** 2 + g[None, :, None] ** 2 + g[None, None, :] ** 2
                occ[r2 > (n / 2.0) ** 2] = 0
                samples.append((occ, np.eye(3)))
            out.append({**_exact_samples(L, samples, case, CG, CM, [m]), "ndip": None})
            del L
        return out
    grid, kd = _grid(case), _spacing(case)
    L = _Lattice(grid, kd)
    if kind == "orientations":
        occ = _ellipsoid(grid, case["b_a"], case["c_a"])
        samples = [(occ, R) for R in _rotations(case["count"], case["mc"], seed)]
        return _exact_samples(L, samples, case, case["solver"], case["model"], [_index(case, seed)])
    if kind == "realisations":
        rot = _rotations(case["count"], True, seed)
        samples = [(_porous(grid, case["packing"], seed + 1000 * (k + 1)), rot[k]) for k in range(case["count"])]
        return _exact_samples(L, samples, case, case["solver"], case["model"], [complex(np.float32(m.real), np.float32(m.imag)) for m in _POROUS])
    if kind == "linear":
        occ, alpha, rhs = _linear_rhs(case, seed)
        al = _t(alpha)[_t(occ, torch.int64)]
        b = _t(rhs).permute(3, 0, 1, 2)
        x = L.solve(al, b, CG, 1e-13, 200)
        return x.permute(1, 2, 3, 0).contiguous()
    occ, m, k = _ellipsoid(grid, case["b_a"], case["c_a"]), _index(case, seed), (0, 0, 1)
    if kind == "plain":
        normals, ksc = _planes(case["nplanes"], case["theta_step"])
        ksc, E = ksc.astype(np.float32).astype(float), ((1, 0, 0), (0, 1, 0))
        out = {"esc": [], "cabs": [], "cext": []}
        for e in E:
            alpha = np.array([0, _alpha(case["model"], kd, m, k, e)], np.complex64)
            p, al = L.sample(occ, alpha, k, e, case["solver"], case["err_max"], case["max_step"])
            out["esc"].append(L.farfield(p, ksc.reshape(-1, 3)).cpu().numpy().reshape(ksc.shape))
            ca, ce = L.sections(p, al, k, e)
            out["cabs"].append(ca)
            out["cext"].append(ce)
        out["mueller"] = _mueller(k, ksc, normals, E, out["esc"])
        return out
    alpha = np.array([0, _alpha(CMRR, kd, m, k, (1, 0, 0))])
    p, al = L.sample(occ, alpha, k, (1, 0, 0), case["solver"], case["err_max"], case["max_step"])
    ca, ce = L.sections(p, al, k, (1, 0, 0))
    _, ksc = _planes(1, case["theta_step"])
    return {"esc": L.farfield(p, ksc[0]), "cabs": ca, "cext": ce, "p": p.permute(1, 2, 3, 0).contiguous()}
