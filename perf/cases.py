"""Timed cases of the self-consistent dipole / quadrupole solve.

Every case is work that a program of this package's users asks for through
its public entry points: whole spectra (``dipole_solver``), batched solves
and single operator applications on device tensors (``capi.Field``), near
fields (``Near_Field``) and gradients (``adjoint.extinction_loss``).  The
spheres are those of the benchmark: Drude metal (eps_inf 4, omega_p 1.8 eV,
gamma 0.1 eV), hexagonal monolayers of radius 5 nm at 12 nm spacing, random
packings of equal spheres (volume fraction 0.1) or of radii 1-4 nm (0.15),
rock-salt lattices and open clusters.  Lengths handed to ``capi.Field`` are in
units of the smallest radius.

``exact`` gives the answers in 64 bits from the physics, by other means than
the package's: spheres that do not overlap interact as point dipoles, so a
plain Ewald sum (own splitting parameter, structure factors over the wave
vectors themselves, no grid) or a plain pair sum gives the operator, and dense
LU the solution.  It therefore differs from any correct output by the spectral
discretisation that the caller's Ewald tolerance asks for (about 1e-5 for equal
spheres at 1e-6, 2e-3 for radii that differ fourfold) and, for solves, by the
solve's tolerance.
"""
import math

import numpy as np
import torch

import cumpm_b200 as cuMPM
from cumpm_b200 import adjoint, capi

EPS_M = 1.77
XI = 0.5
EWALD_TOL = 1e-6


# ------------------------------------------------------------------ cases


def listed():
    return [
        # an isolated cluster's spectrum, whole call: the smallest system a
        # program solves; launches and host work count
        {"name": "cluster_spectrum", "kind": "cluster", "n": 100, "freqs": 10, "solver": "gmres", "precision": "auto"},
        # one operator application of an open system in double precision, as
        # the gradient of an open cluster applies it
        {"name": "open_apply", "kind": "open", "n": 2000, "cols": 30, "fp32": False},
        # the monolayer's operator on the batch of a 10-frequency spectrum
        {"name": "layer_apply", "kind": "layer", "n": 4000, "cols": 30, "fp32": True},
        # a 3-D packing at one frequency: three polarisations, default precision
        {"name": "packing_apply", "kind": "packing", "n": 8000, "cols": 3, "fp32": True},
        # dipoles and quadrupoles of a packing, four frequencies at once
        {"name": "quadrupole_apply", "kind": "quads", "n": 2000, "cols": 12, "fp32": True},
        # the polydisperse operator on 16 frequencies
        {"name": "poly_apply", "kind": "poly", "n": 1000, "cols": 48, "fp32": True},
        # one right-hand side, plain double-precision solve
        {"name": "packing_solve", "kind": "packing_solve", "n": 500, "cols": 1},
        # the benchmark's headline: 30 right-hand sides of the monolayer
        {"name": "layer_solve", "kind": "layer_solve", "n": 4000, "freqs": 10},
        # the polydisperse packing's 192 right-hand sides
        {"name": "poly_solve", "kind": "poly_solve", "n": 1000, "freqs": 64},
        # a design loop's step: loss and all gradients of a rock-salt crystal
        {"name": "gradient", "kind": "gradient", "cells": 8, "layers": 8, "freqs": 8},
        # an intensity map above a monolayer
        {"name": "near_field", "kind": "near", "n": 1000, "points": 10000},
        # the reference's own benchmark script: the monolayer's spectrum at
        # the default tolerance, one frequency after another, whole call
        {"name": "layer_spectrum", "kind": "sweep", "n": 4000, "freqs": 10, "solver": "gmres", "batched": False},
    ]


def _log(rng, lo, hi):
    """A whole number spread over the logarithm of [lo, hi]."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["cluster", "open", "layer", "packing", "quads", "poly", "packing_solve", "layer_solve",
                       "poly_solve", "gradient", "near", "sweep"])
    if kind == "cluster":
        return {"kind": kind, "n": _log(rng, 20, 400), "freqs": rng.randint(3, 16),
                "solver": rng.choice(["gmres", "bicgstab"]), "precision": rng.choice(["auto", "double"])}
    if kind == "open":
        return {"kind": kind, "n": _log(rng, 100, 3000), "cols": _log(rng, 1, 30), "fp32": rng.random() < 0.5}
    if kind == "layer":
        return {"kind": kind, "n": _log(rng, 500, 4000), "cols": _log(rng, 1, 30), "fp32": rng.random() < 0.7}
    if kind == "packing":
        return {"kind": kind, "n": _log(rng, 300, 8000), "cols": _log(rng, 1, 6), "fp32": rng.random() < 0.7}
    if kind == "quads":
        return {"kind": kind, "n": _log(rng, 200, 2000), "cols": _log(rng, 1, 12), "fp32": rng.random() < 0.7}
    if kind == "poly":
        return {"kind": kind, "n": _log(rng, 200, 1000), "cols": _log(rng, 1, 48), "fp32": rng.random() < 0.7}
    if kind == "packing_solve":
        return {"kind": kind, "n": _log(rng, 250, 1500), "cols": rng.randint(1, 3)}
    if kind == "layer_solve":
        return {"kind": kind, "n": _log(rng, 800, 4000), "freqs": rng.randint(2, 10)}
    if kind == "poly_solve":
        return {"kind": kind, "n": _log(rng, 250, 1000), "freqs": _log(rng, 4, 64)}
    if kind == "gradient":
        cells, layers = rng.choice([(6, 6), (6, 8), (6, 10), (6, 12), (6, 14), (8, 6), (8, 8)])
        return {"kind": kind, "cells": cells, "layers": layers, "freqs": rng.randint(2, 8)}
    if kind == "near":
        return {"kind": kind, "n": _log(rng, 500, 2000), "points": _log(rng, 500, 10000)}
    return {"kind": kind, "n": _log(rng, 500, 4000), "freqs": rng.randint(3, 10),
            "solver": rng.choice(["gmres", "bicgstab"]), "batched": rng.random() < 0.3}


# ----------------------------------------------------------------- inputs


def _rng(case, seed):
    return np.random.default_rng([int(seed), sum(map(ord, case["kind"])), int(case.get("n", case.get("cells", 0)))])


def _drude(omega):
    return 4.0 - 1.8 ** 2 / (omega ** 2 + 1j * omega * 0.1)


def _hex(n, spacing, rng, jitter):
    """Rows of 2*ceil(sqrt(n)) sites, odd rows shifted, each site moved in the
    plane by up to jitter (all at z = 0)."""
    lim = int(np.ceil(np.sqrt(n))) * 2
    j, i = np.divmod(np.arange(n), lim)
    pos = np.stack([(i + 0.5 * (j % 2)) * spacing, j * (np.sqrt(3) / 2) * spacing, np.zeros(n)], axis=1)
    pos[:, :2] += rng.uniform(-jitter, jitter, (n, 2))
    return pos


def _layer(case, rng):
    """The benchmark's monolayer (nm) and its box."""
    n = case["n"]
    pos = _hex(n, 12.0, rng, 0.5)
    lim = int(np.ceil(np.sqrt(n))) * 2
    rows = (n + lim - 1) // lim
    least = 2.1 * 5.256522 * 5.0
    box = np.array([max((lim + 0.5) * 12.0, least), max(rows * 12.0 * np.sqrt(3) / 2, 80.0, least), 1000.0])
    return pos, box


def _packing(radii, phi, rng):
    """Random non-overlapping spheres in a periodic cube: rounds of random
    sequential addition, a candidate is dropped when it meets a placed sphere
    or an earlier candidate of its round."""
    n = len(radii)
    L = float((np.sum(4.0 / 3.0 * np.pi * radii ** 3) / phi) ** (1.0 / 3.0))
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    order = np.argsort(-radii, kind="stable")            # the largest first
    rad = torch.tensor(radii[order], device=dev)
    pos = torch.zeros((n, 3), dtype=torch.float64, device=dev)
    placed = torch.zeros(n, dtype=torch.bool, device=dev)
    while not bool(placed.all()):
        todo = torch.nonzero(~placed).flatten()[:4096]
        new = torch.tensor(rng.uniform(0, L, (len(todo), 3)), device=dev)
        pos[todo] = new
        live = placed.clone()
        live[todo] = True
        d2 = torch.zeros((len(todo), n), dtype=torch.float64, device=dev)
        for c in range(3):
            d = new[:, c, None] - pos[None, :, c]
            d2 += (d - L * torch.round(d / L)) ** 2
        hit = (d2 < (rad[todo][:, None] + rad[None, :]) ** 2) & live[None, :]
        rank = torch.arange(n, device=dev)
        hit &= placed[None, :] | (rank[None, :] < todo[:, None])
        placed[todo] = ~hit.any(dim=1)
    out = np.empty((n, 3))
    out[order] = pos.cpu().numpy()
    return out, np.array([L, L, L])


def _radii(n, rng):
    """Radii spread evenly over 1-4 nm, in random order."""
    return rng.permutation(np.linspace(1.0, 4.0, n))


def _problem(case, seed):
    """The case's host inputs (numpy), from the seed alone."""
    rng = _rng(case, seed)
    kind = case["kind"]
    p = {"rng": rng}
    if kind in ("layer", "layer_solve", "sweep", "near"):
        p["pos"], p["box"] = _layer(case, rng)
        p["radius"] = np.full(case["n"], 5.0)
    elif kind in ("packing", "quads", "packing_solve"):
        p["radius"] = np.full(case["n"], 5.0)
        p["pos"], p["box"] = _packing(p["radius"], 0.10, rng)
    elif kind in ("poly", "poly_solve"):
        p["radius"] = _radii(case["n"], rng)
        p["pos"], p["box"] = _packing(p["radius"], 0.15, rng)
    elif kind in ("cluster", "open"):
        p["radius"] = np.full(case["n"], 5.0) if kind == "cluster" else _radii(case["n"], rng)
        p["pos"], p["box"] = _packing(p["radius"], 0.10, rng)
    elif kind == "gradient":
        n = case["cells"]
        sites = [np.arange(n), np.arange(n), np.arange(case["layers"])]
        g = np.stack(np.meshgrid(*sites, indexing="ij"), axis=-1).reshape(-1, 3)
        p["pos"] = g * 7.0 + rng.uniform(-0.3, 0.3, (len(g), 3))
        p["box"] = np.array([n, n, case["layers"]]) * 7.0
        p["species"] = np.where(g.sum(axis=1) % 2 == 0, 0, -1)
        p["radius"] = np.where(p["species"] == 0, 3.0, 2.0) * rng.uniform(0.98, 1.02, len(g))
    p["unit"] = float(p["radius"].min())
    return p


def _columns(case, p):
    """Moments, right-hand sides and self coefficients of the device cases,
    [row][column] as the operator takes them (units of the smallest radius)."""
    n = len(p["pos"])
    rng = p["rng"]
    a3 = (p["radius"] / p["unit"]) ** 3
    if "freqs" in case:
        omega = np.linspace(0.2, 1.2 if case["kind"] == "poly_solve" else 1.0, case["freqs"])
        m, k = 3 * case["freqs"], 3
    else:
        m, k = case["cols"], min(3, case["cols"])
        omega = np.array([0.5]) if case["kind"] == "packing_solve" else np.linspace(0.2, 1.0, -(-m // k))
    eps = np.repeat(_drude(omega), k)[:m] / EPS_M
    p["self"] = 3.0 / (4 * np.pi * (eps[None, :] - 1.0)) / a3[:, None]
    B = np.zeros((3 * n, m), complex)
    for c in range(m):
        B[c % k::3, c] = 1.0
    phi = np.sum(4.0 / 3.0 * np.pi * a3) / np.prod(p["box"] / p["unit"])
    beta = (eps - 1) / (eps + 2)
    p["rhs"] = B
    p["guess"] = B * (4 * np.pi * beta / (1 - beta * phi))[None, :] * np.repeat(a3, 3)[:, None]
    rows = 3 * n + (5 * n if case["kind"] == "quads" else 0)
    p["moments"] = rng.standard_normal((rows, m)) + 1j * rng.standard_normal((rows, m))


def _dev(a):
    return torch.tensor(a, dtype=torch.complex128, device="cuda")


def _near_points(case, p):
    """A regular map of points at random height 3-4 radii above the layer."""
    k = int(math.ceil(math.sqrt(case["points"])))
    u = (np.arange(k) + p["rng"].uniform()) / k
    xy = np.stack(np.meshgrid(u * p["box"][0], u * p["box"][1], indexing="ij"), axis=-1).reshape(-1, 2)
    z = p["rng"].uniform(15.0, 20.0)
    return np.concatenate([xy, np.full((len(xy), 1), z)], axis=1)[:case["points"]]


def prepare(case, seed):
    p = _problem(case, seed)
    kind = case["kind"]
    s = {"case": case, "pos": p["pos"] / p["unit"]}
    if kind in ("open", "layer", "packing", "quads", "poly", "packing_solve", "layer_solve", "poly_solve"):
        _columns(case, p)
        box, rad = p["box"] / p["unit"], p["radius"] / p["unit"]
        if kind == "open":
            s["field"] = capi.Field(capi.FIELD_DIRECT, radius=rad)
        elif kind in ("poly", "poly_solve"):
            s["field"] = capi.Field(capi.FIELD_POLY, box, EWALD_TOL, XI, radius=rad)
        else:
            s["field"] = capi.Field(capi.FIELD_MONO, box, EWALD_TOL, XI, solve_quads=kind == "quads")
        s["self"] = _dev(p["self"])
        if kind.endswith("_solve"):
            s["rhs"], s["guess"] = _dev(p["rhs"]), _dev(p["guess"])
            s["x"] = torch.empty_like(s["guess"])
        else:
            s["moments"] = _dev(p["moments"])
            s["field"].set_positions(s["pos"])
    elif kind in ("cluster", "sweep"):
        s["pos_nm"], s["box"] = p["pos"], p["box"]
        omega = np.linspace(0.2, 1.0, case["freqs"])
        s["eps"] = _drude(omega)
    elif kind == "gradient":
        t = lambda v: torch.tensor(v, dtype=torch.float64, requires_grad=True)  # noqa: E731
        s["leaves"] = [t(p["pos"]), t(p["radius"]), t([1.8]), t([0.1])]
        s["args"] = _gradient_args(case, p)
    else:
        rng = p["rng"]
        pts = _near_points(case, p)
        dip = (rng.standard_normal((case["n"], 3)) + 1j * rng.standard_normal((case["n"], 3))) * 200.0
        s["near"] = cuMPM.Near_Field(p["box"], [1.0, 0.0, 0.0], radius=5.0, dip=dip, dip_pos=p["pos"],
                                     field_points=pts, xi=XI, errortol=EWALD_TOL)
    return s


def _gradient_args(case, p):
    omega = np.linspace(0.3, 1.0, case["freqs"])
    return dict(box=p["box"], omega=omega, species=p["species"], eps_inf=[4.0], eps_m=EPS_M,
                eps_const=np.where(p["species"] < 0, 2.5, 0.0).astype(complex), E0=((1.0, 0.0, 0.0),),
                wavenumber=adjoint.wavenumber_from_ev(omega, EPS_M), tol=EWALD_TOL, solve_tol=1e-9)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("open", "layer", "packing", "quads", "poly"):
        return state["field"].apply(state["moments"], self_coef=state["self"], recip_fp32=case["fp32"])
    if kind == "packing_solve":
        state["field"].set_positions(state["pos"])
        state["x"].copy_(state["guess"])
        state["field"].batch_solve(state["rhs"], state["x"], state["self"], tol=1e-6, restart=30, recip_fp32=False)
        return state["x"]
    if kind in ("layer_solve", "poly_solve"):
        state["field"].set_positions(state["pos"])
        state["x"].copy_(state["guess"])
        state["field"].batch_solve(state["rhs"], state["x"], state["self"], tol=1e-6, refine=True)
        return state["x"]
    if kind == "cluster":
        d = cuMPM.dipole_solver(state["box"], state["eps"], radius=5.0, eps_m=EPS_M, tol=1e-6, quiet=True,
                                field_type="direct", solver_type=case["solver"], precision=case["precision"])
        d.compute(state["pos_nm"])
        return [d.get_eff_polarizability(), d.get_dipoles()]
    if kind == "sweep":
        d = cuMPM.dipole_solver(state["box"], state["eps"], radius=5.0, eps_m=EPS_M, tol=1e-3, quiet=True,
                                solver_type=case["solver"])
        if case["batched"]:
            d.set_solver_options(batch_all=True, refine=True)
        d.compute(state["pos_nm"])
        return [d.get_eff_polarizability(), d.get_dipoles()]
    if kind == "gradient":
        for t in state["leaves"]:
            t.grad = None
        loss = adjoint.extinction_loss(*state["leaves"], **state["args"])
        loss.backward()
        return [loss.detach()] + [t.grad for t in state["leaves"]]
    return state["near"].calculate()


# ------------------------------------------------------- work, tolerances


def work(case):
    """Inputs read and outputs written once; operations of the method: the
    pair sum (open systems: all pairs; periodic: those within the cutoff) and
    spread, transforms and contraction on the grid that the Ewald tolerance
    asks for, times the operator applications that a solve needs at least."""
    kind = case["kind"]
    n = case["cells"] ** 2 * case["layers"] if kind == "gradient" else case["n"]
    m = 3 * case["freqs"] if kind in ("cluster", "sweep", "layer_solve", "poly_solve") else case.get("cols", 1)
    if kind == "gradient":
        m = case["freqs"]
    rows = 8 * n if kind == "quads" else 3 * n
    out = 16 * rows * m
    bytes_ = {"near": 16 * 3 * n + 24 * (n + case.get("points", 0)) + 8 * case.get("points", 0),
              "gradient": 8 * 4 * n * 2, "cluster": 24 * n + out, "sweep": 24 * n + out,
              "packing_solve": 3 * out + 16 * n * m + 24 * n, "layer_solve": 3 * out + 16 * n * m + 24 * n,
              "poly_solve": 3 * out + 16 * n * m + 24 * n}.get(kind, 2 * out + 16 * n * m)
    # applications: iterations to the tolerance, on the distinct right-hand
    # sides where the frequencies share their Krylov space
    applies, cols = {"cluster": (8, m), "packing_solve": (6, m), "layer_solve": (13, 3), "poly_solve": (13, 3),
                     "gradient": (20, m), "sweep": (4, m)}.get(kind, (1, m))
    if kind in ("cluster", "open"):
        flops = 60.0 * n * n
    elif kind == "near":
        flops = 60.0 * 40 * case["points"] + 8 * 27 * (n + case["points"])
    else:
        comps = 1 if kind in ("poly", "poly_solve", "gradient") else 8 if kind == "quads" else 3
        support = 12 ** 3 if comps == 1 else 81 if kind in ("layer", "layer_solve", "sweep") else 9 ** 3
        pts = {"layer": 7.0, "layer_solve": 7.0, "sweep": 4.0, "poly": 1260.0, "poly_solve": 1260.0,
               "gradient": 200.0}.get(kind, 70.0) * n
        flops = 60.0 * 15 * n + comps * (8.0 * support * n + 10.0 * pts * math.log2(pts))
    return {"bytes": float(bytes_), "flops": float(flops * applies * cols)}


def tolerance(case):
    return _TOLERANCE[case["kind"]](case)


# An operator application in 32-bit reciprocal space against one in 64 bits:
# 2.5e-8 of the whole (the self terms and pairs are in 64 bits), 2e-7 for the
# worst value; the open sum in 32 bits 6e-8 and 1.8e-6 (close pairs); in 64
# bits 1e-16.  Solves against a solution at 1e-11 on the double operator:
# 5e-8 to 5e-7 by where the last step lands below the tolerance, 2e-5 for the
# worst value.  Spectra at 1e-3 by GMRES against BiCGSTAB: 5e-5 and 1e-3.
# Four times these, about.
_APPLY32, _APPLY64 = {"rel": 1e-7, "max": 1e-6}, {"rel": 1e-14, "max": 1e-13}

_TOLERANCE = {
    "open": lambda c: {"rel": 3e-7, "max": 8e-6} if c["fp32"] else _APPLY64,
    "layer": lambda c: _APPLY32 if c["fp32"] else _APPLY64,
    "packing": lambda c: _APPLY32 if c["fp32"] else _APPLY64,
    "quads": lambda c: _APPLY32 if c["fp32"] else _APPLY64,
    "poly": lambda c: _APPLY32 if c["fp32"] else _APPLY64,
    "cluster": lambda c: {"rel": 1.2e-6, "max": 2e-5},
    "packing_solve": lambda c: {"rel": 1e-6, "max": 1e-5},
    "layer_solve": lambda c: {"rel": 2e-6, "max": 2e-5},
    "poly_solve": lambda c: {"rel": 2e-6, "max": 1e-4},
    "gradient": lambda c: {"rel": 5e-10, "max": 5e-9},
    "near": lambda c: {"rel": 1e-6, "max": 1e-5},
    "sweep": lambda c: {"rel": 1e-3, "max": 1e-2} if c["batched"] else {"rel": 2e-4, "max": 4e-3},
}


# ------------------------------------------------------------------ exact


_ACC = 5.3      # erfc and Gaussian cut: exp(-5.3^2) = 6e-13


class _Ewald:
    """Point-dipole Ewald sum of a periodic box (conducting boundary, no mean
    field), in units of 1 / (4 pi eps_0) = 1 / (4 pi)."""

    def __init__(self, box, dev):
        self.box = torch.tensor(np.asarray(box, float), device=dev)
        self.rc = float(np.min(box)) / 2 * (1 - 1e-12)
        self.alpha = _ACC / self.rc
        self.volume = float(np.prod(box))
        kmax = 2 * self.alpha * _ACC
        g = [np.arange(-int(kmax * L / (2 * np.pi)), int(kmax * L / (2 * np.pi)) + 1) * 2 * np.pi / L for L in box]
        k = np.stack(np.meshgrid(*g, indexing="ij"), axis=-1).reshape(-1, 3)
        k2 = np.sum(k * k, axis=1)
        # half of the wave vectors, each standing for +k and -k
        half = (k[:, 0] > 0) | ((k[:, 0] == 0) & ((k[:, 1] > 0) | ((k[:, 1] == 0) & (k[:, 2] > 0))))
        keep = half & (k2 <= kmax * kmax)
        self.k = torch.tensor(k[keep], device=dev)
        self.k2 = torch.sum(self.k * self.k, dim=1)
        self.green = 2.0 * torch.exp(-self.k2 / (4 * self.alpha ** 2)) / (self.k2 * self.volume)

    def pair_tensor(self, src, tgt, same):
        """Screened pair tensor T (nt, ns, 3, 3): field at tgt = T p."""
        d = src[None, :, :] - tgt[:, None, :]
        d = d - self.box * torch.round(d / self.box)
        r2 = torch.sum(d * d, dim=-1)
        out = r2 > self.rc ** 2
        if same is not None:
            out = out | same
        r2 = torch.where(out, torch.ones_like(r2), r2)
        r, a = torch.sqrt(r2), self.alpha
        ex = 2 * a / math.sqrt(math.pi) * torch.exp(-a * a * r2)
        b = torch.erfc(a * r) / (r2 * r) + ex / r2
        c = 3 * b / r2 + 2 * a * a * ex / r2
        b = torch.where(out, torch.zeros_like(b), b)
        c = torch.where(out, torch.zeros_like(c), c)
        eye = torch.eye(3, dtype=d.dtype, device=d.device)
        return (c[..., None, None] * d[..., :, None] * d[..., None, :] - b[..., None, None] * eye) / (4 * math.pi)

    def self_field(self):
        return 4 * self.alpha ** 3 / (3 * math.sqrt(math.pi)) / (4 * math.pi)

    def waves(self, chunk):
        for c0 in range(0, len(self.k), chunk):
            yield self.k[c0:c0 + chunk], self.green[c0:c0 + chunk]

    def wave_field(self, src, tgt, P):
        """k-space field at tgt of moments P (ns, 3, m) complex."""
        E = torch.zeros((len(tgt), 3, P.shape[2]), dtype=P.dtype, device=P.device)
        for k, g in self.waves(max(1, int(3e7 / max(len(src), len(tgt), 16 * P.shape[2])))):
            ps, pt = src @ k.T, tgt @ k.T
            kp = torch.einsum("kc,scm->skm", k.to(P.dtype), P)
            c, s = torch.cos(ps), torch.sin(ps)
            a = torch.einsum("sk,skm->km", c.to(P.dtype), kp) * g[:, None]
            b = torch.einsum("sk,skm->km", s.to(P.dtype), kp) * g[:, None]
            ct, st = torch.cos(pt).to(P.dtype), torch.sin(pt).to(P.dtype)
            for d in range(3):
                w = k[:, d, None].to(P.dtype)
                E[:, d] -= ct @ (a * w) + st @ (b * w)
        return E

    def field(self, pos, P):
        """Field at the particles of all others and of all images."""
        E = self.wave_field(pos, pos, P) + self.self_field() * P
        chunk = max(1, int(2e6 / len(pos)))
        idx = torch.arange(len(pos), device=pos.device)
        for c0 in range(0, len(pos), chunk):
            T = self.pair_tensor(pos, pos[c0:c0 + chunk], idx[c0:c0 + chunk, None] == idx[None, :])
            T = T.permute(0, 2, 1, 3).reshape(-1, 3 * len(pos)).to(P.dtype)
            E[c0:c0 + chunk] += (T @ P.reshape(3 * len(pos), -1)).reshape(-1, 3, P.shape[2])
        return E

    def matrix(self, pos):
        """The (3n, 3n) real matrix of field()."""
        n = len(pos)
        A = torch.zeros((n, 3, n, 3), dtype=torch.float64, device=pos.device)
        chunk = max(1, int(2e6 / n))
        idx = torch.arange(n, device=pos.device)
        for c0 in range(0, n, chunk):
            T = self.pair_tensor(pos, pos[c0:c0 + chunk], idx[c0:c0 + chunk, None] == idx[None, :])
            A[c0:c0 + chunk] = T.permute(0, 2, 1, 3)
        for k, g in self.waves(max(1, int(6e7 / n))):
            ph = pos @ k.T
            c, s = torch.cos(ph), torch.sin(ph)
            for i in range(3):
                for j in range(i, 3):
                    w = g * k[:, i] * k[:, j]
                    v = (c * w) @ c.T + (s * w) @ s.T
                    A[:, i, :, j] -= v
                    if i != j:
                        A[:, j, :, i] -= v
        A = A.reshape(3 * n, 3 * n)
        A += self.self_field() * torch.eye(3 * n, dtype=A.dtype, device=A.device)
        return A


def _open_tensor(src, tgt, same):
    d = src[None, :, :] - tgt[:, None, :]
    r2 = torch.sum(d * d, dim=-1)
    r2 = torch.where(same, torch.ones_like(r2), r2)
    r3 = r2 * torch.sqrt(r2)
    eye = torch.eye(3, dtype=d.dtype, device=d.device)
    T = (3 * d[..., :, None] * d[..., None, :] / r2[..., None, None] - eye) / r3[..., None, None] / (4 * math.pi)
    return torch.where(same[..., None, None], torch.zeros_like(T), T)


def _open_matrix(pos):
    n = len(pos)
    idx = torch.arange(n, device=pos.device)
    T = _open_tensor(pos, pos, idx[:, None] == idx[None, :])
    return T.permute(0, 2, 1, 3).reshape(3 * n, 3 * n)


def _solve_columns(field_matrix, a, self_, rhs):
    """x with (s + 1 / (4 pi a^3) - T) x = b per column; columns that share
    their self coefficients share a factorisation."""
    diag0 = (1.0 / (4 * math.pi * a ** 3)).repeat_interleave(3)
    X = torch.empty_like(rhs)
    m = rhs.shape[1]
    c = 0
    while c < m:
        e = c
        while e < m and torch.equal(self_[:, e], self_[:, c]):
            e += 1
        A = (-field_matrix).to(torch.complex128)
        A.diagonal().add_(diag0 + self_[:, c].repeat_interleave(3))
        X[:, c:e] = torch.linalg.solve(A, rhs[:, c:e])
        del A
        c = e
    return X


def exact(case, seed):
    kind = case["kind"]
    # the quadrupole operator takes its dipole-quadrupole couplings with one
    # sign in its pair sum and the other in its wave sum, as the program it
    # replaces does: it is no Ewald sum of one interaction, so no independent
    # value exists
    if kind == "quads":
        return None
    # the polydisperse rule cuts the largest spheres' profiles off at 2e-3 of
    # the operator (see poly_apply), and the resonances of a whole spectrum
    # carry that to a tenth of the solution: a value from the physics would
    # not show what the arithmetic does
    if kind == "poly_solve":
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    f8 = lambda v: torch.tensor(np.asarray(v, dtype=np.float64), device=dev)  # noqa: E731
    p = _problem(case, seed)
    pos, box, a = p["pos"] / p["unit"], p["box"] / p["unit"], f8(p["radius"] / p["unit"])
    if kind in ("open", "layer", "packing", "poly", "packing_solve", "layer_solve"):
        _columns(case, p)
        S = torch.tensor(p["self"], device=dev)
        if kind.endswith("_solve"):
            A = _Ewald(box, dev).matrix(f8(pos))
            return _solve_columns(A, a, S, torch.tensor(p["rhs"], device=dev))
        P = torch.tensor(p["moments"], device=dev).reshape(len(pos), 3, -1)
        if kind == "open":
            E = (_open_matrix(f8(pos)).to(P.dtype) @ P.reshape(3 * len(pos), -1)).reshape(P.shape)
        else:
            E = _Ewald(box, dev).field(f8(pos), P)
        Y = (S + 1.0 / (4 * math.pi * a[:, None] ** 3))[:, None, :] * P - E
        return Y.reshape(3 * len(pos), -1)
    if kind in ("cluster", "sweep"):
        W = case["freqs"]
        eps = _drude(np.linspace(0.2, 1.0, W)) / EPS_M
        n = len(pos)
        A = _open_matrix(f8(pos)) if kind == "cluster" else _Ewald(box, dev).matrix(f8(pos))
        S = torch.tensor(np.repeat(3.0 / (4 * np.pi * (eps - 1.0)), 3)[None, :] * np.ones((n, 1)), device=dev)
        rhs = torch.zeros((3 * n, 3 * W), dtype=torch.complex128, device=dev)
        for c in range(3 * W):
            rhs[c % 3::3, c] = 1.0
        X = _solve_columns(A, a, S, rhs).reshape(n, 3, W, 3).permute(2, 0, 3, 1) * (EPS_M * p["unit"] ** 3)
        X = X.cpu().numpy()                                # (W, n, polarisation, 3)
        return [X.mean(axis=1), X]
    if kind == "gradient":
        return _exact_gradient(case, p, dev)
    # near field: |E + E0|^2 with E = (pair part) - (wave part), the signs the
    # interaction field is defined with; the wave part is the Gaussian-screened
    # sum over the spheres' form factors at the splitting parameter XI, the pair
    # part the rest of the whole field
    rng = p["rng"]
    pts = f8(_near_points(case, p) / p["unit"])
    n = case["n"]
    dip = (rng.standard_normal((n, 3)) + 1j * rng.standard_normal((n, 3))) * 200.0
    P = torch.tensor(dip, device=dev).reshape(n, 3, 1)
    ew = _Ewald(box, dev)
    src = f8(pos)
    whole = ew.wave_field(src, pts, P)
    for c0 in range(0, len(pts), 2000):
        T = ew.pair_tensor(src, pts[c0:c0 + 2000], None).permute(0, 2, 1, 3).reshape(-1, 3 * n).to(P.dtype)
        whole[c0:c0 + 2000] += (T @ P.reshape(3 * n, 1)).reshape(-1, 3, 1)
    wave = _Ewald(box, dev)
    wave.alpha = XI
    kmax = 2 * XI * 4.6
    g = [np.arange(-int(kmax * L / (2 * np.pi)), int(kmax * L / (2 * np.pi)) + 1) * 2 * np.pi / L for L in box]
    k = np.stack(np.meshgrid(*g, indexing="ij"), axis=-1).reshape(-1, 3)
    k2 = np.sum(k * k, axis=1)
    half = (k[:, 0] > 0) | ((k[:, 0] == 0) & ((k[:, 1] > 0) | ((k[:, 1] == 0) & (k[:, 2] > 0))))
    keep = half & (k2 <= kmax * kmax)
    wave.k = f8(k[keep])
    k1 = torch.sqrt(torch.sum(wave.k ** 2, dim=1))
    form = 3 * (torch.sin(k1) / k1 - torch.cos(k1)) / (k1 * k1)      # 3 j1(k) / k
    wave.green = 2.0 * torch.exp(-k1 ** 2 / (4 * XI ** 2)) * form ** 2 / (k1 ** 2 * wave.volume)
    recip = wave.wave_field(src, pts, P)
    # in the operator's sign (field = -E): wave part -recip, pair part -(whole - recip)
    E = (recip - (whole - recip))[:, :, 0]
    E0 = torch.tensor([1.0, 0.0, 0.0], dtype=E.dtype, device=dev)
    return torch.sum(torch.abs(E + E0) ** 2, dim=1).cpu().numpy()


def _exact_gradient(case, p, dev):
    """Loss and gradients of the summed extinction: dense solves of the
    problem and of its adjoint, then derivatives of the bilinear form
    lambda^T A p by automatic differentiation of the plain sums."""
    args = _gradient_args(case, p)
    omega, species = args["omega"], p["species"]
    n, unit = len(species), p["unit"]
    f8 = lambda v: torch.tensor(np.asarray(v, dtype=np.float64), device=dev)  # noqa: E731
    pos = f8(p["pos"]).requires_grad_(True)
    rad = f8(p["radius"]).requires_grad_(True)
    wp = f8([1.8]).requires_grad_(True)
    gm = f8([0.1]).requires_grad_(True)
    drude = torch.tensor(species == 0, device=dev)

    def self_coef():
        """s + 1 / (4 pi a^3), (n, frequencies)."""
        w = f8(omega)[None, :]
        e = (4.0 - wp ** 2 / (w * w + 1j * w * gm)).expand(n, -1)
        e = torch.where(drude[:, None], e, torch.full_like(e, 2.5)) / EPS_M
        a3 = (rad / unit)[:, None] ** 3
        return 3.0 / (4 * math.pi * (e - 1.0) * a3) + 1.0 / (4 * math.pi * a3)

    ew = _Ewald(p["box"] / unit, dev)
    W = len(omega)
    with torch.no_grad():
        D = self_coef()
        T = ew.matrix(pos / unit)
        B = torch.zeros((3 * n, 1), dtype=torch.complex128, device=dev)
        B[0::3] = 1.0
        X = torch.empty((3 * n, W), dtype=torch.complex128, device=dev)
        for w in range(W):
            A = (-T).to(torch.complex128)
            A.diagonal().add_(D[:, w].repeat_interleave(3))
            X[:, w] = torch.linalg.solve(A, B)[:, 0]
        cw = f8(4.0 * math.pi * args["wavenumber"] * EPS_M * unit ** 3)
        loss = torch.sum(torch.imag(torch.sum(X[0::3], dim=0)) * cw)
        lam = X * cw                                # A is symmetric and E0 real: the adjoint solution
    # dL = -Im(lambda^T dA p)
    L3, X3 = lam.reshape(n, 3, W), X.reshape(n, 3, W)
    (-torch.imag(torch.sum(torch.sum(L3 * X3, dim=1) * self_coef()))).backward()
    idx = torch.arange(n, device=dev)
    Wt = torch.imag(torch.einsum("iam,jbm->ijab", L3, X3))
    for c0 in range(0, n, 512):
        x = pos / unit
        Tc = ew.pair_tensor(x, x[c0:c0 + 512], idx[c0:c0 + 512, None] == idx[None, :])
        torch.sum(Wt[c0:c0 + 512] * Tc).backward()
    for k, g in ew.waves(max(1, int(2e7 / n))):
        ph = (pos / unit) @ k.T
        c, s = torch.cos(ph), torch.sin(ph)
        kc = k.to(torch.complex128)
        lk = torch.einsum("kc,icm->ikm", kc, L3)
        pk = torch.einsum("kc,icm->ikm", kc, X3)
        lc, ls = (torch.einsum("ik,ikm->km", t.to(lk.dtype), lk) for t in (c, s))
        pc, ps = (torch.einsum("ik,ikm->km", t.to(pk.dtype), pk) for t in (c, s))
        (-torch.imag(torch.sum(g[:, None] * (lc * pc + ls * ps)))).backward()
    return [loss.cpu(), pos.grad.cpu(), rad.grad.cpu(), wp.grad.cpu(), gm.grad.cpu()]
