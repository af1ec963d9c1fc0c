"""Cases for timing the framework's public entry points, with their plain 64-bit results.

A case is a dict of plain values; everything that decides its amount of work (atom counts, shells per
atom, k-meshes) follows from the case alone, and the seed draws the values: elements of the stated
shells, cells, positions, table amplitudes, targets.  Cells and tables come from the generators that the
rest of the repository uses (triclinic cells with a minimum distance, exponentially decaying integrals).

Kinds:
  properties  ``compute_multi_element_properties`` on one cell and an offset Monkhorst-Pack mesh
  bands       the same call on a path of k-points (a band structure)
  pdos        the same call with eigenvectors, then ``compute_atom_projected_dos``
  forces      ``finite_difference_forces`` of one cell
  batch       ``compute_properties_batch``: many cells in one call (screening, a served batch)
  fit         ``adjoint.differentiable_properties`` and ``backward`` of the fitting loss on a batch of cells: the
              forward and the adjoint of a fitting step, without the optimiser (a pass leaves the parameters alone)

Left out of the returned properties: the k-point indices of the band edges and ``is_direct_gap`` /
``is_direct_semiconductor`` (k and -k carry equal edges, so the last bit decides between them), and the
iteration count of the Fermi search.
"""
import math
import random

import numpy as np
import torch

from slakonet_gb300 import adjoint as A
from slakonet_gb300 import engine as E
from slakonet_gb300 import model as M
from slakonet_gb300 import pdos as P
from slakonet_gb300 import synthetic as syn
from slakonet_gb300 import training as T

DEVICE = "cuda"
H2E = 27.211
CUTOFF = 10.0
SHELLS = {"s": (1, 2), "sp": tuple(range(3, 21)) + tuple(range(31, 37)) + tuple(range(49, 55)),
          "spd": tuple(range(21, 31)) + tuple(range(37, 49)), "spdf": tuple(range(58, 66))}
NORB = {"s": 1, "sp": 4, "spd": 9, "spdf": 16}
MIXED = (("s", 0.05), ("sp", 0.45), ("spd", 0.37), ("spdf", 0.13))     # shares of Z = 1-65
STATS = ("fermi_ev", "gap_ev", "vbm_ev", "cbm_ev", "vwidth", "cwidth", "min_dgap", "efermi_ev", "bandgap_ev",
         "dos_fermi", "dos_gapc", "dos_total", "band_energy_ha")


def listed():
    return [
        # one k-point of a primitive cell: the smallest call, all latency
        {"name": "cell-1k", "kind": "properties", "layout": 1, "atoms": 2, "shells": "sp", "k1": 1, "k2": 1, "k3": 1},
        # 2-atom sp3d cell on 8x8x8 (512 k-points, n = 18): the plain method's headline configuration
        {"name": "cell-512k", "kind": "properties", "layout": 2, "atoms": 2, "shells": "spd", "k1": 8, "k2": 8, "k3": 8},
        # an ordinary unit cell: 23 atoms, 3x3x3, about 160 orbitals
        {"name": "cell-23", "kind": "properties", "layout": 3, "atoms": 23, "shells": "mixed", "k1": 3, "k2": 3, "k3": 3},
        # a large unit cell with few k-points (about 430 orbitals): one request of the serving stream
        {"name": "cell-61", "kind": "properties", "layout": 4, "atoms": 61, "shells": "mixed", "k1": 2, "k2": 2, "k3": 2},
        # a supercell whose matrices go to the device-wide eigensolver (n = 1152, 2 k-points)
        {"name": "supercell-128", "kind": "properties", "layout": 5, "atoms": 128, "shells": "spd", "k1": 2, "k2": 1, "k3": 1},
        # a band structure: 4 segments of 41 points, 7 atoms
        {"name": "bands-164", "kind": "bands", "layout": 6, "atoms": 7, "shells": "mixed", "segments": 4, "points": 41},
        # atom-projected DOS from eigenvectors: 6 atoms of nine orbitals each, 4x4x4
        {"name": "pdos-64k", "kind": "pdos", "layout": 7, "atoms": 6, "shells": "spd", "k1": 4, "k2": 4, "k3": 4},
        # finite-difference forces of a 3-atom cell: 18 displaced cells x 125 k-points in one call
        {"name": "forces-3", "kind": "forces", "layout": 8, "atoms": 3, "shells": "mixed"},
        # screening of primitive cells: many small problems
        {"name": "batch-primitive", "kind": "batch", "layout": 9, "cells": 48, "nmin": 1, "nmax": 6, "kdens": 1000.0},
        # a small uneven batch with coarse meshes
        {"name": "batch-11", "kind": "batch", "layout": 10, "cells": 11, "nmin": 2, "nmax": 32, "kdens": 150.0},
        # uneven batch of 2-64 atoms at ~1000 k*atoms per cell: the batched headline workload, at 96 of its 256 cells
        {"name": "batch-uneven", "kind": "batch", "layout": 11, "cells": 96, "nmin": 2, "nmax": 64, "kdens": 1000.0},
        # forward with eigenvectors and adjoint of one fitting step on 8 cells of 4-24 atoms
        {"name": "fit-8", "kind": "fit", "layout": 12, "cells": 8, "nmin": 4, "nmax": 24, "kdens": 500.0},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed ranges."""
    kind = rng.choice(("properties", "properties", "bands", "pdos", "forces", "batch", "batch", "fit"))
    layout = rng.randrange(1, 1 << 20)
    if kind == "properties":
        n = _log_int(rng, 1, 130)
        top = max(1, min(8, int((2000.0 / n ** 1.6) ** (1.0 / 3.0))))
        k = [rng.randint(1, top) for _ in range(3)]
        return {"kind": kind, "layout": layout, "atoms": n, "shells": "spd" if n > 64 else rng.choice(("sp", "spd", "mixed")),
                "k1": k[0], "k2": k[1] if n <= 64 else 1, "k3": k[2] if n <= 64 else 1}
    if kind == "bands":
        return {"kind": kind, "layout": layout, "atoms": _log_int(rng, 1, 16), "shells": rng.choice(("sp", "spd", "mixed")),
                "segments": rng.randint(1, 5), "points": rng.randint(5, 50)}
    if kind == "pdos":
        k = [rng.randint(1, 4) for _ in range(3)]
        return {"kind": kind, "layout": layout, "atoms": _log_int(rng, 1, 14), "shells": rng.choice(("sp", "spd")),
                "k1": k[0], "k2": k[1], "k3": k[2]}
    if kind == "forces":
        return {"kind": kind, "layout": layout, "atoms": rng.randint(1, 5), "shells": rng.choice(("sp", "spd", "mixed"))}
    if kind == "batch":
        cells = _log_int(rng, 2, 90)
        nmax = rng.choice((4, 9, 17, 33, 64))
        return {"kind": kind, "layout": layout, "cells": cells, "nmin": rng.randint(1, 3), "nmax": nmax,
                "kdens": float(_log_int(rng, 30, 900))}
    return {"kind": kind, "layout": layout, "cells": _log_int(rng, 1, 8), "nmin": 2, "nmax": rng.randint(4, 24),
            "kdens": float(_log_int(rng, 50, 500))}


# ------------------------------------------------------------------ what a case holds (from the case alone)

def _classes(rng, atoms, shells):
    if shells != "mixed":
        return [shells] * atoms
    return rng.choices([c for c, _ in MIXED], [w for _, w in MIXED], k=atoms)


def _cells(case):
    """[(shell class per atom, mesh or None)] of a case's cells."""
    rng = random.Random(case["layout"])
    if case["kind"] in ("batch", "fit"):
        out = []
        for _ in range(case["cells"]):
            n = _log_int(rng, case["nmin"], case["nmax"])
            f = [math.exp(rng.gauss(0.0, 0.25)) for _ in range(3)]
            scale = (max(1.0, case["kdens"] / n) / (f[0] * f[1] * f[2])) ** (1.0 / 3.0)
            out.append((_classes(rng, n, "mixed"), tuple(max(1, round(x * scale)) for x in f)))
        return out
    return [(_classes(rng, case["atoms"], case["shells"]), None)]


def _problems(case):
    """[(orbitals, complex k-points, real k-points, grids of the DOS)] of a case's cells."""
    out = []
    for classes, mesh in _cells(case):
        n = sum(NORB[c] for c in classes)
        if case["kind"] in ("batch", "fit"):
            nk, real = math.prod(mesh), math.prod(2 if m % 2 == 0 else 1 for m in mesh)
        elif case["kind"] == "bands":
            nk, real = case["segments"] * case["points"], 0
        elif case["kind"] == "forces":
            out += [(n, 124, 1)] * (6 * case["atoms"])
            continue
        else:
            m = (case["k1"], case["k2"], case["k3"])
            nk, real = math.prod(m), 1 if all(x % 2 for x in m) else 0
            real = nk if m == (1, 1, 1) else real
        out.append((n, nk - real, real))
    return out


def work(case):
    """Positions, tables and k-points read once and the spectrum and DOS written once; the flops of the dense
    generalised eigenproblem (Cholesky 4/3, reduction 4, tridiagonalisation 16/3 n^3 per complex k-point, a
    quarter of that per real one), with eigenvectors also 12 n^3, in a fitting step also 4 n^3 for the projectors."""
    vec = case["kind"] in ("pdos", "fit")
    flops = rows = 0.0
    for n, nc, nr in _problems(case):
        per = 32.0 / 3.0 + (12.0 if vec else 0.0) + (4.0 if case["kind"] == "fit" else 0.0)
        flops += per * float(n) ** 3 * (nc + nr / 4.0)
        rows += n * (nc + nr)
    points = 1000 if case["kind"] in ("batch", "fit", "pdos") else 1 if case["kind"] == "forces" else 5000
    return {"bytes": 8.0 * (rows + points * len(_cells(case)) + 661 * 2 * 40), "flops": flops}


# ------------------------------------------------------------------ inputs

def _grid_cell(rng, n, spacing=3.0, jitter=0.06):
    """A jittered, slightly sheared site grid: cells too large for placement by rejection."""
    g = [max(1, round(n ** (1.0 / 3.0)))] * 3
    while g[0] * g[1] * g[2] < n:
        g[int(np.argmin(g))] += 1
    edge = np.array(g) * spacing * syn.ANGSTROM_TO_BOHR
    cell = np.diag(edge) + rng.uniform(-0.04, 0.04, (3, 3)) * edge.min()
    sites = np.array([[i, j, k] for i in range(g[0]) for j in range(g[1]) for k in range(g[2])], dtype=float)
    sites = sites[np.sort(rng.permutation(len(sites))[:n])] / np.array(g)
    return sites @ cell + rng.normal(0.0, jitter * syn.ANGSTROM_TO_BOHR, (n, 3)), cell


def _inputs(case, seed):
    """(structures, element numbers, tables) in host memory, from the case and the seed alone."""
    rng = np.random.default_rng([int(seed), int(case["layout"])])
    cells = _cells(case)
    used = sorted({c for classes, _ in cells for c in classes})
    many = {"s": 1, "sp": 3, "spd": 3, "spdf": 1}
    palette = {c: [int(z) for z in rng.choice(SHELLS[c], many[c], replace=False)] for c in used}
    pick = random.Random(case["layout"] + 2)          # which of the palette's elements an atom has: the case's
    sts = []
    for classes, mesh in cells:
        n = len(classes)
        if n > 64 or case["kind"] == "forces":        # forces: bonded atoms, so that they stand clear of rounding
            pos, cell = _grid_cell(rng, n, 2.6, 0.25) if n <= 64 else _grid_cell(rng, n)
        else:
            st = syn.random_structure(rng, n, min_dist_angstrom=2.0)
            pos, cell = st["positions"], st["cell"]
        numbers = np.array([palette[c][pick.randrange(len(palette[c]))] for c in classes])
        st = {"numbers": numbers, "positions": pos, "cell": cell}
        if mesh is not None:
            st["kpoints"] = syn.gamma_centred_kpoints(mesh)
            st["weights"] = np.full(len(st["kpoints"]), 1.0 / len(st["kpoints"]))
        sts.append(st)
    zs = sorted({z for zz in palette.values() for z in zz})
    return sts, zs, syn.make_tables(zs, seed=int(rng.integers(1 << 31))), rng


def _klines(case):
    rng = random.Random(case["layout"] + 1)
    corners = [[0.0, 0.0, 0.0]] + [[rng.choice((0.0, 0.25, 0.375, 0.5, 0.625)) + 0.001 * i for _ in range(3)]
                                   for i in range(1, case["segments"] + 1)]
    return [corners[i] + corners[i + 1] + [float(case["points"])] for i in range(case["segments"])]


def _targets(rng, cells):
    """Smooth target DOS curves [cells, 1000] and gaps [cells], as a fit against external data has them."""
    e = np.linspace(T.DOS_RANGE[0], T.DOS_RANGE[1], T.DOS_POINTS)
    c, a = rng.uniform(-15.0, 8.0, (cells, 12, 1)), rng.uniform(0.5, 6.0, (cells, 12, 1))
    return (a * np.exp(-0.5 * ((e - c) / 0.8) ** 2)).sum(1), rng.uniform(0.0, 3.0, cells)


def prepare(case, seed):
    sts, zs, tables, rng = _inputs(case, seed)
    sd = syn.default_shell_dict()
    shell_dict = {z: list(sd[z]) for z in zs}
    state = {"case": dict(case), "shell_dict": shell_dict}
    state["model"] = M.MultiElementSkfParameterOptimizer.from_tables(tables).to(DEVICE)
    if case["kind"] in ("batch", "fit"):
        state["structures"] = sts
    else:
        state["structure"] = sts[0]
        state["geometry"] = M.Geometry(sts[0]["numbers"], sts[0]["positions"], sts[0]["cell"])
    if case["kind"] == "bands":
        state["klines"] = torch.tensor(_klines(case), dtype=torch.float64)
    elif case["kind"] in ("properties", "pdos"):
        state["mesh"] = torch.tensor([case["k1"], case["k2"], case["k3"]])
    elif case["kind"] == "fit":
        dos, gap = _targets(rng, len(sts))
        state["dos"] = torch.as_tensor(dos, device=DEVICE)
        state["gap"] = torch.as_tensor(gap, device=DEVICE)
        state["weights"] = torch.as_tensor([float(len(st["numbers"])) for st in sts], dtype=torch.float64, device=DEVICE)
    return state


# ------------------------------------------------------------------ one pass

KEPT = ("fermi_energy_eV", "fermi_energy_Ha", "band_gap_eV", "vbm_eV", "cbm_eV", "valence_band_width_eV",
        "conduction_band_width_eV", "minimum_direct_gap_eV", "nkpoints", "nbands", "nelectrons", "dos_at_fermi",
        "dos_gap_center_eV", "dos_total_states", "dos_energy_grid_tensor", "dos_values_tensor", "fermi_converged",
        "efermi", "bandgap", "eigenvalues")


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    model, sd = state["model"], state["shell_dict"]
    if kind == "batch":
        res = model.compute_properties_batch(state["structures"], sd, DEVICE, dos_range=(-20.0, 10.0), dos_points=1000,
                                             dos_window=9.0)
        return {"eig": res.eig, "mu": res.mu, "dos": res.dos, "grid": res.dos_grid,
                "stats": {k: res.stats[:, E.STAT[k]] for k in STATS}}
    if kind == "fit":
        for p in model.parameters():
            p.grad = None
        eig, dos, gap, _ = A.differentiable_properties(model, state["structures"], sd, DEVICE, dos_range=T.DOS_RANGE,
                                                       dos_points=T.DOS_POINTS, dos_window=9.0)
        per = ((dos - state["dos"]) ** 2).mean(1) + (gap - state["gap"]).abs()
        loss = (per * state["weights"]).sum() / state["weights"].sum()
        loss.backward()
        return {"loss": loss.detach(), "eig": eig.detach(),
                "grads": torch.cat([(torch.zeros_like(p) if p.grad is None else p.grad).reshape(-1)
                                    for p in model.parameters()])}
    if kind == "forces":
        return {"forces": model.finite_difference_forces(state["structure"], sd, DEVICE)}
    if kind == "bands":
        props, _ = model.compute_multi_element_properties(geometry=state["geometry"], shell_dict=sd,
                                                          klines=state["klines"], get_fermi=True, device=DEVICE)
    else:
        props, _ = model.compute_multi_element_properties(geometry=state["geometry"], shell_dict=sd,
                                                          kpoints=state["mesh"], get_fermi=True, device=DEVICE,
                                                          with_eigenvectors=kind == "pdos")
    out = {k: math.nan if props[k] is None else props[k] for k in KEPT}
    if kind == "pdos":
        grid, by_type, types = P.compute_atom_projected_dos(props, state["geometry"])
        out["pdos_grid"] = grid
        out["pdos"] = [by_type[t] for t in types]
    return out


# ------------------------------------------------------------------ the same results in plain 64-bit torch

def _harmonics(v, l):
    """Real harmonics, m = -l..l, of unit vectors ``v`` [..., 3]; any norm that is common to the set."""
    x, y, z = v[..., 0], v[..., 1], v[..., 2]
    if l == 0:
        return torch.ones_like(x)[..., None]
    if l == 1:
        return torch.stack([y, z, x], -1)
    if l == 2:
        r = math.sqrt(3.0)
        return torch.stack([r * x * y, r * y * z, 0.5 * (3 * z * z - 1), r * x * z, 0.5 * r * (x * x - y * y)], -1)
    a, b, c = math.sqrt(5.0 / 8.0), math.sqrt(15.0), math.sqrt(3.0 / 8.0)
    return torch.stack([a * y * (3 * x * x - y * y), b * x * y * z, c * y * (5 * z * z - 1), 0.5 * z * (5 * z * z - 3),
                        c * x * (5 * z * z - 1), 0.5 * b * z * (x * x - y * y), a * x * (x * x - 3 * y * y)], -1)


def _rotations(u, l):
    """D [bonds, 2l+1, 2l+1] that turns harmonics about z into harmonics about u, by a linear fit on fixed points."""
    other = torch.where((u[:, :1].abs() < 0.6), torch.tensor([1.0, 0.0, 0.0], dtype=torch.float64), torch.tensor([0.0, 1.0, 0.0], dtype=torch.float64))
    e1 = torch.linalg.cross(other, u)
    e1 = e1 / e1.norm(dim=1, keepdim=True)
    R = torch.stack([e1, torch.linalg.cross(u, e1), u], -1)
    g = torch.Generator().manual_seed(7)
    pts = torch.randn(64, 3, generator=g, dtype=torch.float64)
    pts = pts / pts.norm(dim=1, keepdim=True)
    fit = torch.linalg.pinv(_harmonics(pts, l))                       # [2l+1, 64]
    return torch.einsum("ap,bpm->bam", fit, _harmonics(torch.einsum("bca,pc->bpa", R, pts), l))


def _bonds(st):
    """i, j, T, distance and direction of every directed bond 0 < d < CUTOFF."""
    pos, cell = torch.as_tensor(st["positions"]), torch.as_tensor(st["cell"])
    inv = torch.linalg.inv(cell)
    frac = pos @ inv
    r = (CUTOFF * inv.norm(dim=0) + (frac.max(0)[0] - frac.min(0)[0])).floor().int() + 1
    T_ = torch.cartesian_prod(*[torch.arange(-int(x), int(x) + 1).double() for x in r]).reshape(-1, 3)
    got = []
    for lo in range(0, len(T_), 64):
        t = T_[lo:lo + 64]
        vec = pos[None, None] + (t @ cell)[:, None, None] - pos[None, :, None]        # [T, i, j, 3]
        d = vec.norm(dim=-1)
        c, i, j = torch.nonzero((d < CUTOFF) & (d > 0.0), as_tuple=True)
        got.append((i, j, t[c], d[c, i, j], vec[c, i, j]))
    i, j, t, d, vec = (torch.cat(x) for x in zip(*got))
    return i, j, t, d, vec / d[:, None]


def _matrices(st, sd, pairs, onsite, step):
    """H(R) and S(R) entries of a cell as (T, row, column, value of H, value of S), differentiable in the tables."""
    z = [int(v) for v in st["numbers"]]
    norb = torch.tensor([sum(2 * l + 1 for l in sd[v]) for v in z])
    off = torch.cumsum(norb, 0) - norb
    i, j, t, d, u = _bonds(st)
    zi, zj = torch.tensor(z)[i], torch.tensor(z)[j]
    D = {l: _rotations(u, l) for l in range(4)}
    parts = []
    for a, b in sorted(set(zip(zi.tolist(), zj.tolist()))):
        here = torch.nonzero((zi == a) & (zj == b))[:, 0]
        oa = 0
        for la in sd[a]:
            ob = 0
            for lb in sd[b]:
                lo = min(la, lb)
                straight = torch.full((len(here),), la < lb) if la != lb else i[here] <= j[here]
                for way in (True, False):
                    q = here[straight if way else ~straight]
                    if not len(q):
                        continue
                    tabs = pairs[(a, b)] if way else pairs[(b, a)]
                    key = (la, lb) if way else (lb, la)
                    ng = tabs["H"][key].shape[-1]
                    last = ((d[q] / step).floor().long() + 5).clamp(9, ng)
                    nodes = (last[:, None] - 8 + torch.arange(8)).double() * step
                    w = torch.ones(len(q), 8, dtype=torch.float64)
                    for m in range(8):
                        for o in range(8):
                            if o != m:
                                w[:, m] *= (d[q] - nodes[:, o]) / (nodes[:, m] - nodes[:, o])
                    rows = last[:, None] - 9 + torch.arange(8)
                    shape = torch.einsum("bxm,bym->bmxy", D[la][q][:, :, la - lo:la + lo + 1],
                                         D[lb][q][:, :, lb - lo:lb + lo + 1])
                    if not way and (la + lb) % 2:
                        shape = -shape
                    v = [torch.einsum("bmxy,bm->bxy", shape,
                                      torch.stack([(tabs[x][key][abs(m)][rows] * w).sum(1) for m in range(-lo, lo + 1)], 1))
                         for x in ("H", "S")]
                    row = (off[i[q]] + oa)[:, None, None] + torch.arange(2 * la + 1)[:, None]
                    col = (off[j[q]] + ob)[:, None, None] + torch.arange(2 * lb + 1)
                    one = torch.zeros(len(q), 2 * la + 1, 2 * lb + 1, dtype=torch.long)
                    parts.append((q[:, None, None] + one, row + one, col + one, v[0], v[1]))
                ob += 2 * lb + 1
            oa += 2 * la + 1
    n = int(norb.sum())
    flat = [torch.cat([p[m].reshape(-1) for p in parts]) if parts else torch.zeros(0) for m in range(5)]
    diag = torch.cat([torch.tensor(np.concatenate([[onsite[v][l]] * (2 * l + 1) for l in sd[v]])) for v in z])
    return n, t, flat, diag


def _at_k(real_space, k):
    n, t, (bond, row, col, h, s), diag = real_space
    H = torch.zeros(n * n, dtype=torch.complex128)
    S = torch.zeros(n * n, dtype=torch.complex128)
    if len(bond):
        ph = torch.exp(2j * math.pi * (t @ torch.as_tensor(k)))[bond.long()]
        at = (row * n + col).long()
        H = H.index_add(0, at, h * ph)
        S = S.index_add(0, at, s * ph)
    H, S = H.reshape(n, n), S.reshape(n, n)
    return H + torch.diag(diag).to(H.dtype), S + torch.eye(n, dtype=S.dtype)


def _solve(H, S, vectors=False):
    L = torch.linalg.cholesky(S)
    A = torch.linalg.solve_triangular(L, H, upper=False)
    A = torch.linalg.solve_triangular(L, A.mH, upper=False)
    A = 0.5 * (A + A.mH)
    if not vectors:
        return torch.linalg.eigvalsh(A), None
    e, y = torch.linalg.eigh(A)
    return e, torch.linalg.solve_triangular(L.mH, y, upper=True)


def _fermi(e, w, nelec, kT=0.01):
    """The half-step Newton search on (N(mu) - Ne)^2; returns mu and whether it stopped by itself."""
    mu = float(e.mean())
    for _ in range(100):
        x = torch.exp((e - mu) / kT)
        f = 1.0 / (x + 1.0)
        diff = 2.0 * float((w[:, None] * f).sum()) - nelec
        grad = 4.0 * diff * float((w[:, None] * f * f * x).sum()) / kT
        if abs(grad) < 1e-6:
            return mu, True
        mu = mu - diff * diff / (grad + 1e-12)
    return mu, False


def _dos(e, w, mu, lo, hi, points, sigma=0.1, window=None):
    grid = torch.linspace(lo, hi, points, dtype=torch.float64)
    out = torch.zeros(points, dtype=torch.float64)
    ev, ww = ((e - mu) * H2E).reshape(-1), w[:, None].expand_as(e).reshape(-1)
    for a in range(0, points, 250):
        t = (grid[a:a + 250, None] - ev[None]) / sigma
        g = torch.exp(-0.5 * t * t)
        if window is not None:
            g = torch.where((ev[None] >= grid[a:a + 250, None] - window * sigma) &
                            (ev[None] <= grid[a:a + 250, None] + window * sigma), g, torch.zeros_like(g))
        out[a:a + 250] = (g * ww[None]).sum(1) / (sigma * math.sqrt(2.0 * math.pi))
    return grid, out


def _stats(e, w, mu, grid, dos):
    """Band edges, gaps and DOS figures (eV) of one cell, by name."""
    ev, fe, x = e * H2E, mu * H2E, (e - mu) * H2E
    occ, un = ev < fe, ev >= fe
    metal = bool(((ev - fe).abs() < 1e-3).any())
    found = bool(occ.any()) and bool(un.any())
    v, c = (fe, fe) if metal else (float(ev[occ].max()), float(ev[un].min())) if found else (0.0, 0.0)
    kv = torch.where(x < 0, x, torch.full_like(x, -math.inf)).max(1)[0]
    kc = torch.where(x > 0, x, torch.full_like(x, math.inf)).min(1)[0]
    dg = kc - kv
    dg = float(dg[torch.isfinite(dg)].min()) if torch.isfinite(dg).any() else math.nan
    lo, hi = e[e <= mu], e[e > mu]
    width = lambda y: float(y.max() - y.min()) if len(y) else 0.0   # noqa: E731
    near = torch.where(grid.abs() < 2.0, dos, torch.full_like(dos, math.inf))
    be = torch.where(e == 0, torch.zeros_like(e), 1.0 / (1.0 + torch.exp((e - mu) / (0.025 / H2E))))
    shown = fe if (metal or found) else 0.0
    return {"fermi_ev": shown, "gap_ev": c - v, "vbm_ev": v, "cbm_ev": c, "vwidth": width(x[x < 0]),
            "cwidth": width(x[x >= 0]), "min_dgap": dg, "efermi_ev": fe,
            "bandgap_ev": max(0.0, float(hi.min() - lo.max())) * H2E if len(lo) and len(hi) else math.inf,
            "dos_fermi": float(dos[grid.abs().argmin()]), "dos_gapc": float(grid[near.argmin()]),
            "dos_total": float(torch.trapezoid(dos, grid)), "band_energy_ha": float((w[:, None] * be * e).sum())}


def _offset_mesh(m):
    return torch.cartesian_prod(*[(torch.arange(x).double() + 0.5) / x for x in m]).reshape(-1, 3)


def exact(case, seed):
    cost = sum(n ** 3 * (nc + nr) * 2.5e-9 + (nc + nr) * 4e-3 for n, nc, nr in _problems(case))
    if cost * (3.0 if case["kind"] in ("pdos", "fit") else 1.0) > 14.0:
        return None
    sts, zs, tables, rng = _inputs(case, seed)
    sd = syn.default_shell_dict()
    pairs = {k: {x: {kk: torch.tensor(vv) for kk, vv in v[x].items()} for x in ("H", "S")} for k, v in tables["pairs"].items()}
    onsite = {z: tables["elements"][z]["on_sites"] for z in zs}
    electrons = lambda st: float(sum(tables["elements"][int(z)]["occupations"].sum() for z in st["numbers"]))  # noqa: E731
    step = tables["step"]
    if case["kind"] == "fit":
        return _exact_fit(case, sts, sd, pairs, onsite, electrons, step, rng)
    if case["kind"] == "forces":
        st, mesh = sts[0], _offset_mesh((5, 5, 5))
        F = torch.zeros(1, len(st["numbers"]), 3, dtype=torch.float64)
        for a in range(F.shape[1]):
            for x in range(3):
                for sign in (1.0, -1.0):
                    p = np.array(st["positions"])
                    p[a, x] += sign * 1e-2
                    rs = _matrices(dict(st, positions=p), sd, pairs, onsite, step)
                    total = sum(float(_solve(*_at_k(rs, k))[0].sum()) for k in mesh)
                    F[0, a, x] -= sign * total / 2e-2
        return {"forces": F}
    out = []
    for st in sts:
        if case["kind"] == "batch":
            ks = torch.as_tensor(st["kpoints"])
        elif case["kind"] == "bands":
            rows = torch.tensor(_klines(case), dtype=torch.float64)
            ks = torch.stack([r[:3] + (r[3:6] - r[:3]) / (r[6] - 1.0) * i for r in rows for i in range(int(r[6]))])
        else:
            ks = _offset_mesh((case["k1"], case["k2"], case["k3"]))
        w = torch.full((len(ks),), 1.0 / len(ks), dtype=torch.float64)
        rs = _matrices(st, sd, pairs, onsite, step)
        sol = [_solve(*_at_k(rs, k), vectors=case["kind"] == "pdos") for k in ks]
        e = torch.stack([s[0] for s in sol])
        mu, stopped = _fermi(e, w, electrons(st))
        if case["kind"] == "batch":
            grid, dos = _dos(e, w, mu, -20.0, 10.0, 1000, window=9.0)
        else:
            grid, dos = _dos(e, w, mu, -10.0, 10.0, 5000)
        out.append((e, mu, dos, grid, _stats(e, w, mu, grid, dos), stopped, sol))
    if case["kind"] == "batch":
        return {"eig": torch.cat([o[0].reshape(-1) for o in out]), "mu": torch.tensor([o[1] for o in out], dtype=torch.float64),
                "dos": torch.stack([o[2] for o in out]), "grid": out[0][3],
                "stats": {k: torch.tensor([o[4][k] for o in out], dtype=torch.float64) for k in STATS}}
    e, mu, dos, grid, s, stopped, sol = out[0]
    got = {"fermi_energy_eV": s["fermi_ev"], "fermi_energy_Ha": s["fermi_ev"] / H2E, "band_gap_eV": s["gap_ev"],
           "vbm_eV": s["vbm_ev"], "cbm_eV": s["cbm_ev"], "valence_band_width_eV": s["vwidth"],
           "conduction_band_width_eV": s["cwidth"], "minimum_direct_gap_eV": s["min_dgap"],
           "nkpoints": e.shape[0], "nbands": e.shape[1], "nelectrons": int(electrons(sts[0])), "dos_at_fermi": s["dos_fermi"],
           "dos_gap_center_eV": s["dos_gapc"], "dos_total_states": s["dos_total"], "dos_energy_grid_tensor": grid,
           "dos_values_tensor": dos, "fermi_converged": stopped, "efermi": torch.tensor([[[s["efermi_ev"]]]], dtype=torch.float64),
           "bandgap": torch.tensor([s["bandgap_ev"]], dtype=torch.float64), "eigenvalues": e[None]}
    if case["kind"] == "pdos":
        z = [int(v) for v in sts[0]["numbers"]]
        per = e.shape[1] // len(z)
        pg = torch.linspace(-8.0, 6.0, 1000, dtype=torch.float64)
        x = (e * H2E - s["fermi_ev"]).reshape(-1)
        g = torch.exp(-0.5 * ((pg[:, None] - x[None]) / 0.1) ** 2) / (0.1 * math.sqrt(2.0 * math.pi))
        c2 = torch.stack([q[1].abs() ** 2 for q in sol])                       # [k, orbital, band]
        got["pdos_grid"] = pg
        got["pdos"] = []
        for t in dict.fromkeys(z):
            rows = torch.tensor([a * per + o for a in range(len(z)) if z[a] == t for o in range(per)])
            got["pdos"].append((g * c2[:, rows].sum(1).reshape(-1)[None]).sum(1) / e.shape[0])
    return got


def _exact_fit(case, sts, sd, pairs, onsite, electrons, step, rng):
    dos_t, gap_t = (torch.as_tensor(x) for x in _targets(rng, len(sts)))
    params = [pairs[k][x][key].requires_grad_() for k in sorted(pairs) for x in ("H", "S") for key in pairs[k][x]]
    loss, eig = 0.0, []
    for s, st in enumerate(sts):
        ks = torch.as_tensor(st["kpoints"])
        w = torch.full((len(ks),), 1.0 / len(ks), dtype=torch.float64)
        rs = _matrices(st, sd, pairs, onsite, step)
        e = []
        for k in ks:
            H, S = _at_k(rs, k)
            with torch.no_grad():
                e0, c = _solve(H, S, vectors=True)
            # first order about the solution: e_n + Re c_n^H (H - e_n S) c_n, whose value is e_n
            lin = ((c.conj() * (H @ c)).sum(0) - e0 * (c.conj() * (S @ c)).sum(0)).real
            e.append(e0 + lin - lin.detach())
        e = torch.stack(e)
        eig.append(e.detach().reshape(-1))
        mu, _ = _fermi(e.detach(), w, electrons(st))
        _, d = _dos(e, w, mu, T.DOS_RANGE[0], T.DOS_RANGE[1], T.DOS_POINTS, window=9.0)
        ev, fe = e * H2E, mu * H2E
        gap = torch.zeros((), dtype=torch.float64)
        if not bool(((ev - fe).abs() < 1e-3).any()) and bool((ev < fe).any()) and bool((ev >= fe).any()):
            gap = ev[ev >= fe].min() - ev[ev < fe].max()
        loss = loss + (((d - dos_t[s]) ** 2).mean() + (gap - gap_t[s]).abs()) * len(st["numbers"])
    loss = loss / sum(len(st["numbers"]) for st in sts)
    loss.backward()
    return {"loss": loss.detach(), "eig": torch.cat(eig),
            "grads": torch.cat([(torch.zeros_like(p) if p.grad is None else p.grad).reshape(-1) for p in params])}
