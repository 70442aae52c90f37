"""What a user has this library do, over the sizes it is used at.

Kinds of case
  reference   the reference's own driver and numerics on a small molecule (``scf_hf``: Harris guess,
              stored integrals): the smallest call, where launches and latency count
  molecule    one step of a geometry optimisation on a small molecule: set the basis, FP64 SCF, gradient
  scf         the energy of a water cluster: set the basis, mixed-precision SCF with incremental
              builds, every result matrix back
  batch       many conformers in one call, mixed SCF and gradients
  fock        one direct Fock build for a density in hand (what a caller with an SCF driver of its
              own runs once per iteration), FP64 or mixed
  gradient    the analytic gradient for a density and an energy-weighted density in hand
  diagonal    the Roothaan-Hall step F, X -> C, D, eps
  eigen       a symmetric eigenproblem

The systems are water clusters on a jittered 3 Angstrom grid with distorted monomers (snapshots of
a liquid), in the basis sets the library's tests and benchmark use.  Inputs are host arrays, because
the library's interface takes and returns host arrays.
"""
import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "haskell-abinitio_gb300"))

from gbhf import _lib, basis as B, hartree_fock, molecules  # noqa: E402
from gbhf.flops_model import F_ALG  # noqa: E402

# ---------------------------------------------------------------- the cases


def listed():
    return [
        # water/STO-3G through the reference's driver: 7 functions, the call the reference's own sample makes
        {"name": "reference-water", "kind": "reference", "waters": 1, "basis": "sto-3g"},
        # one optimisation step of a single water: 13 functions, all latency
        {"name": "molecule-water", "kind": "molecule", "waters": 1, "basis": "6-31g"},
        # the benchmark's molecule: 208 functions, mixed SCF end to end
        {"name": "scf-16", "kind": "scf", "waters": 16, "basis": "6-31g"},
        # 48 uneven conformers in one call (1 to 12 waters), energies and gradients
        {"name": "batch-48", "kind": "batch", "molecules": 48, "largest": 12},
        # a dimer's Fock matrix in FP64: 26 functions, an ordinary small build
        {"name": "fock-2-fp64", "kind": "fock", "waters": 2, "basis": "6-31g", "mixed": False},
        # 208 functions in FP64
        {"name": "fock-16-fp64", "kind": "fock", "waters": 16, "basis": "6-31g", "mixed": False},
        # 832 functions, the largest system of the benchmark, mixed
        {"name": "fock-64-mixed", "kind": "fock", "waters": 64, "basis": "6-31g", "mixed": True},
        # d functions, an odd number of molecules: 133 functions
        {"name": "fock-7-polar", "kind": "fock", "waters": 7, "basis": "6-31g*", "mixed": True},
        # the benchmark's gradient molecule: 104 functions, FP64
        {"name": "gradient-8-fp64", "kind": "gradient", "waters": 8, "basis": "6-31g", "mixed": False},
        # d functions in the gradient, mixed: 95 functions
        {"name": "gradient-5-polar", "kind": "gradient", "waters": 5, "basis": "6-31g*", "mixed": True},
        # the dense step of the benchmark's molecule
        {"name": "diagonal-208", "kind": "diagonal", "n": 208},
        # a larger, odd dense problem
        {"name": "eigen-333", "kind": "eigen", "n": 333},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo - 0.49), math.log(hi + 0.49)))))))


def draw(rng):
    kind = rng.choice(("molecule", "scf", "batch", "fock", "fock", "fock", "gradient", "gradient", "diagonal", "eigen"))
    if kind == "molecule":
        return {"kind": kind, "waters": _log_int(rng, 1, 4), "basis": rng.choice(("sto-3g", "6-31g", "6-31g*"))}
    if kind == "scf":
        return {"kind": kind, "waters": _log_int(rng, 2, 20), "basis": rng.choice(("sto-3g", "6-31g", "6-31g"))}
    if kind == "batch":
        return {"kind": kind, "molecules": _log_int(rng, 6, 48), "largest": rng.randint(3, 12)}
    if kind in ("diagonal", "eigen"):
        return {"kind": kind, "n": _log_int(rng, 7, 400)}
    basis = rng.choice(("sto-3g", "6-31g", "6-31g", "6-31g*"))
    mixed = rng.random() < 0.5
    if kind == "fock":
        top = {"sto-3g": 64, "6-31g": 48 if mixed else 28, "6-31g*": 10}[basis]
    else:
        top = {"sto-3g": 20, "6-31g": 12 if mixed else 8, "6-31g*": 5}[basis]
    return {"kind": kind, "waters": _log_int(rng, 1, top), "basis": basis, "mixed": mixed}


# ---------------------------------------------------------------- inputs


def _waters(n, rng):
    """Coordinates (3n, 3) in bohr: jittered grid sites, random orientations, monomers with bond
    lengths and angles spread as thermal motion spreads them, no contact below 1.5 Angstrom."""
    k = 1
    while k ** 3 < n:
        k += 1
    sites = np.array([(i, j, l) for i in range(k) for j in range(k) for l in range(k)][:n], float) * 3.0
    atoms = np.zeros((0, 3))
    for site in sites:
        while True:
            r1, r2 = 0.9572 + 0.02 * rng.standard_normal(2)
            half = math.radians(104.52 + 3.0 * rng.standard_normal()) / 2
            mono = np.array([[0, 0, 0], [r1 * math.sin(half), 0, r1 * math.cos(half)],
                             [-r2 * math.sin(half), 0, r2 * math.cos(half)]])
            q = rng.standard_normal(4)
            w, x, y, z = q / np.linalg.norm(q)
            rot = np.array([[1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w)],
                            [2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w)],
                            [2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)]])
            new = mono @ rot.T + site + rng.uniform(-0.3, 0.3, 3)
            if not len(atoms) or np.min(np.linalg.norm(atoms[:, None] - new[None], axis=2)) > 1.5:
                break
        atoms = np.concatenate([atoms, new])
    return atoms * B.ANGSTROM_TO_BOHR


def _cluster(waters, basis, rng):
    return B.make_atoms(molecules.water_labels(waters), _waters(waters, rng), basis)


def _density_like(fb, rng, core, valence, spread):
    """A flat symmetric matrix that falls off with the distance between its functions' atoms, as a
    density, an energy-weighted density or a core Hamiltonian of such a cluster does."""
    pos = fb.xyz[fb.cgf_atom]
    r = np.linalg.norm(pos[:, None] - pos[None], axis=2)
    m = rng.standard_normal((fb.n_cgf, fb.n_cgf))
    m = spread * (m + m.T) * np.exp(-r / 1.6)
    first = np.concatenate([[True], fb.cgf_atom[1:] != fb.cgf_atom[:-1]]) & (fb.charge[fb.cgf_atom] > 2)
    m[np.diag_indices(fb.n_cgf)] = np.where(first, core, valence * rng.uniform(0.5, 1.5, fb.n_cgf))
    return m[np.triu_indices(fb.n_cgf)].copy()


def _geometry(case, seed):
    """(atoms or list of atoms, generator) of a molecular case."""
    rng = np.random.default_rng([seed, 17])
    if case["kind"] == "batch":
        sizes = rng.permutation([1 + i % case["largest"] for i in range(case["molecules"])])
        return [_cluster(int(n), "sto-3g" if i % 2 == 0 else "6-31g", rng) for i, n in enumerate(sizes)], rng
    return _cluster(case["waters"], case["basis"], rng), rng


def _dense(case, seed):
    """Inputs of the dense cases: a matrix with the spectrum of a Fock matrix (core levels, occupied
    and virtual levels), for ``diagonal`` in a non-orthogonal basis with its orthogonaliser."""
    n = case["n"]
    rng = np.random.default_rng([seed, n, 23])
    core = max(1, n // 13)
    levels = np.concatenate([np.linspace(-20.7, -20.4, core), np.linspace(-1.4, 4.2, n - core)])
    gap = np.concatenate([np.full(core, 0.3 / core), np.full(n - core, 5.6 / max(1, n - core))])
    levels = levels + 0.3 * gap * rng.uniform(-1, 1, n)
    q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    a = (q * levels) @ q.T
    if case["kind"] == "eigen":
        return {"a": (a + a.T) / 2}
    u, _ = np.linalg.qr(rng.standard_normal((n, n)))
    s = np.exp(rng.uniform(-1.5, 1.0, n))          # eigenvalues of the overlap
    x, xi = (u * s ** -0.5) @ u.T, (u * s ** 0.5) @ u.T
    f = xi @ a @ xi
    return {"f": ((f + f.T) / 2)[np.triu_indices(n)].copy(), "x": (x + x.T) / 2, "occ": (5 * n) // 13}


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind}
    if kind in ("diagonal", "eigen"):
        return s | _dense(case, seed) | {"ctx": _lib.Context(0)}
    atoms, rng = _geometry(case, seed)
    if kind == "reference":
        return s | {"atoms": atoms}
    s["ctx"] = _lib.Context(0)
    if kind == "batch":
        s["flats"] = [B.flatten(a) for a in atoms]
        s["opts"] = _lib.baseline_opts(precision=_lib.PREC_MIXED, incremental=1, final_fp64=0, full_rebuild_every=0)
        return s
    s["fb"] = fb = B.flatten(atoms)
    if kind == "molecule":
        s["opts"] = _lib.baseline_opts()
    elif kind == "scf":
        s["opts"] = _lib.baseline_opts(precision=_lib.PREC_MIXED, incremental=1, final_fp64=0, full_rebuild_every=0)
    else:
        s["ctx"].set_basis(fb)
        s["precision"] = _lib.PREC_MIXED if case["mixed"] else _lib.PREC_FP64
        s["d"] = _density_like(fb, rng, 2.1, 0.6, 0.15)
        s["w"] = _density_like(fb, rng, -41.0, -0.7, 0.2)
        s["h"] = _density_like(fb, rng, -33.0, -8.0, 1.5)
    return s


def _phased(v):
    """Eigenvectors with the largest component of each column positive: their signs are free."""
    return v * np.where(v[np.abs(v).argmax(axis=0), np.arange(v.shape[1])] < 0, -1.0, 1.0)


def run(s):
    kind = s["kind"]
    if kind == "reference":
        r = hartree_fock.scf_hf(s["atoms"])
        return {"energy": r.energy, "fock": r.fock, "density": r.density, "orb_energies": r.orb_energies,
                "coeff": _phased(r.coeff), "iterations": r.iterations}
    ctx = s["ctx"]
    if kind == "eigen":
        w, v = ctx.eigen_solve(s["a"])
        return {"values": w, "vectors": _phased(v)}
    if kind == "diagonal":
        c, d, e = ctx.diagonal_hf(s["f"], s["x"], s["occ"])
        return {"coeff": _phased(c), "density": d, "orb_energies": e}
    if kind == "fock":
        return ctx.fock(s["h"], s["d"], _lib.MODE_EXACT, s["precision"])
    if kind == "gradient":
        return ctx.gradient(s["d"], s["w"], precision=s["precision"])
    if kind == "batch":
        energies, _, _, grads = ctx.scf_batch(s["flats"], s["opts"], gradients=True)
        return {"energies": energies, "gradients": np.concatenate(grads)}
    ctx.set_basis(s["fb"])
    r = ctx.scf(s["opts"])
    # the orbitals are part of the call; they are compared through the density and the Fock matrix
    # they diagonalise, because near-degenerate levels of a cluster leave them free to rotate
    out = {"energy": r["energy"], "fock": r["fock"], "density": r["density"], "orb_energies": r["orb_energies"]}
    if kind == "molecule":
        out["gradient"] = ctx.gradient()
    return out


# ---------------------------------------------------------------- the work of a pass


def _quartet_flops(fb, cutoff=1e-12):
    """Operations of one direct build: the unique primitive shell quartets whose overlap estimate
    passes the screening, each at its class's count."""
    start = np.flatnonzero(np.concatenate([[True], (fb.cgf_lxyz.sum(1)[1:] != fb.cgf_lxyz.sum(1)[:-1])
                                           | (fb.cgf_atom[1:] != fb.cgf_atom[:-1])
                                           | (fb.cgf_lxyz.sum(1)[1:] == 0)]))
    # first function of each shell: a run of components on one atom; equal-l shells of one atom are
    # split where the components start over
    shells = []
    for i, f in enumerate(start):
        end = start[i + 1] if i + 1 < len(start) else fb.n_cgf
        l = int(fb.cgf_lxyz[f].sum())
        step = (l + 1) * (l + 2) // 2
        shells += list(range(f, end, step))
    off = np.concatenate([[0], np.cumsum(fb.cgf_nprim)])
    site = [(int(fb.cgf_lxyz[f].sum()), fb.cgf_atom[f], fb.prim_coef[k], fb.prim_exp[k])
            for f in shells for k in range(off[f], off[f + 1])]
    l, at, c, e = (np.array(v) for v in zip(*site))
    i, j = np.triu_indices(len(site))
    hi, lo = np.maximum(l[i], l[j]), np.minimum(l[i], l[j])
    p = e[i] + e[j]
    r2 = ((fb.xyz[at[i]] - fb.xyz[at[j]]) ** 2).sum(1)
    k = np.abs(c[i] * c[j]) * np.exp(-e[i] * e[j] / p * r2) * 4.0 / p ** 1.25
    names = [a + b for n, a in enumerate("spd") for b in "spd"[:n + 1]]
    top, bins = {}, {}
    for h, name in enumerate(names):
        sel = (hi == "spd".index(name[0])) & (lo == "spd".index(name[1])) & (k > 1e-14)
        bins[name] = np.bincount(np.clip(((2 - np.log10(k[sel])) * 4).astype(int), 0, 64), minlength=65).astype(float)
    reach = int((4 - math.log10(cutoff)) * 4)
    total = 0.0
    for h, a in enumerate(names):
        for b in names[:h + 1]:
            cum = np.cumsum(bins[b])
            pairs = sum(bins[a][x] * cum[min(64, reach - x)] for x in range(65) if reach - x >= 0)
            total += pairs * (0.5 if a == b else 1.0) * F_ALG[a + b]
    return total


def work(case):
    kind = case["kind"]
    if kind == "eigen":
        n = case["n"]
        return {"bytes": 8.0 * (2 * n * n + n), "flops": (4 / 3 + 2) * n ** 3}
    if kind == "diagonal":
        n = case["n"]
        return {"bytes": 8.0 * (n * (n + 1) + 2 * n * n + n), "flops": (4 / 3 + 2 + 4 + 2 + 1) * n ** 3}
    geo, _ = _geometry(case, 0)
    flats = [B.flatten(a) for a in geo] if kind == "batch" else [B.flatten(geo)]
    nn = sum(f.n_cgf ** 2 for f in flats)
    n3 = sum(float(f.n_cgf) ** 3 for f in flats)
    quartets = sum(_quartet_flops(f) for f in flats)
    if kind == "fock":
        return {"bytes": 8.0 * 1.5 * nn, "flops": quartets}
    if kind == "gradient":
        return {"bytes": 8.0 * (nn + flats[0].xyz.size), "flops": 4 * quartets}
    # an SCF: at least one build of every quartet, ten iterations' dense algebra
    grad = 4 * quartets if kind in ("molecule", "batch") else 0.0
    return {"bytes": 8.0 * 4 * nn, "flops": quartets + grad + 10 * 12 * n3}


# ---------------------------------------------------------------- the same in 64 bits, plainly


class _Boys(torch.autograd.Function):
    """F_0 .. F_M of a tensor, stacked; dF_m/dT = -F_(m+1)."""

    @staticmethod
    def forward(ctx, t, m):
        top = m + 1
        small = t < 45.0
        ts = torch.where(small, t, torch.zeros_like(t))
        term = torch.full_like(t, 1.0 / (2 * top + 1))
        acc = term.clone()
        for i in range(1, 230):
            term = term * (2 * ts / (2 * top + 2 * i + 1))
            acc += term
        ex = torch.exp(-ts)
        f = [None] * (top + 1)
        f[top] = acc * ex
        for k in range(top - 1, -1, -1):
            f[k] = (2 * ts * f[k + 1] + ex) / (2 * k + 1)
        tl = torch.where(small, torch.full_like(t, 45.0), t)
        exl = torch.exp(-tl)
        g = 0.5 * torch.sqrt(math.pi / tl) * torch.erf(torch.sqrt(tl))
        out = []
        for k in range(top + 1):
            out.append(torch.where(small, f[k], g))
            g = ((2 * k + 1) * g - exl) / (2 * tl)
        f = torch.stack(out)
        ctx.save_for_backward(f)
        return f[:top]

    @staticmethod
    def backward(ctx, grad):
        f, = ctx.saved_tensors
        return -(grad * f[1:]).sum(0), None


def _hermite_r(top, alpha, v, scale):
    """{(t, u, v): R_tuv} for t + u + v <= top; v: the vector's three components."""
    f = _Boys.apply(alpha * (v[0] ** 2 + v[1] ** 2 + v[2] ** 2), top)
    level = {}
    for n in range(top, -1, -1):
        new = {(0, 0, 0): scale * (-2 * alpha) ** n * f[n]}
        for s in range(1, top - n + 1):
            for t in range(s + 1):
                for u in range(s - t + 1):
                    k = [t, u, s - t - u]
                    x = next(i for i in range(3) if k[i])
                    one = list(k)
                    one[x] -= 1
                    val = v[x] * level[tuple(one)]
                    if one[x]:
                        two = list(one)
                        two[x] -= 1
                        val = val + one[x] * level[tuple(two)]
                    new[tuple(k)] = val
        level = new
    return level


def _e_axis(i, j, p, pa, pb):
    """E^(ij)_t for t = 0 .. i + j on one axis, without the Gaussian factor."""
    tab = {(0, 0): [torch.ones_like(p)]}

    def get(a, b):
        if (a, b) not in tab:
            low, x = (get(a - 1, b), pa) if a else (get(a, b - 1), pb)
            out = []
            for t in range(a + b + 1):
                val = torch.zeros_like(p)
                if t < len(low):
                    val = val + x * low[t]
                if t >= 1:
                    val = val + low[t - 1] / (2 * p)
                if t + 1 < len(low):
                    val = val + (t + 1) * low[t + 1]
                out.append(val)
            tab[(a, b)] = out
        return tab[(a, b)]
    return get(i, j)


class _Plain:
    """One- and two-electron integrals of a small molecule; differentiable in the coordinates."""

    def __init__(self, fb, grad=False):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.fb, self.n = fb, fb.n_cgf
        self.xyz = torch.tensor(fb.xyz, dtype=torch.float64, device=dev, requires_grad=grad)
        self.z = torch.tensor(fb.charge, dtype=torch.float64, device=dev)
        off = np.concatenate([[0], np.cumsum(fb.cgf_nprim)])
        sites, of = {}, []
        for f in range(fb.n_cgf):
            of.append([(sites.setdefault((int(fb.cgf_atom[f]), float(fb.prim_exp[k])), len(sites)),
                        float(fb.prim_coef[k]), float(fb.prim_exp[k])) for k in range(off[f], off[f + 1])])
        ns = len(sites)
        s_at = torch.tensor([k[0] for k in sites], device=dev)
        s_ex = torch.tensor([k[1] for k in sites], dtype=torch.float64, device=dev)
        si, sj = torch.triu_indices(ns, ns, device=dev)
        number = torch.zeros((ns, ns), dtype=torch.long, device=dev)
        number[si, sj] = torch.arange(len(si), device=dev)
        self.p = s_ex[si] + s_ex[sj]
        self.P = (s_ex[si, None] * self.xyz[s_at[si]] + s_ex[sj, None] * self.xyz[s_at[sj]]) / self.p[:, None]
        lmax = int(fb.cgf_lxyz.sum(1).max())
        self.top = 2 * lmax
        self.herm = [(t, u, v) for t in range(self.top + 1) for u in range(self.top + 1 - t)
                     for v in range(self.top + 1 - t - u)]
        at_h = {h: i for i, h in enumerate(self.herm)}
        fi, fj = np.triu_indices(self.n)
        self.tri = (torch.tensor(fi, device=dev), torch.tensor(fj, device=dev))
        groups = {}
        for m, (f, g) in enumerate(zip(fi, fj)):
            rows = groups.setdefault((tuple(fb.cgf_lxyz[f]), tuple(fb.cgf_lxyz[g])), [])
            rows += [(m, int(fb.cgf_atom[f]), int(fb.cgf_atom[g]), x[0], y[0], x[1] * y[1], x[2], y[2])
                     for x in of[f] for y in of[g]]
        npair, nsite = len(fi), len(si)
        a = torch.zeros(len(self.herm) * npair * nsite, dtype=torch.float64, device=dev)
        s = torch.zeros(npair, dtype=torch.float64, device=dev)
        kin = torch.zeros(npair, dtype=torch.float64, device=dev)
        for (lf, lg), rows in groups.items():
            col = list(zip(*rows))
            m, af, ag, xs, ys = (torch.tensor(v, device=dev) for v in col[:5])
            c, ef, eg = (torch.tensor(v, dtype=torch.float64, device=dev) for v in col[5:])
            A, C = self.xyz[af], self.xyz[ag]
            p = ef + eg
            P = (ef[:, None] * A + eg[:, None] * C) / p[:, None]
            k = c * torch.exp(-ef * eg / p * ((A - C) ** 2).sum(1))
            e = [_e_axis(lf[x], lg[x], p, P[:, x] - A[:, x], P[:, x] - C[:, x]) for x in range(3)]
            where = number[torch.minimum(xs, ys), torch.maximum(xs, ys)]
            for t in range(len(e[0])):
                for u in range(len(e[1])):
                    for v in range(len(e[2])):
                        a = a.index_add(0, (at_h[(t, u, v)] * npair + m) * nsite + where,
                                        k * e[0][t] * e[1][u] * e[2][v])
            g3 = k * (math.pi / p) ** 1.5
            s = s.index_add(0, m, g3 * e[0][0] * e[1][0] * e[2][0])
            for x in range(3):
                other = e[(x + 1) % 3][0] * e[(x + 2) % 3][0]
                l = lg[x]
                up = _e_axis(lf[x], l + 2, p, P[:, x] - A[:, x], P[:, x] - C[:, x])[0]
                val = eg * (2 * l + 1) * e[x][0] - 2 * eg ** 2 * up
                if l >= 2:
                    val = val - 0.5 * l * (l - 1) * _e_axis(lf[x], l - 2, p, P[:, x] - A[:, x], P[:, x] - C[:, x])[0]
                kin = kin.index_add(0, m, g3 * other * val)
        self.A = a.view(len(self.herm), npair, nsite)
        self.s = s
        r = _hermite_r(self.top, self.p[:, None].expand(-1, len(self.z)),
                       [self.P[:, None, x] - self.xyz[None, :, x] for x in range(3)],
                       -(2 * math.pi / self.p)[:, None] * self.z[None])
        self.h = kin + sum(self.A[i] @ r[h].sum(1) for i, h in enumerate(self.herm))

    def square(self, flat):
        m = torch.zeros((self.n, self.n), dtype=torch.float64, device=flat.device)
        m[self.tri] = flat
        return m + m.T - torch.diag(torch.diagonal(m))

    def flat(self, m):
        return m[self.tri]

    def eri(self):
        """(pairs, pairs) of the unique function pairs."""
        out, sign = 0.0, [(-1.0) ** sum(h) for h in self.herm]
        step = max(1, int(6e6 // len(self.p)))
        for q0 in range(0, len(self.p), step):
            q = self.p[None, q0:q0 + step]
            p = self.p[:, None]
            r = _hermite_r(2 * self.top, p * q / (p + q),
                           [self.P[:, None, x] - self.P[None, q0:q0 + step, x] for x in range(3)],
                           2 * math.pi ** 2.5 / (p * q * torch.sqrt(p + q)))
            for j, hk in enumerate(self.herm):
                half = sum(self.A[i] @ r[tuple(a + b for a, b in zip(hb, hk))] for i, hb in enumerate(self.herm))
                out = out + half @ (sign[j] * self.A[j][:, q0:q0 + step]).T
        return out

    def full(self, eri):
        n = self.n
        number = torch.zeros((n, n), dtype=torch.long, device=eri.device)
        number[self.tri] = torch.arange(len(self.tri[0]), device=eri.device)
        number = torch.maximum(number, number.T).view(-1)
        return eri[number][:, number].view(n, n, n, n)

    def two_electron(self, full, d):
        return torch.einsum("ijkl,kl->ij", full, d) - 0.5 * torch.einsum("ikjl,kl->ij", full, d)

    def gradient(self, d, w):
        full = self.full(self.eri())
        r = self.xyz[:, None] - self.xyz[None]
        i, j = np.triu_indices(len(self.z), 1)
        rep = (self.z[i] * self.z[j] / torch.sqrt((r[i, j] ** 2).sum(1))).sum()
        e = (d * self.square(self.h)).sum() + 0.5 * (d * self.two_electron(full, d)).sum() - (w * self.square(self.s)).sum()
        return torch.autograd.grad(e + rep, self.xyz)[0], rep.detach()


def _plain_scf(pl, nocc):
    """Converged closed-shell SCF: (electronic energy, F, D, eps, C)."""
    s, h, full = pl.square(pl.s), pl.square(pl.h), pl.full(pl.eri())
    sv, su = torch.linalg.eigh(s)
    x = (su * sv ** -0.5) @ su.T
    f, errs, focks, last = h, [], [], 1e9
    for it in range(200):
        e, c = torch.linalg.eigh(x @ f @ x)
        c = x @ c
        d = 2 * c[:, :nocc] @ c[:, :nocc].T
        f = h + pl.two_electron(full, d)
        err = x @ (f @ d @ s - s @ d @ f) @ x
        size = float(err.abs().max())
        if size < 3e-11 or (it > 60 and size >= last):
            break
        last = size
        errs, focks = (errs + [err])[-8:], (focks + [f])[-8:]
        m = len(errs)
        b = torch.zeros((m + 1, m + 1), dtype=torch.float64, device=f.device)
        b[:m, :m] = torch.stack([torch.stack([(p * q).sum() for q in errs]) for p in errs])
        b[:m, :m] /= b[:m, :m].abs().max()
        b[m, :m] = b[:m, m] = -1
        rhs = torch.zeros(m + 1, dtype=torch.float64, device=f.device)
        rhs[m] = -1
        coef = torch.linalg.lstsq(b.cpu(), rhs[:, None].cpu(), driver="gelsd").solution.to(f.device)[:m, 0]
        f = sum(k * v for k, v in zip(coef, focks))
    e, c = torch.linalg.eigh(x @ f @ x)
    c = x @ c
    d = 2 * c[:, :nocc] @ c[:, :nocc].T
    return 0.5 * (d * (h + f)).sum(), f, d, e, c


def exact(case, seed):
    kind = case["kind"]
    if kind == "eigen":
        w, v = np.linalg.eigh(_dense(case, seed)["a"])
        return {"values": w, "vectors": _phased(v)}
    if kind == "diagonal":
        s = _dense(case, seed)
        n = case["n"]
        f = np.zeros((n, n))
        f[np.triu_indices(n)] = s["f"]
        f = f + f.T - np.diag(np.diag(f))
        e, v = np.linalg.eigh(s["x"].T @ f @ s["x"])
        c = s["x"] @ v
        d = 2 * c[:, :s["occ"]] @ c[:, :s["occ"]].T
        return {"coeff": _phased(c), "density": d[np.triu_indices(n)], "orb_energies": e}
    if kind in ("reference", "batch"):
        return None          # the reference's own numerics; many molecules
    small = {"sto-3g": 6, "6-31g": 4, "6-31g*": 2} if kind == "fock" else {"sto-3g": 3, "6-31g": 2, "6-31g*": 1}
    if case["waters"] > small[case["basis"]]:
        return None
    atoms, rng = _geometry(case, seed)
    fb = B.flatten(atoms)
    pl = _Plain(fb, grad=kind in ("gradient", "molecule"))
    if kind in ("fock", "gradient"):
        d, w, h = (torch.tensor(_density_like(fb, rng, *a), device=pl.p.device)
                   for a in ((2.1, 0.6, 0.15), (-41.0, -0.7, 0.2), (-33.0, -8.0, 1.5)))
        if kind == "gradient":
            return pl.gradient(pl.square(d), pl.square(w))[0].cpu().numpy()
        with torch.no_grad():
            return (h + pl.flat(pl.two_electron(pl.full(pl.eri()), pl.square(d)))).cpu().numpy()
    nocc = fb.n_occupied
    with torch.no_grad():
        energy, f, d, e, c = _plain_scf(pl, nocc)
        w = 2 * (c[:, :nocc] * e[:nocc]) @ c[:, :nocc].T
        r = pl.xyz[:, None] - pl.xyz[None]
        i, j = np.triu_indices(len(pl.z), 1)
        rep = (pl.z[i] * pl.z[j] / torch.sqrt((r[i, j] ** 2).sum(1))).sum()
        out = {"energy": float(energy + rep), "fock": pl.flat(f).cpu().numpy(), "density": pl.flat(d).cpu().numpy(),
               "orb_energies": e.cpu().numpy()}
    if kind == "molecule":
        out["gradient"] = pl.gradient(d, w)[0].cpu().numpy()
    return out
