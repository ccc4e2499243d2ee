"""
The work that a program has GFN-xTB on the GPU do, as measurable cases.

A case is a dict of plain values with a "kind":

- "batch": energies (and forces) of many molecules at once through a
  calculator with zero-padded input: screening, data generation, ensembles.
- "molecule": energy and forces of one molecule, positions that change from
  call to call: geometry optimisation, molecular dynamics.
- "hessian": the nuclear Hessian of one molecule (6 N displaced single
  points in one call): frequencies, thermochemistry.
- "integrals": overlap, dipole and quadrupole matrices of one molecule and
  their gradients through the integral wrappers: programs that build their
  own Hamiltonian on the basis.

Molecules come from the package's seeded generator, in the size ranges of its
benchmark sets: 3-9, 10-60 and 30-120 atoms, and single ones above that. The
seed of ``prepare`` displaces every atom by about 0.02 Bohr, as a step of an
optimisation or of dynamics does: the same molecules, other inputs. "mode" is
the SCF: "implicit", converged to 1e-10, or "full", the calculator's default
options (Anderson mixing to 1e-4).

GFN1 SCFs of some of the larger random molecules have several solutions, and
which one is reached hangs on the last bit: GFN1 cases keep to molecules up to
20 atoms, where none does, and to one fragment of 24 (GFN2 has none in its sets
when converged; the default options do not converge for all above 20 atoms).
"""

from __future__ import annotations

import functools
import json
import math
import warnings
from pathlib import Path

import numpy as np
import torch

import dxtb_gb300
from dxtb_gb300 import GFN1Calculator, GFN2Calculator
from dxtb_gb300.integrals import dipint, overlap, quadint
from dxtb_gb300.solvation import GeneralizedBorn
from dxtb_gb300.workloads import config_molecules, fixed_composition, random_molecule

WATER = (np.array([8, 1, 1], dtype=np.int64),
         np.array([[0.0, 0.0, 0.22], [0.0, 1.43, -0.89], [0.0, -1.43, -0.89]]))
#: seeds of the single larger molecules
LARGE_SEED = 9000


@functools.lru_cache(maxsize=None)
def _set(name: str) -> tuple:
    """The molecules of a size range: (numbers, positions in Bohr)."""
    if name == "3-9":
        return tuple(random_molecule(7000 + i, 3 + i % 7) for i in range(256))
    if name == "10-20":
        return tuple(m for m in _set("10-60") if len(m[0]) <= 20)
    return tuple(config_molecules({"10-60": 2, "30-120": 3}[name]))


@functools.lru_cache(maxsize=None)
def _one(source: str, index: int) -> tuple:
    if source == "water":
        return WATER
    if source == "C8N2O2H12":
        return fixed_composition(1000, {6: 8, 7: 2, 8: 2, 1: 12})
    if source == "large":  # index: its atoms
        return random_molecule(LARGE_SEED + index, index)
    mols = _set(source)
    return mols[index % len(mols)]


def _molecules(case: dict) -> list:
    if case["kind"] == "batch":
        mols = _set(case["set"])
        return [mols[(case["first"] + k) % len(mols)] for k in range(case["count"])]
    return [_one(case["set"], case["first"])]


def _displaced(pos: np.ndarray, rng) -> np.ndarray:
    return pos + 0.02 * rng.standard_normal(pos.shape)


# Shells (angular momenta) of the elements of the molecules, for work()
_AO = {"gfn1": {1: 2}, "gfn2": {1: 1}}
_AO_D = (16,)  # elements with a d shell here


def _nao(method: str, numbers) -> int:
    return sum(_AO[method].get(int(z), 9 if int(z) in _AO_D else 4) for z in numbers)


# --------------------------------------------------------------------------

def listed() -> list:
    return [
        # one water molecule in a dynamics loop, default options: the smallest call, latency alone
        {"name": "water_step", "kind": "molecule", "set": "water", "first": 0, "method": "gfn2",
         "mode": "full", "solvent": 0.0, "charge": 0},
        # one drug-like fragment of 24 atoms in an optimisation, tightly converged
        {"name": "fragment_step", "kind": "molecule", "set": "C8N2O2H12", "first": 0,
         "method": "gfn1", "mode": "implicit", "solvent": 0.0, "charge": 0},
        # one molecule of about 100 atoms, GFN2, one optimisation step
        {"name": "molecule_100_step", "kind": "molecule", "set": "30-120", "first": 0,
         "method": "gfn2", "mode": "implicit", "solvent": 0.0, "charge": 0},
        # the largest single molecule: 150 atoms
        {"name": "molecule_150_step", "kind": "molecule", "set": "large", "first": 150,
         "method": "gfn2", "mode": "implicit", "solvent": 0.0, "charge": 0},
        # a cation in a continuum solvent (ALPB water)
        {"name": "solvated_cation_step", "kind": "molecule", "set": "10-60", "first": 5,
         "method": "gfn2", "mode": "full", "solvent": 78.9, "charge": 1},
        # screening many tiny molecules
        {"name": "batch_tiny", "kind": "batch", "set": "3-9", "first": 0, "count": 256,
         "method": "gfn2", "mode": "full", "forces": True},
        # the package's headline batch: 256 molecules of 10-60 atoms, energy and forces
        {"name": "batch_256", "kind": "batch", "set": "10-60", "first": 0, "count": 256,
         "method": "gfn2", "mode": "implicit", "forces": True},
        # GFN1 energies of a small batch (a rerank), an odd count
        {"name": "batch_gfn1_energy", "kind": "batch", "set": "10-20", "first": 11, "count": 37,
         "method": "gfn1", "mode": "full", "forces": False},
        # a batch of larger molecules, energy and forces
        {"name": "batch_large", "kind": "batch", "set": "30-120", "first": 0, "count": 64,
         "method": "gfn2", "mode": "implicit", "forces": True},
        # frequencies of a small molecule
        {"name": "hessian_9", "kind": "hessian", "set": "3-9", "first": 6, "method": "gfn2"},
        # integrals and their gradients of one molecule of 22 atoms
        {"name": "integrals", "kind": "integrals", "set": "10-60", "first": 0, "method": "gfn2"},
    ]


def draw(rng) -> dict:
    kind = rng.choice(["batch", "batch", "molecule", "molecule", "hessian", "integrals"])
    method = rng.choice(["gfn1", "gfn2", "gfn2"])
    middle = "10-20" if method == "gfn1" else rng.choice(["10-20", "10-60"])
    if kind == "hessian":
        return {"kind": kind, "set": "3-9", "first": rng.randrange(256), "method": method}
    if kind == "integrals":
        return {"kind": kind, "set": "10-60", "first": rng.randrange(256), "method": method}
    name = rng.choice(["3-9", middle, middle, "30-120"])
    if name == "30-120":
        method = "gfn2"
    mode = "implicit" if name in ("10-60", "30-120") else rng.choice(["implicit", "full"])
    most = {"30-120": 64, "10-20": 53}.get(name, 256)
    first = rng.randrange(most)
    if kind == "batch":
        return {"kind": kind, "set": name, "first": first,
                "count": int(round(math.exp(rng.uniform(math.log(2), math.log(most))))),
                "method": method, "mode": mode, "forces": rng.random() < 0.7}
    solvent = 0.0 if name == "30-120" else rng.choice([0.0, 0.0, 78.9, 4.8])
    return {"kind": kind, "set": name, "first": first, "method": method, "mode": mode,
            "solvent": solvent, "charge": 0}


# --------------------------------------------------------------------------

def _options(mode: str) -> dict:
    opts = {"exclude": ["disp", "d4sc"], "guess": "sad"}
    if mode == "implicit":
        opts |= {"scf_mode": "implicit", "x_atol": 1e-10, "f_atol": 1e-10, "maxiter": 250}
    else:
        opts |= {"mixer": "anderson"}
    return opts


def prepare(case: dict, seed: int) -> dict:
    rng = np.random.default_rng(seed)
    mols = _molecules(case)
    nat = max(len(z) for z, _ in mols)
    num = torch.zeros(len(mols), nat, dtype=torch.int64)
    pos = torch.zeros(len(mols), nat, 3, dtype=torch.float64)
    for i, (z, p) in enumerate(mols):
        num[i, : len(z)] = torch.as_tensor(z)
        pos[i, : len(z)] = torch.as_tensor(_displaced(p, rng))
    if case["kind"] != "batch":
        num, pos = num[0], pos[0]
    pos = pos.cuda()
    state = {"kind": case["kind"], "numbers": num, "positions": pos}
    if case["kind"] == "integrals":
        n = _nao(case["method"], num)
        up = [torch.as_tensor(rng.standard_normal(s)).cuda() for s in ((n, n), (3, n, n), (9, n, n))]
        return state | {"method": case["method"], "upstream": up,
                        "positions": pos.requires_grad_(True)}
    cls = {"gfn1": GFN1Calculator, "gfn2": GFN2Calculator}[case["method"]]
    inter = None
    if case.get("solvent"):
        inter = [GeneralizedBorn(num, case["solvent"])]
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        calc = cls(num, opts=_options(case.get("mode", "implicit")), interaction=inter, device="cuda")
    return state | {"calc": calc, "charge": case.get("charge", 0), "forces": case.get("forces", True)}


def run(state: dict):
    pos = state["positions"]
    if state["kind"] == "integrals":
        num, method = state["numbers"], state["method"]
        out = {}
        for name, fn, up in zip("SDQ", (overlap, dipint, quadint), state["upstream"]):
            m = fn(num, pos, method)
            (g,) = torch.autograd.grad(m, pos, up)
            out[name], out["grad_" + name] = m.detach(), g
        return out
    calc = state["calc"]
    if state["kind"] == "hessian":
        return {"hessian": calc.hessian(pos)}
    calc.reset()  # new positions in a user's loop; the same ones here
    out = {}
    if state["forces"]:
        out["forces"] = calc.get_forces(pos, chrg=state["charge"])
    out["energy"] = calc.get_energy(pos, chrg=state["charge"])
    return out


def work(case: dict) -> dict:
    """
    What the path cannot do without: positions in, results out. An SCF needs
    at least one density from one Fock matrix per iteration; its operations are
    counted as 15 iterations of a symmetric eigenproblem and the density
    (11.3 n^3 each), whatever the solver.
    """
    mols = _molecules(case)
    nbytes = flops = 0.0
    for z, _ in mols:
        n, nat = _nao(case["method"], z), len(z)
        if case["kind"] == "integrals":
            nbytes += 8.0 * (2 * 13 * n * n + 4 * 3 * nat)
            flops += 13 * n * n * 16 * 20.0
            continue
        points = 6 * nat if case["kind"] == "hessian" else 1
        out = 9 * nat * nat if case["kind"] == "hessian" else 1 + 3 * nat
        nbytes += 8.0 * (4 * nat + out)
        flops += points * 15 * 11.3 * n**3
    return {"bytes": nbytes, "flops": flops}


# --------------------------------------------------------------------------
# integrals in 64 bits, from the definition: Gauss-Hermite quadrature of the
# products of primitives (exact for their polynomials), one axis at a time

_CART = {0: [(0, 0, 0)], 1: [(0, 1, 0), (0, 0, 1), (1, 0, 0)],
         2: [(2, 0, 0), (1, 1, 0), (1, 0, 1), (0, 2, 0), (0, 1, 1), (0, 0, 2)]}
_S3 = math.sqrt(3.0)
_SPH = {0: [[1.0]], 1: np.eye(3).tolist(),
        2: [[0, _S3, 0, 0, 0, 0], [0, 0, 0, 0, _S3, 0], [-0.5, 0, 0, -0.5, 0, 1],
            [0, 0, _S3, 0, 0, 0], [_S3 / 2, 0, 0, -_S3 / 2, 0, 0]]}


def _overlap_s(a, ca, b, cb, l):
    p = a[:, None] + b[None, :]
    odd = math.prod(range(1, 2 * l, 2))
    return float((ca[:, None] * cb[None, :] * (math.pi / p) ** 1.5 * odd / (2.0 * p) ** l).sum())


@functools.lru_cache(maxsize=None)
def _basis(method: str) -> dict:
    """Per element the shells (l, exponents, coefficients) of the published
    parametrisation: STO-nG expansions of unit norm, the second s shell of an
    element of GFN1 without valence orthogonal to the first."""
    data = Path(dxtb_gb300.__file__).parent / "data"
    sto = np.load(data / "stong.npz")
    out = {}
    for z, e in json.loads((data / f"{method}.json").read_text())["element"].items():
        out[int(z)] = shells = []
        for k, l in enumerate(e["angular"]):
            coeff, alpha = (v.astype(np.float64) for v in
                            sto[f"sto{e['ngauss'][k]}g"][:, e["pqn"][k] + (0, 4, 7)[l] - 1])
            alpha = alpha * e["slater"][k] ** 2
            coeff = coeff * alpha ** (0.75 + 0.5 * l)
            if method == "gfn1" and not e["valence"][k]:
                _, a1, c1 = shells[-1]
                coeff = coeff / math.sqrt(_overlap_s(alpha, coeff, alpha, coeff, l))
                s = _overlap_s(a1, c1, alpha, coeff, 0)
                alpha, coeff = np.concatenate([alpha, a1]), np.concatenate([coeff, -s * c1])
            coeff = coeff / math.sqrt(_overlap_s(alpha, coeff, alpha, coeff, l))
            shells.append((l, alpha, coeff))
    return out


def exact(case: dict, seed: int):
    """Integral matrices and their gradients; None where an SCF is part of the result."""
    if case["kind"] != "integrals":
        return None
    rng = np.random.default_rng(seed)
    ((z, p),) = _molecules(case)
    pos = torch.tensor(_displaced(p, rng), requires_grad=True)
    n = _nao(case["method"], z)
    up = [torch.as_tensor(rng.standard_normal(s)) for s in ((n, n), (3, n, n), (9, n, n))]
    atom, alpha, power, rows, cols, vals = [], [], [], [], [], []
    ao = 0
    for i, el in enumerate(z):
        for l, ex, co in _basis(case["method"])[int(el)]:
            for c, pw in enumerate(_CART[l]):
                for e, k in zip(ex, co):
                    for m in range(2 * l + 1):
                        if _SPH[l][m][c]:
                            rows.append(ao + m), cols.append(len(atom)), vals.append(k * _SPH[l][m][c])
                    atom.append(i), alpha.append(e), power.append(pw)
            ao += 2 * l + 1
    con = torch.zeros(ao, len(atom), dtype=torch.float64)
    con[rows, cols] = torch.tensor(vals, dtype=torch.float64)
    a = torch.tensor(alpha, dtype=torch.float64)
    r = pos[torch.tensor(atom)]
    tot = a[:, None] + a[None, :]
    root, weight = (torch.as_tensor(v) for v in np.polynomial.hermite.hermgauss(4))
    axes = []
    for x in range(3):
        u = r[:, x]
        ctr = (a[:, None] * u[:, None] + a[None, :] * u[None, :]) / tot
        pref = torch.exp(-a[:, None] * a[None, :] / tot * (u[:, None] - u[None, :]) ** 2) / tot.sqrt()
        pw = torch.tensor([q[x] for q in power])
        mom = [0.0, 0.0, 0.0]
        for t, w in zip(root, weight):
            at = ctr + t / tot.sqrt()
            di, dj = at - u[:, None], at - u[None, :]
            one = torch.ones_like(di)
            fi = torch.where(pw[:, None] == 0, one, torch.where(pw[:, None] == 1, di, di * di))
            fj = torch.where(pw[None, :] == 0, one, torch.where(pw[None, :] == 1, dj, dj * dj))
            f = w * pref * fi * fj
            mom = [mom[0] + f, mom[1] + f * at, mom[2] + f * at * at]
        axes.append(mom)

    def matrix(ex, ey, ez):
        return con @ (axes[0][ex] * axes[1][ey] * axes[2][ez]) @ con.T

    unit = [(1, 0, 0), (0, 1, 0), (0, 0, 1)]
    got = {"S": matrix(0, 0, 0), "D": torch.stack([matrix(*e) for e in unit]),
           "Q": torch.stack([matrix(*(np.array(e) + np.array(f))) for e in unit for f in unit])}
    out = {}
    for name, w in zip("SDQ", up):
        (g,) = torch.autograd.grad((got[name] * w).sum(), pos, retain_graph=True)
        out[name], out["grad_" + name] = got[name].detach(), g
    return out
