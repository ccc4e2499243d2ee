"""
The digit-plane products and the iterated eigenvectors (csrc/eigemm.cuh)
against the oracle, at the sizes where they can go wrong: one block of 16
orbitals and its edges, the 128 terms of one float32 accumulation, the edges
of the size classes; symmetric molecules and free atoms, whose eigenvalues are
exactly degenerate; and the float64 path that stands in where the workspace
has no room for the planes.

Tolerances are those of the other parity tests (energies 1e-8 Eh, forces
1e-6 Eh/Bohr), which the float64 path is held to. C and its orbital energies
are checked by what they must fulfil at the final potential: C S C^T = 1 and
P = C^T occ C to 1e-11 (a 54-bit operand and n <= 140 terms: about 140 x 2^-53
x |C|^2 / 1e2), eigenvalues ascending.
"""

import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

E_TOL, F_TOL, ORTHO = 1e-8, 1e-6, 1e-11


def _molecule(n: int, seed: int = 11):
    """A random molecule of exactly n GFN2 orbitals and an even electron count."""
    from dxtb_gb300.workloads import build_geometry

    rng = np.random.default_rng(seed + n)
    heavy = max(0, (n - 2) // 6) if n > 4 else 0
    nh = n - 4 * heavy
    z = [6] * heavy
    if nh % 2 and heavy:
        z[0] = 7
    if not heavy:
        return np.ones(n, dtype=np.int64), np.array([[0.0, 0.0, 1.6 * k] for k in range(n)])
    return build_geometry(rng, z, nh)


@pytest.mark.parametrize("n", [2, 15, 16, 17, 32, 33, 48, 111, 112, 127, 128, 129, 136, 137])
def test_block_edges_match_oracle(n):
    from dxtb_gb300.calculators import tables
    from dxtb_gb300.engine import PackedBatch, run
    from oracle import xtb_oracle as X

    num, pos = _molecule(n)
    pb = PackedBatch(tables("gfn2"), [num], [torch.tensor(pos)])
    assert int(pb.nao[0]) == n
    r = run(pb, forces=True, tol=1e-10)
    assert int(r.status[0]) == 0
    ref = X.singlepoint("gfn2", num, pos, grad=n <= 48, tol=1e-10)
    assert abs(float(r.energy[0]) - ref.energy) <= E_TOL
    if n <= 48:
        assert np.abs(r.gradient.cpu().numpy() - ref.extra["gradient"].numpy()).max() <= F_TOL
    s = {k: r.state[k][: n * n].view(n, n).cpu() for k in ("S", "P", "C")}
    ev, occ = r.state["evals"][:n].cpu(), r.state["occ"][:n].cpu()
    assert (ev[1:] >= ev[:-1]).all()
    assert (ev - ref.eps).abs().max() <= 1e-8
    m = int((s["C"].abs().sum(1) > 0).sum())
    c = s["C"][:m]
    assert (c @ s["S"] @ c.T - torch.eye(m)).abs().max() <= ORTHO
    assert (c.T @ (occ[:m, None] * c) - s["P"]).abs().max() <= ORTHO
    assert torch.equal(s["P"], s["P"].T)


@pytest.mark.parametrize("heavy,nh,n", [([6, 6], 4, 12), ([7, 6], 5, 13)])
def test_both_sides_of_the_float64_order(heavy, nh, n):
    """The largest molecule of the float64 path and the smallest on the planes."""
    from dxtb_gb300.calculators import tables
    from dxtb_gb300.engine import PackedBatch, run
    from dxtb_gb300.workloads import build_geometry
    from oracle import xtb_oracle as X

    num, pos = build_geometry(np.random.default_rng(n), heavy, nh)
    pb = PackedBatch(tables("gfn2"), [num], [torch.tensor(pos)])
    assert int(pb.nao[0]) == n
    r = run(pb, forces=True, tol=1e-10)
    assert int(r.status[0]) == 0
    ref = X.singlepoint("gfn2", num, pos, grad=True, tol=1e-10)
    assert abs(float(r.energy[0]) - ref.energy) <= E_TOL
    assert np.abs(r.gradient.cpu().numpy() - ref.extra["gradient"].numpy()).max() <= F_TOL


@pytest.mark.parametrize("method", ["gfn1", "gfn2"])
@pytest.mark.parametrize("case", ["atoms", "methane", "waters"])
def test_degenerate_levels_match_oracle(method, case):
    """Exactly degenerate eigenvalues: free atoms, T_d symmetry, identical far copies."""
    from dxtb_gb300.calculators import tables
    from dxtb_gb300.engine import PackedBatch, run
    from oracle import xtb_oracle as X

    w = np.array([[0, 0, 0.22], [0, 1.43, -0.89], [0, -1.43, -0.89]])
    d = 1.19
    mols = {
        "atoms": [(np.array([z]), np.zeros((1, 3))) for z in (2, 10, 18)],
        "methane": [(np.array([6, 1, 1, 1, 1]),
                     d * np.array([[0, 0, 0], [1, 1, 1], [-1, -1, 1], [-1, 1, -1], [1, -1, -1]]))],
        "waters": [(np.array([8, 1, 1] * 8), np.concatenate(
            [w + sp * np.array([i, j, k]) for i in range(2) for j in range(2) for k in range(2)]))
            for sp in (5.5, 40.0)],
    }[case]
    pb = PackedBatch(tables(method), [m[0] for m in mols], [torch.tensor(m[1]) for m in mols])
    r = run(pb, forces=True, tol=1e-10)
    assert (r.status.cpu() == 0).all()
    for i, (num, pos) in enumerate(mols):
        ref = X.singlepoint(method, num, pos, tol=1e-10)
        assert abs(float(r.energy[i]) - ref.energy) <= E_TOL


def test_without_room_for_the_planes():
    """dxtb_scf_noalloc takes the float64 path for a molecule whose workspace
    fits its array only without the planes; both paths give one answer."""
    from dxtb_gb300 import _lib
    from dxtb_gb300.calculators import tables
    from dxtb_gb300.data import radii
    from dxtb_gb300.engine import PackedBatch, run
    from dxtb_gb300.workloads import random_molecule

    num, pos = random_molecule(8800, 130)
    pb = PackedBatch(tables("gfn2"), [num], [torch.tensor(pos)])
    n, nat = int(pb.nao[0]), int(pb.nat[0])
    L = _lib.lib()
    room = 1 << 21
    base = 8 * n * n + 519 * (n + 9 * nat)  # the leading terms without the planes
    assert base < 0.97 * room < room < L.dxtb_scf_workspace_mol(n, nat)
    ref = run(pb, forces=True)
    assert int(ref.status[0]) == 0
    s, dev = ref.state, pb.device
    nm, na = n * n, nat
    out = {k: torch.full((c,), float("nan"), dtype=torch.float64, device=dev) for k, c in
           [("P", nm), ("W", nm), ("C", nm), ("ev", n), ("occ", n), ("q", n), ("dp", 3 * na),
            ("qp", 6 * na), ("vorb", n), ("vdp", 3 * na), ("vqp", 6 * na), ("en", 4)]}
    status = torch.full((1,), -1, dtype=torch.int32, device=dev)
    rc = L.dxtb_scf_noalloc(
        C.byref(pb.struct), pb.t["par_f"].data_ptr(), pb.t["par_i"].data_ptr(), s["S"].data_ptr(),
        s["H"].data_ptr(), s["D"].data_ptr(), s["Q"].data_ptr(), s["gamma"].data_ptr(),
        s["hd"].data_ptr(), s["sd"].data_ptr(), s["dd"].data_ptr(), s["sq"].data_ptr(), None,
        pb.t["n0"].data_ptr(), pb.t["nel"].data_ptr(), 300.0 * radii.KELVIN2AU, 250, 1e-10,
        pb.t["order"].data_ptr(), out["P"].data_ptr(), out["W"].data_ptr(), out["C"].data_ptr(),
        out["ev"].data_ptr(), out["occ"].data_ptr(), out["q"].data_ptr(), out["dp"].data_ptr(),
        out["qp"].data_ptr(), out["vorb"].data_ptr(), out["vdp"].data_ptr(), out["vqp"].data_ptr(),
        out["en"].data_ptr(), status.data_ptr(), _lib.stream_ptr())
    torch.cuda.synchronize()
    assert rc == 0 and int(status[0]) == 0
    assert abs(float(out["en"][:2].sum() - s["energies"][:2].sum())) <= E_TOL
    assert (out["P"] - s["P"][:nm]).abs().max().item() <= 1e-8
    assert (out["W"] - s["W"][:nm]).abs().max().item() <= 1e-8
    assert (out["ev"] - s["evals"][:n]).abs().max().item() <= 1e-8


@pytest.mark.parametrize("lanes", [1, 40])
def test_teams_by_share_match_one_cta(lanes):
    """Both sides of every size where the team changes (for a lone batch and
    for one that shares the SMs) against one CTA per molecule. Residuals of
    1e-10 enter energies squared and forces times a response of about 10."""
    from dxtb_gb300 import _lib
    from dxtb_gb300.calculators import tables
    from dxtb_gb300.engine import PackedBatch, run, scf_launches

    L = _lib.lib()
    mols = [_molecule(n) for n in (9, 29, 30, 59, 60, 89, 90, 129, 130, 136)]
    pb = PackedBatch(tables("gfn2"), [m[0] for m in mols], [torch.tensor(m[1]) for m in mols])
    pb.lanes = lanes
    thr = (C.c_int32 * 5)()
    assert L.dxtb_scf_team_sizes(pb._nao32.ctypes.data, pb.nmol, lanes, thr) == 0
    got = tuple(thr)
    assert list(got) == sorted(got) and got[0] <= 136
    if lanes == 1:  # few molecules: the largest teams that pay
        assert got[0] <= 32 and got[1:] == (60, 60, 90, 130) and scf_launches(got, 136) == 6
    else:
        assert got[1] > 60
    r = run(pb, forces=True, tol=1e-10)
    assert (r.status.cpu() == 0).all()
    e, g = r.energy.cpu().clone(), r.gradient.cpu().clone()
    saved = (C.c_int32 * 5)()
    assert L.dxtb_scf_get_size_classes(saved) == 0
    try:
        assert L.dxtb_scf_set_size_classes((C.c_int32 * 5)(*range(1000, 1005))) == 0
        assert L.dxtb_scf_team_sizes(pb._nao32.ctypes.data, pb.nmol, lanes, thr) == 0
        assert tuple(thr) == (1000, 1001, 1002, 1003, 1004)  # a set policy holds
        ref = run(pb, forces=True, tol=1e-10)
    finally:
        assert L.dxtb_scf_set_size_classes(saved) == 0
    assert (ref.energy.cpu() - e).abs().max() <= 1e-10
    assert (ref.gradient.cpu() - g).abs().max() <= 1e-8
    bad = (C.c_int32 * 5)(3, 2, 4, 5, 6)
    assert L.dxtb_scf_team_sizes(None, pb.nmol, lanes, thr) != 0
    assert L.dxtb_scf_team_sizes(pb._nao32.ctypes.data, pb.nmol, 0, thr) != 0
    assert L.dxtb_scf_teams(*[None] * 15, 0.0, *[None] * 21, bad, None) != 0
