"""
The digit products (csrc/eigemm.cuh) where their float32 sums are carried: six
digits carry order 2 every 32 terms and all orders every 64, three digits all
every 128. Sizes on both sides of one and two full carries, on one CTA of
either size and on clusters, and an overlap that is nearly singular.

The other side is the float64 path of the same call (workspaces without planes):
Householder vectors and float64 products, none of the kernels under test. Both
SCFs end on 1e-10, which enters energies squared and first-order quantities by a
response of about 10: 1e-10 and 1e-8. Operands have 60 bits and results 58, so
that C S C^T = 1 and P = C^T occ C hold to 140 x 2^-58 x |C|^2 < 1e-12 (the bound
adds a decade).
"""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _both(pb_of, classes=None):
    from dxtb_gb300.engine import run

    out = []
    for planes in (True, False):
        pb = pb_of()
        pb.classes = classes
        if not planes:
            pb.drop_planes()
        r = run(pb, forces=True, tol=1e-10)
        assert (r.status == 0).all()
        out.append(r)
    return pb, *out


def _agree(pb, a, b, e_tol=1e-10, f_tol=1e-8, ortho=1e-11):
    assert (a.energy - b.energy).abs().max() <= e_tol
    assert (a.gradient - b.gradient).abs().max() <= f_tol
    for k, t in (("P", "mat"), ("W", "mat"), ("evals", "aos"), ("q", "aos")):
        n = pb.total[t]
        assert (a.state[k][:n] - b.state[k][:n]).abs().max() <= f_tol, k
    for m in range(pb.nmol):
        n, at, o = int(pb.nao[m]), int(pb.mat_off[m]), int(pb.ao_off[m])
        s, p, c = (a.state[k][at : at + n * n].view(n, n) for k in ("S", "P", "C"))
        k = int((c.abs().sum(1) > 0).sum())
        c, occ = c[:k], a.state["occ"][o : o + k]
        assert (c @ s @ c.T - torch.eye(k, device=c.device)).abs().max() <= ortho
        assert (c.T @ (occ[:, None] * c) - p).abs().max() <= ortho


def _molecule(n: int):
    """A random molecule of exactly n GFN2 orbitals."""
    from dxtb_gb300.workloads import build_geometry

    heavy = (n - 2) // 6
    nh = n - 4 * heavy
    return build_geometry(np.random.default_rng(40 + n), [7 if nh % 2 else 6] + [6] * (heavy - 1), nh)


@pytest.mark.parametrize("classes", [(900, 901, 902, 903, 904), (1, 901, 902, 903, 904), (1, 1, 1, 903, 904),
                                     (1, 1, 1, 1, 1)])
def test_both_sides_of_a_carry(classes):
    from dxtb_gb300.calculators import tables
    from dxtb_gb300.engine import PackedBatch

    sizes = (31, 32, 33, 63, 64, 65, 80, 81, 127, 128, 129)
    mols = [_molecule(n) for n in sizes]
    pb, a, b = _both(lambda: PackedBatch(tables("gfn2"), [m[0] for m in mols], [torch.tensor(m[1]) for m in mols]),
                     classes)
    assert tuple(pb.nao) == sizes
    _agree(pb, a, b)


@pytest.mark.parametrize("method,d,smallest", [("gfn2", 0.1, 2e-3), ("gfn2", 0.01, 2e-5), ("gfn1", 0.1, 2e-3)])
def test_nearly_dependent_basis(method, d, smallest):
    """Two hydrogen atoms d Bohr apart: X = L^-1, from which P is built, has rows
    of norm 1 / sqrt(smallest eigenvalue of S), where P has entries of order 1. The
    errors of both paths grow with the inverse of that eigenvalue."""
    from dxtb_gb300.calculators import tables
    from dxtb_gb300.engine import PackedBatch
    from dxtb_gb300.workloads import build_geometry

    z, pos = build_geometry(np.random.default_rng(7), [6] * 10 + [8], 16)
    h = np.flatnonzero(z == 1)
    pos = pos.copy()
    pos[h[1]] = pos[h[0]] + d * np.array([1.0, 2.0, -1.0]) / np.sqrt(6.0)
    pb, a, b = _both(lambda: PackedBatch(tables(method), [z], [torch.tensor(pos)]))
    n = int(pb.nao[0])
    lam = torch.linalg.eigvalsh(a.state["S"][: n * n].view(n, n).cpu())[0].item()
    assert 0.0 < lam < smallest
    _agree(pb, a, b, e_tol=1e-9, ortho=1e-12 / lam)
