"""
SCFs that end on the default 1e-4 of the Anderson mixer, of small molecules
with a small gap: 30 and more steps, mixing systems that are singular to working
precision, and forces that follow the last bit of every operation by up to 1e-6
of their size. They keep the float64 path, and so the forces that were recorded
with it before the digit planes came (golden/loose_scf.npz, written on a GB300
by commit c74580e; geometries among them where the planes gave others).

Equal bits in the SCF leave the order of the sums in the gradient: some 1000
terms of up to 10 Eh/Bohr, 1e-13; the bound is 1e-12. Alone and among others the
molecules run on other teams by their share of the batch, but up to 32 orbitals
not here.
"""

from pathlib import Path

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

OPTS = dict(tol=1e-4, maxiter=100, scf={"mixer": "anderson", "x_atol": 1e-4, "f_atol": 1e-4})


@pytest.mark.parametrize("method", ["gfn1", "gfn2"])
@pytest.mark.parametrize("copies", [0, 1, 40])
def test_forces_of_the_float64_path(method, copies):
    from dxtb_gb300.calculators import tables
    from dxtb_gb300.engine import PackedBatch, run

    d = np.load(Path(__file__).parent / "golden" / "loose_scf.npz")
    off, grad = d[f"{method}_off"], d[f"{method}_gradient"]
    z, pos = d[f"{method}_numbers"].astype(np.int64), torch.tensor(d[f"{method}_positions"])
    mols = [(z[a:b], pos[a:b]) for a, b in zip(off[:-1], off[1:])]
    batches = [mols * copies] if copies else [[m] for m in mols]  # 0: each alone
    got, its = [], []
    for mol in batches:
        pb = PackedBatch(tables(method), [m[0] for m in mol], [m[1] for m in mol])
        assert int(pb.nao.max()) <= 32
        r = run(pb, forces=True, **OPTS)
        assert (r.status.cpu() == 0).all()
        got.append(r.gradient.cpu().numpy())
        its.append(r.iterations.cpu().numpy())
    got = np.concatenate(got).reshape(max(copies, 1), len(grad), 3)
    assert (np.concatenate(its).reshape(-1, len(mols)) == d[f"{method}_iterations"]).all()
    assert np.abs(got - grad).max() <= 1e-12


@pytest.mark.parametrize("n", [31, 32, 33, 34])
def test_the_launches_that_are_counted(n):
    """Alone, molecules of 30 orbitals and more take a CTA of 512 threads, loose
    Anderson SCFs from 33 on: one class fewer, of which a call launches one SCF
    and, with forces, three gradient kernels."""
    from dxtb_gb300.calculators import tables
    from dxtb_gb300.engine import PackedBatch, run
    from dxtb_gb300.workloads import build_geometry

    heavy, nh = (n - 2) // 6, n - 4 * ((n - 2) // 6)
    z, pos = build_geometry(np.random.default_rng(n), [7 if nh % 2 else 6] + [6] * (heavy - 1), nh)
    pb = PackedBatch(tables("gfn2"), [z], [torch.tensor(pos)])
    assert int(pb.nao[0]) == n
    assert run(pb, forces=True).launches == 3 + 2 * 4
    r = run(pb, forces=True, **OPTS)
    assert int(r.status[0]) == 0 and r.launches == 3 + (1 if n <= 32 else 2) * 4
