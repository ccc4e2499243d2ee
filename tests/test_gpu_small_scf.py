"""
Molecules of up to 12 orbitals keep the float64 path and the order of its
operations in the implicit mode too: forces converged to 1e-10, whose last bits a
Hessian multiplies by 500. Recorded forces (golden/small_scf.npz, written on a
GB300 by commit c74580e, before the digit planes; the geometries whose forces
moved most, by up to 1e-11, when the mixer's sums were fused). Equal bits in the
SCF leave the order of the gradient's sums: 1e-13, the bound is 1e-12.
"""

from pathlib import Path

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method", ["gfn1", "gfn2"])
@pytest.mark.parametrize("copies", [0, 1, 30])
def test_forces_of_the_float64_path(method, copies):
    from dxtb_gb300.calculators import tables
    from dxtb_gb300.engine import PackedBatch, run

    d = np.load(Path(__file__).parent / "golden" / "small_scf.npz")
    off, grad = d[f"{method}_off"], d[f"{method}_gradient"]
    z, pos = d[f"{method}_numbers"].astype(np.int64), torch.tensor(d[f"{method}_positions"])
    mols = [(z[a:b], pos[a:b]) for a, b in zip(off[:-1], off[1:])]
    got, its = [], []
    for mol in [mols * copies] if copies else [[m] for m in mols]:  # 0: each alone
        pb = PackedBatch(tables(method), [m[0] for m in mol], [m[1] for m in mol])
        assert int(pb.nao.max()) <= 12
        r = run(pb, forces=True, tol=1e-10)
        assert (r.status.cpu() == 0).all()
        got.append(r.gradient.cpu().numpy())
        its.append(r.iterations.cpu().numpy())
    got = np.concatenate(got).reshape(max(copies, 1), len(grad), 3)
    assert (np.concatenate(its).reshape(-1, len(mols)) == d[f"{method}_iterations"]).all()
    assert np.abs(got - grad).max() <= 1e-12
