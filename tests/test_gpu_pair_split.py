"""
How the geometry and gradient kernels share their pairs out, against the oracle
and against each other: few shell pairs (several lanes for an s-s or s-p pair)
and many (a lane each), odd numbers of p-p pairs (two at a time), d shells,
one atom, 8 and 9 atoms (a CTA takes 8), 33 atoms (a warp's lanes go round).

The forces of a molecule alone and in a batch are sums of the same terms in
another order over an SCF converged to 1e-10: 1e-9. Against the oracle the
bounds of the other parity tests (1e-8 Eh, 1e-6 Eh/Bohr).
"""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _mols():
    from dxtb_gb300.workloads import build_geometry

    rng = np.random.default_rng(5)
    return [(np.array([2]), np.zeros((1, 3)))] + [
        build_geometry(rng, heavy, nh)
        for heavy, nh in (([6], 4), ([16], 2), ([7, 6], 5), ([16, 8], 6), ([6, 16, 7], 6), ([6] * 9 + [8, 16], 22))
    ]


@pytest.mark.parametrize("method", ["gfn1", "gfn2"])
@pytest.mark.parametrize("copies", [1, 24])
def test_forces_of_few_and_many_pairs(method, copies):
    from dxtb_gb300.calculators import tables
    from dxtb_gb300.engine import PackedBatch, run
    from oracle import xtb_oracle as X

    mols = _mols()
    assert {len(z) for z, _ in mols} >= {1, 8, 9, 33}
    pb = PackedBatch(tables(method), [z for z, _ in mols] * copies, [torch.tensor(p) for _, p in mols] * copies)
    r = run(pb, forces=True, tol=1e-10)
    assert (r.status.cpu() == 0).all()
    g, e = r.gradient.cpu().numpy(), r.energy.cpu().numpy()
    at = np.concatenate([[0], np.cumsum(pb.nat)])
    for i, (z, p) in enumerate(mols):
        alone = run(PackedBatch(tables(method), [z], [torch.tensor(p)]), forces=True, tol=1e-10)
        for k in range(i, pb.nmol, len(mols)):
            assert np.abs(g[at[k] : at[k + 1]] - alone.gradient.cpu().numpy()).max() <= 1e-9
        if copies == 1:
            ref = X.singlepoint(method, z, p, grad=True, tol=1e-10)
            assert abs(e[i] - ref.energy) <= 1e-8
            assert np.abs(g[at[i] : at[i + 1]] - ref.extra["gradient"].numpy()).max() <= 1e-6
