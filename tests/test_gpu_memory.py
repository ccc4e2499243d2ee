"""
Calls whose digit planes do not fit still run: a batch falls back to float64
workspaces, the Hessian's points go in several packs, a served request within
its budget runs without planes.

SCFs converged to 1e-10 on two paths: energies to 1e-9, forces to 1e-8; Hessian
elements are forces' differences over 2e-3 Bohr, 1e-5 at most and as a rule
1e-8: bound 1e-6.
"""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_batch_without_room_for_the_planes():
    """The allocator is held to what the float64 workspaces need (a limit of
    PyTorch's own, taken back at the end)."""
    from dxtb_gb300.calculators import tables
    from dxtb_gb300.engine import GraphStep, PackedBatch, point_bytes, run
    from dxtb_gb300.workloads import config_molecules

    mols = config_molecules(2)[:160]
    tb = tables("gfn2")

    def batch():
        return PackedBatch(tb, [m[0] for m in mols], [torch.tensor(m[1]) for m in mols])

    pb = batch()
    ref = run(pb, forces=True)
    e, g = ref.energy.clone(), ref.gradient.clone()
    sizes = list(zip(pb.nao.tolist(), pb.nat.tolist(), pb.nsh.tolist()))
    bare, full = (sum(point_bytes(tb, *s, planes=p) for s in sizes) for p in (False, True))
    assert full - bare > 200 << 20
    del ref, pb
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    try:
        torch.cuda.set_per_process_memory_fraction(
            (torch.cuda.memory_reserved() + bare + (100 << 20)) / total)
        pb = batch()
        with pytest.warns(UserWarning, match="digit planes"):
            r = run(pb, forces=True)
        assert not pb.planes and (r.status == 0).all()
        assert (r.energy - e).abs().max() <= 1e-9
        assert (r.gradient - g).abs().max() <= 1e-8
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    step = GraphStep(pb, forces=True)  # the batch keeps its layout, captured too
    r = step.replay([torch.tensor(m[1]) for m in mols])
    assert not pb.planes and (r.energy - e).abs().max() <= 1e-9


def test_a_captured_step_outlives_the_planes_of_its_batch():
    """A graph captured with planes keeps its layout when the batch drops them."""
    from dxtb_gb300.calculators import tables
    from dxtb_gb300.engine import GraphStep, PackedBatch, run
    from dxtb_gb300.workloads import config_molecules

    mols = config_molecules(2)[:12]
    pb = PackedBatch(tables("gfn2"), [m[0] for m in mols], [torch.tensor(m[1]) for m in mols])
    step = GraphStep(pb, forces=True)
    e = step.first.energy.clone()
    pb.drop_planes()
    assert (run(pb, forces=True).energy - e).abs().max() <= 1e-9
    junk = [torch.full((256,), -1, dtype=torch.int64, device="cuda") for _ in range(64)]
    assert (step.replay().energy - e).abs().max() <= 1e-10
    del junk


def test_no_memory_for_a_captured_step():
    """A calculator whose graph does not fit beside its state launches eagerly,
    with the planes it has."""
    from dxtb_gb300 import GFN2Calculator
    from dxtb_gb300.workloads import config_molecules

    mols = config_molecules(2)[:31]
    nat = max(len(z) for z, _ in mols)
    num, pos = torch.zeros(len(mols), nat, dtype=torch.int64), torch.zeros(len(mols), nat, 3, dtype=torch.float64)
    for i, (z, p) in enumerate(mols):
        num[i, : len(z)], pos[i, : len(z)] = torch.as_tensor(z), torch.as_tensor(p)
    opts = {"exclude": ["disp", "d4sc"], "guess": "sad", "scf_mode": "implicit", "x_atol": 1e-10,
            "f_atol": 1e-10, "maxiter": 250}
    calc = GFN2Calculator(num, opts=opts, device="cuda")
    e = calc.get_energy(pos.cuda()).clone()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    try:
        torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (40 << 20)) / total)
        calc.reset()
        with pytest.warns(UserWarning, match="capture failed"):
            again = calc.get_energy(pos.cuda())
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert calc._pb.planes and (again - e).abs().max() <= 1e-10


@pytest.mark.parametrize("method", ["gfn1", "gfn2"])
def test_hessian_in_packs(method):
    from dxtb_gb300.calculators import tables
    from dxtb_gb300.engine import point_bytes
    from dxtb_gb300.hessian import hessian
    from dxtb_gb300.workloads import random_molecule

    z, pos = random_molecule(7004, 7)
    tb = tables(method)
    one, mu = hessian(tb, z, pos, matrix=True, dipole_derivative=True)
    n = int(tb.el_nao[z].sum())
    each = point_bytes(tb, n, len(z), int(tb.el_nsh[z].sum())) + 8 * 13 * n * n
    for packs in (1, 5, 41):  # one point at a time; a count that does not divide 42; all but one
        h, m = hessian(tb, z, pos, matrix=True, dipole_derivative=True, max_bytes=packs * each)
        assert (h - one).abs().max() <= 1e-6 and (m - mu).abs().max() <= 1e-6
    with pytest.raises(ValueError, match="empty batch"):
        hessian(tb, np.zeros(0, dtype=np.int64), np.zeros((0, 3)))


def test_a_request_that_the_budget_holds_without_planes():
    from dxtb_gb300.engine import point_bytes
    from dxtb_gb300.serving import CudaExecutor, Request, Server
    from dxtb_gb300.workloads import random_molecule

    z, pos = random_molecule(8200, 40)
    ex = CudaExecutor(slots=1)
    tb = ex.tables["gfn2"]
    size = (int(tb.el_nao[z].sum()), len(z), int(tb.el_nsh[z].sum()))
    bare, full = (point_bytes(tb, *size, planes=p) for p in (False, True))
    out = {}
    for budget in (full, (bare + full) // 2, bare - 1):
        srv = Server(ex, hbm_budget=budget, slots=1)
        (out[budget],) = srv.serve([Request(0, "gfn2", z, pos)])
        assert srv.stats.max_bytes <= budget
    a, b, c = out.values()
    assert a.status == 0 and b.status == 0 and c.error is not None
    assert abs(a.energy - b.energy) <= 1e-9 and np.abs(a.forces - b.forces).max() <= 1e-8
