"""
The SMs that the admission loop counts for a pack are those that the pack's
launch takes: teams follow each molecule's share of its pack and the number of
slots.
"""

import numpy as np
import pytest

from dxtb_gb300.serving import Request, Server


class _Fake:
    """Teams of 16 SMs for a pack of one, 16 / len of the pack for more."""

    def __init__(self):
        self.packs = []

    norb = staticmethod(lambda r: 2 * len(r.numbers))
    nbytes = staticmethod(lambda r: 1)

    def pack_sms(self, reqs):
        return len(reqs) * (16 // len(reqs))

    def team_sms(self, r):
        return 16

    def launch(self, reqs, slot):
        self.packs.append([r.rid for r in reqs])
        return reqs

    def ready(self, h):
        return False


def _req(rid, nat):
    return Request(rid, "gfn2", np.ones(nat, dtype=np.int64), np.zeros((nat, 3)))


def test_a_pack_counts_the_teams_it_takes():
    ex = _Fake()
    srv = Server(ex, slots=4, large_slots=3, large_n=200, large_pack=4, order="size", large_sms=40,
                 clock=lambda: 0.0)
    for rid, nat in enumerate([10] + [150] * 9):
        srv.submit(_req(rid, nat))
    srv.pump()
    assert sorted(len(p) for p in ex.packs) == [1, 4, 4]
    assert srv.sms_used == 32  # two packs of four; the ninth (16 SMs alone) waits
    assert len(srv.queues["large"]) == 1


@pytest.mark.gpu
@pytest.mark.parametrize("slots", [1, 8, 12])
def test_counted_teams_are_the_launched_ones(slots):
    """Around the fixed thresholds of the size classes, alone and in packs:
    the launch has one SCF kernel for each class up to its largest molecule's."""
    from dxtb_gb300.serving import CudaExecutor
    from dxtb_gb300.workloads import random_molecule

    ex = CudaExecutor(slots=slots, maxiter=2)
    reqs = [Request(i, "gfn2", *random_molecule(8100 + i, nat), forces=False)
            for i, nat in enumerate((50, 52, 86, 128, 168))]
    assert {100 < ex.norb(r) < 450 for r in reqs} == {True}

    def launched(pack):  # SMs of the largest molecule's team
        h = ex.launch(pack, 0)
        h["event"].synchronize()
        classes = h["res"].launches - 3
        ex.collect(h)
        return 1 if classes <= 2 else 1 << (classes - 2)

    for r in reqs:
        assert ex.team_sms(r) == launched([r])
    for k in (2, 5):
        pack = sorted(reqs, key=ex.norb)[-k:]
        alone = [ex.team_sms(r) for r in pack]
        total = ex.pack_sms(pack)
        assert launched(pack) <= total <= sum(alone)
        assert ex.pack_sms([pack[-1]] * 16) == 16 * launched([pack[-1]] * 16)
