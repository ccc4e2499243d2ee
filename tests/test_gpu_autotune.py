"""
What the autotuner changes: the thresholds of the batch it is asked about, and
nothing for the batches after it. Molecules of 100-140 orbitals and the
candidate {1, 2, 3, 4, 5} (every molecule on 16 CTAs) tell the two apart.
"""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _batch(first: int, count: int):
    from dxtb_gb300.calculators import tables
    from dxtb_gb300.engine import PackedBatch
    from dxtb_gb300.workloads import config_molecules

    mols = config_molecules(2)[first : first + count]
    return PackedBatch(tables("gfn2"), [m[0] for m in mols], [torch.tensor(m[1]) for m in mols])


@pytest.fixture
def fresh(tmp_path, monkeypatch):
    from dxtb_gb300 import autotune

    monkeypatch.setenv("DXTB_CACHE_DIR", str(tmp_path))
    monkeypatch.setattr(autotune, "_applied", {})
    assert autotune.get_classes() == autotune.DEFAULT
    yield autotune
    autotune.set_classes(autotune.DEFAULT)


def test_a_tuned_batch_leaves_the_others_alone(fresh, monkeypatch):
    """ensure() tunes for its batch only: the process's classes and the launches
    of the next batch stay, from the tuner and from its cache."""
    from dxtb_gb300.engine import run

    wide = (1, 2, 3, 4, 5)
    monkeypatch.setattr(fresh, "CANDIDATES", [fresh.DEFAULT, wide])
    monkeypatch.setattr(fresh, "_time", lambda pb, state, reps: 1.0 if pb.classes == wide else 2.0)
    few, many = _batch(0, 3), _batch(0, 33)
    before = run(few).launches
    e = run(many).energy.clone()
    for source in ("tuned", "tuned", "cache"):  # timed; from this process's record; from the file
        if source == "cache":
            fresh._applied.clear()
        many, again = _batch(0, 33), _batch(0, 3)
        got = fresh.ensure(many)
        assert got["source"] == source and tuple(got["thresholds"]) == wide == many.classes
        assert fresh.get_classes() == fresh.DEFAULT
        assert fresh.ensure(again)["source"] == "default" and again.classes is None
        assert run(again).launches == before
    r = run(many)
    assert r.launches == 3 + 6  # geometry and integrals; all six classes
    assert (r.energy - e).abs().max() <= 1e-10


def test_a_set_policy_stays_and_a_failed_run_changes_nothing(fresh, monkeypatch):
    own = (64, 96, 128, 256, 512)
    fresh.set_classes(own)
    many = _batch(0, 33)
    assert fresh.ensure(many) == {"thresholds": list(own), "source": "set"}
    assert many.classes is None and fresh.get_classes() == own

    def fail(pb, state, reps):
        raise RuntimeError("no run")

    monkeypatch.setattr(fresh, "_time", fail)
    with pytest.raises(RuntimeError, match="no run"):
        fresh.tune(many)
    assert fresh.get_classes() == own and many.classes is None
    fresh.set_classes(fresh.DEFAULT)
    with pytest.raises(RuntimeError, match="no run"):
        fresh.ensure(many)
    assert fresh.get_classes() == fresh.DEFAULT and many.classes is None
