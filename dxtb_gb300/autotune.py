"""
Autotuner of the SCF launch policy: the orbital-count thresholds of the size
classes (``dxtb_scf_set_size_classes``), i.e. which molecules run as one CTA
of 256 threads two per SM, one CTA of 512 threads per SM, or a thread-block
cluster of 2, 4, 8 or 16 CTAs.

``ensure(pb)`` gives the packed batch ``pb`` its thresholds (``pb.classes``):
a choice cached for this GPU and batch shape, or one tuned once per process and
device. No other batch sees them. ``tune(pb)`` is the explicit call: it times
the batch (energy + forces, CUDA events on the current stream, the median of
``reps`` runs after one warm-up) under each candidate threshold set, sets the
fastest for the whole process (``set_classes``) and caches it on disk, keyed by
the GPU (name, SM count), the library build and a signature of the batch's size
distribution. While such a process-wide set is in force ``ensure`` leaves it.
Setting ``DXTB_AUTOTUNE=0`` keeps the library's defaults. The choice changes
only the team each molecule runs on, so results agree to rounding.

The reference has no counterpart: its batched SCF is a padded tensor
program whose shapes PyTorch dispatches.
"""

from __future__ import annotations

import ctypes as C
import hashlib
import json
import os
import time
from pathlib import Path

import numpy as np
import torch

from . import _lib, build

DEFAULT = (112, 136, 160, 320, 640)
# thresholds of classes 1..5 (one-SM CTA, clusters of 2, 4, 8, 16); the default
# stands for the rule by the molecule's share of the batch (dxtb_scf_team_sizes)
CANDIDATES = [
    DEFAULT,
    (80, 136, 160, 320, 640),
    (80, 112, 140, 320, 640),
    (96, 136, 180, 240, 320),
    (112, 160, 220, 260, 320),
    (30, 80, 110, 140, 640),
]
_applied: dict = {}


def cache_path() -> Path:
    root = os.environ.get("DXTB_CACHE_DIR") or os.path.join(
        os.environ.get("XDG_CACHE_HOME") or os.path.expanduser("~/.cache"), "dxtb_gb300")
    return Path(root) / "autotune.json"


def _device_key(dev: torch.device) -> str:
    p = torch.cuda.get_device_properties(dev)
    lib = build.LIB
    stamp = str(int(lib.stat().st_mtime)) if lib.exists() else "nolib"
    return f"{p.name}|{p.multi_processor_count}|{stamp}"


def _batch_key(pb) -> str:
    # the size distribution decides the policy: a histogram of orbital counts
    h, _ = np.histogram(pb.nao, bins=[0, 64, 96, 112, 128, 136, 144, 160, 192, 256, 320, 384, 640, 768,
                                      1 << 20])
    frac = np.round(h / max(1, pb.nmol), 2)
    return hashlib.sha1(f"{pb.tables.method}|{pb.nmol // 64}|{frac.tolist()}".encode()).hexdigest()[:16]


def set_classes(thr) -> None:
    arr = (C.c_int32 * 5)(*[int(v) for v in thr])
    _lib.check(_lib.lib().dxtb_scf_set_size_classes(arr), "size classes")


def get_classes() -> tuple:
    arr = (C.c_int32 * 5)()
    _lib.check(_lib.lib().dxtb_scf_get_size_classes(arr), "size classes")
    return tuple(int(v) for v in arr)


def _time(pb, state: dict, reps: int) -> float:
    from .engine import run

    run(pb, forces=True, state=state)
    times = []
    for _ in range(reps):
        s, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        s.record()
        run(pb, forces=True, state=state)
        e.record()
        e.synchronize()
        times.append(s.elapsed_time(e))
    return float(np.median(times))


def _measure(pb, candidates, reps: int) -> dict:
    """Times every candidate on ``pb`` and returns the choice; ``pb`` and the
    process keep their thresholds. Only to be called under the default set."""
    state: dict = {}
    ms = {}
    before = pb.classes
    try:
        for c in candidates:
            pb.classes = None if c == DEFAULT else c
            ms[c] = _time(pb, state, reps)
    finally:
        pb.classes = before
    best = min(ms, key=ms.get)
    # the rule gives way for 5 % or more: runs of one candidate differ by up to 3 %
    if DEFAULT in ms and ms[best] > 0.95 * ms[DEFAULT]:
        best = DEFAULT
    return {"thresholds": list(best), "ms": {",".join(map(str, c)): v for c, v in ms.items()},
            "source": "tuned", "when": time.strftime("%Y-%m-%dT%H:%M:%S")}


def _save(pb, out: dict) -> None:
    path = cache_path()
    try:
        path.parent.mkdir(parents=True, exist_ok=True)
        data = json.loads(path.read_text()) if path.exists() else {}
        data.setdefault(_device_key(pb.device), {})[_batch_key(pb)] = out
        path.write_text(json.dumps(data, indent=1))
    except OSError:
        pass  # a read-only cache location only costs a re-tune


def tune(pb, candidates=None, reps: int = 3, save: bool = True) -> dict:
    """Times every candidate on ``pb``, applies the fastest process-wide and
    returns it: {"thresholds": [...], "ms": {candidate: median ms}, "source":
    "tuned"}."""
    before = get_classes()
    set_classes(DEFAULT)
    try:
        out = _measure(pb, [tuple(c) for c in (candidates or CANDIDATES)], reps)
    except BaseException:
        set_classes(before)
        raise
    set_classes(out["thresholds"])
    if save:
        _save(pb, out)
    return out


def ensure(pb, min_molecules: int = 32) -> dict:
    """Gives ``pb`` the cached thresholds for this GPU and batch shape, tuning
    once if none are cached. Batches below ``min_molecules``, and all while a
    set other than the default is in force for the process, keep theirs."""
    now = get_classes()
    if os.environ.get("DXTB_AUTOTUNE", "1") == "0" or pb.nmol < min_molecules:
        return {"thresholds": list(now), "source": "default"}
    if now != DEFAULT:
        return {"thresholds": list(now), "source": "set"}
    dkey, bkey = _device_key(pb.device), _batch_key(pb)
    res = _applied.get((dkey, bkey))
    if res is None:
        try:
            hit = json.loads(cache_path().read_text())[dkey][bkey]
            res = dict(hit, source="cache", thresholds=[int(v) for v in hit["thresholds"]])
        except (OSError, KeyError, TypeError, ValueError):
            res = _measure(pb, CANDIDATES, 3)
            _save(pb, res)
        _applied[(dkey, bkey)] = res
    thr = tuple(res["thresholds"])
    pb.classes = None if thr == DEFAULT else thr
    return res
