"""Autotuner of the work decomposition of the class kernels.

Knobs, each chosen by timing on the device (CUDA events on the launching stream):

* ``team`` — lanes per quartet of the register kernel (light classes): each quartet's
  primitive loop is split over `team` lanes (1..32) and the partial [e0|f0] summed with warp
  shuffles.  Few primitives favour small teams, heavily contracted quartets large ones.
* ``variant`` — the heavy classes' kernel: the quadrature kernel (0); the others (1, 2) are
  slower on every workload's blocks together and round differently, so the tuner offers 0 only.
* ``ctas_per_sm`` — the register kernel's grid cap, in resident CTAs per SM (2..16): more
  CTAs shorten the tail of a block, fewer stage the Boys table fewer times.
* ``streams`` — how many concurrent streams the class blocks of a call are spread over
  (class-block grouping: blocks go round robin, largest first, to that many streams).

Per-block knobs are timed with the blocks run one after another (``set_profiling(2)``); the
stream count is timed on whole unique-integral calls.  ``EriBatch.autotune`` does the same for
the block types of a batch.  Choices are stored in a JSON cache keyed by class and log2 of
the block's mean primitive quartets per shell quartet (team: ``"abcd:k"``, variant:
``"v:abcd:k"``, grid cap: ``"c:abcd:k"``; stream count: ``"streams"``), so a new basis or
batch of similar shape starts tuned (``DeviceBasis`` and ``EriBatch`` apply the cache on
creation).  The file names the generation of the kernels that it was measured on (``KERNELS``): a
file of another generation, or of none, is not used.  gbasis has no counterpart: it evaluates one
quartet at a time in NumPy.
"""
from __future__ import annotations

import functools
import json
import math
import os

import numpy as np

from . import _engine

__all__ = ["autotune", "apply_cache", "cache_path", "TEAMS", "CTAS", "STREAMS"]

TEAMS = (1, 2, 4, 8, 16, 32)
CTAS = (2, 4, 8, 16)
STREAMS = (1, 2, 4, 6, 8, 12, 16)
VARIANTS = (0,)
# Generation of the class kernels: raised when a class changes its kernel, its kernel changes what
# a knob does or is best at, or a variant number changes its meaning.  1 had no tag: its variant 1
# was the faster one for many classes that now run 3 to 14 times slower on it than by default, and
# its lane counts belong to another recursion.
KERNELS = 2


# register classes beyond the limit below, after the swap (gen_eri.is_register)
_LARGER = {(3, 0, 2, 0), (3, 1, 1, 0), (3, 0, 1, 1), (2, 2, 1, 0), (1, 3, 1, 0), (3, 3, 0, 0)}


def light_class(cls4):
    """Classes run by the register kernel (the only ones whose team matters): the [e0|f0]
    accumulators and the (ab|cd) block of one quartet fit one thread (170 doubles, the limit
    the kernel generator uses), or, with an s shell's pair run on its other shell, one of six
    larger ones."""
    def nc(l):
        return (l + 1) * (l + 2) // 2
    la, lb, lc, ld = cls4
    ne = sum(nc(e) for e in range(la, la + lb + 1))
    nf = sum(nc(f) for f in range(lc, lc + ld + 1))
    swapped = ((la, lb) if la else (lb, la)) + ((lc, ld) if lc else (ld, lc))
    return ne * nf + nc(la) * nc(lb) * nc(lc) * nc(ld) <= 170 or swapped in _LARGER


def cache_path():
    return os.environ.get("GBX_TUNE_CACHE",
                          os.path.join(os.path.dirname(os.path.abspath(__file__)), "tuning.json"))


@functools.lru_cache(maxsize=4096)
def _bucket_key(cls4, bucket):
    return "%d%d%d%d:%d" % (*cls4, bucket)


def _key(cls4, avg_prims):
    return _bucket_key(cls4, int(round(math.log2(max(avg_prims, 1.0)))))


_loaded = {}  # path -> (modification time, table): read once per change of the file


def _load():
    path = cache_path()
    try:
        mtime = os.stat(path).st_mtime_ns
        hit = _loaded.get(path)
        if hit and hit[0] == mtime:
            return dict(hit[1])
        with open(path) as f:
            table = json.load(f)
        if table.pop("kernels", None) != KERNELS:
            table = {}
        _loaded[path] = (mtime, table)
        return dict(table)
    except (OSError, ValueError):
        return {}


def _store(chosen):
    """The cache file with the choices ``chosen``, without entries of another generation and without
    variants and grid caps that are the default (looked up on every creation for nothing)."""
    table = {**_load(), **chosen, "kernels": KERNELS}
    table = {k: v for k, v in table.items()
             if not (k.startswith("v:") and v == 0 or k.startswith("c:") and v == 8)}
    with open(cache_path(), "w") as f:
        json.dump(table, f, indent=1, sort_keys=True)


# Threads that keep the device busy: 148 SMs of 8 warps, two per scheduler.  Entries as they are,
# this bound, twice it and four times it: one (dp|ps) quartet 0.60, 0.42, 0.42, 0.43 ms, resident s-f
# chain of 7 atoms 6.75, 6.87, 6.96, 7.05 ms, 60-molecule batch 12.58, 12.57, 12.63, 12.68 ms.
FILL = 148 * 256
# Threads below which more lanes than the rule's pay: 148 SMs of 2 warps.  Where a list has more, the
# call's other lists need the room (resident spd tensor of 8 atoms with entries above the rule on every
# list, below FILL threads, below half, below a quarter, on none: 1.924, 1.909, 1.886, 1.871, 1.884 ms;
# of 2 atoms 243, 239, 237, 238, 252 us).
FEW = FILL // 4


def _lanes(entry, team, quartets):
    """Lanes per quartet for a block whose rule says ``team`` and whose cache entry is ``entry``,
    measured with the device to itself.  Fewer lanes than the rule's leave less to add up where the
    list is long: a shorter one takes as many more, up to the rule's, as it needs to fill the
    device.  More lanes shorten each quartet: only where the rule leaves the device nearly empty."""
    if entry > team:
        return entry if quartets * team < FEW else team
    while entry < team and quartets * entry < FILL:
        entry *= 2
    return entry


def apply_cache(db, table=None):
    """Set the knobs of every block whose (class, primitive bucket) the cache knows (lanes as
    ``_lanes`` takes them for the block's length), or ``table``, used as it is, and the stream
    count; returns how many blocks changed."""
    lanes = _lanes if table is None else (lambda entry, team, quartets: entry)
    table = _load() if table is None else table
    configs = any(key.startswith(("v:", "c:")) for key in table)
    n = 0
    for k, (cls4, team, avg, quartets) in enumerate(db.blocks()):
        key = _key(cls4, avg)
        t = table.get(key)
        t = lanes(t, team, quartets) if t else team
        if t != team:
            db.set_team(k, int(t))
            n += 1
        if not configs:
            continue
        v, c = table.get("v:" + key), table.get("c:" + key)
        if v is not None or c is not None:
            db.set_block_config(k, int(v or 0), int(c or 8))
            n += 1
    if table.get("streams"):
        db.set_streams(int(table["streams"]))
    return n


def _call_ms(db, reps):
    import torch
    st = torch.cuda.current_stream()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    best = float("inf")
    for _ in range(reps):
        e0.record(st)
        db.unique(stream=__import__("ctypes").c_void_p(st.cuda_stream))
        e1.record(st)
        e1.synchronize()
        best = min(best, e0.elapsed_time(e1))
    return best


def _pick(values, times, current):
    """The fastest value, or the current one where none is 3 % faster (runs differ by 1 to 2 %)."""
    values, best = list(values), int(np.argmin(times))
    if current in values and times[values.index(current)] * 0.97 <= times[best]:
        return current
    return values[best]


def _sweep(db, blocks, ks, values, setter, reps):
    """Per-block times (values x blocks) of each value of one knob, blocks run in order."""
    times = np.full((len(values), len(blocks)), np.inf)
    for vi, v in enumerate(values):
        for k in ks:
            setter(k, v)
        for _ in range(reps):
            db.unique()
            times[vi] = np.minimum(times[vi], db.block_times())
    return times


def autotune(shells, coord_types=None, reps=3, teams=TEAMS, ctas=CTAS, streams=STREAMS,
             save=True, device=None):
    """Tune the knobs of ``shells``'s class blocks (team, variant, grid cap) and the stream
    count, one knob after another with the earlier choices in place; returns the chosen
    {key: value} and the per-knob timings."""
    # the unique-integral call runs the same class kernels without the N^4 tensor
    db = _engine.DeviceBasis(shells, coord_types, device=device, tuned=False)
    db.set_profiling(2)
    blocks = db.blocks()
    keys = [_key(c4, avg) for c4, _, avg, _ in blocks]
    light = [k for k, (cls4, _, _, _) in enumerate(blocks) if light_class(cls4)]
    heavy = [k for k in range(len(blocks)) if k not in light]
    db.unique()
    chosen, timings = {}, {}
    # lanes per quartet (light classes)
    t_team = _sweep(db, blocks, light, teams, db.set_team, reps)
    for k in light:
        best = _pick(teams, t_team[:, k], blocks[k][1])
        db.set_team(k, best)
        chosen[keys[k]] = best
    timings["team"] = t_team
    # kernel variant (heavy classes) and grid cap (light classes), keeping the other default
    var = {k: 0 for k in range(len(blocks))}
    cap = {k: 8 for k in range(len(blocks))}

    def set_var(k, v):
        var[k] = v
        db.set_block_config(k, v, cap[k])

    def set_cap(k, c):
        cap[k] = c
        db.set_block_config(k, var[k], c)
    t_var = _sweep(db, blocks, heavy, VARIANTS, set_var, reps)
    for k in heavy:
        set_var(k, _pick(VARIANTS, t_var[:, k], 0))
        chosen["v:" + keys[k]] = var[k]
    timings["variant"] = t_var
    t_cap = _sweep(db, blocks, light, ctas, set_cap, reps)
    for k in light:
        set_cap(k, _pick(ctas, t_cap[:, k], 8))
        chosen["c:" + keys[k]] = cap[k]
    timings["ctas_per_sm"] = t_cap
    # stream count, on whole calls with the blocks concurrent
    db.set_profiling(0)
    t_st = []
    for n in streams:
        db.set_streams(n)
        db.unique()
        t_st.append(_call_ms(db, reps))
    chosen["streams"] = _pick(streams, np.array(t_st), 6)
    db.set_streams(chosen["streams"])
    timings["streams"] = np.array(t_st)
    if save:
        _store(chosen)
    db.close()
    return chosen, timings


def main(argv):
    """``python -m gbasis_b200.autotune medium8 chain20 batch512``: tune the named synthetic
    workloads in order (the stream count of the last single-basis workload wins; the batch keeps
    the single-basis stream count) and store the choices in the cache."""
    import torch
    from .synthetic import make_workload
    for name in argv:
        if name == "batch512":
            from .batch import EriBatch
            b = EriBatch(make_workload("batch512"))
            outs = [torch.empty((n,) * 4, dtype=torch.float64, device="cuda") for n in b.nbf]
            chosen, _ = b.autotune(outs)
            b.close()
        else:
            keep = _load().get("streams")
            chosen, _ = autotune(make_workload(name))
            if keep is not None and name != argv[0]:
                # the first single-basis workload sets the stream count
                _store({"streams": keep})
        print(name, json.dumps(chosen, sort_keys=True), flush=True)


if __name__ == "__main__":
    import sys
    main(sys.argv[1:])
