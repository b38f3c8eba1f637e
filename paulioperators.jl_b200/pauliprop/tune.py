"""Autotuner of the bucketed window-1 rotations (no counterpart in the reference).

Four settings change how fast a sequence runs, never what it computes.  The bucketing load
divisor and the rotations launched between host checks are those of an unsharded vector's
rotations (k_bb_block, whose buckets have a fixed capacity).  Bucket capacity (the CTA's
tile of terms) and items per thread choose the variant of k_bk_rotate, which only
key-sharded runs launch (every variant is checked bit for bit against the oracle in
tests/test_gpu_shard_variants.py).  Each pair is timed on the runs that it is for.
`tune()` times each candidate on the device (CUDA events on the vector's stream) on a
representative sequence per word count and writes the choice to a JSON cache keyed by the
device's SM count and compute capability: the default, or the fastest where that is faster
than the runs of one setting differ.  `apply_cached(v)` gives a new vector the cached setting.

Cache file: paulioperators.jl_b200/tuning/sm<count>_cc<major><minor>.json
  {"sm_count": 148, "cc": [10, 0],
   "nw": {"1": {"tuning": [cap, items, load_div, chunk], "terms_per_s": ..., "workload": "..."},
          "2": {...}},
   "candidates": {"1": [[load_div, chunk, terms_per_s], ...], "2": [...]},
   "shard_candidates": {"1": [[cap, items, terms_per_s], ...], "2": [...]}}

Run on the target GPU:  python -m pauliprop.tune [--quick]
"""
import ctypes
import json
import os
import sys

import numpy as np

from . import _lib
from .circuits import lattice64

TUNING_DIR = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tuning")
VARIANTS = [(128, 4), (256, 4), (512, 4), (256, 8), (512, 8), (1024, 8)]
LOAD_DIVS = (4, 5, 6)
CHUNKS = (32, 64, 128)
DEFAULT = (512, 4, 6, 128)
MARGIN = 0.02       # a candidate replaces the default only if it is faster by more: runs of one differ by 1 %

_cache = {}


def device_info(v):
    sm, ma, mi = ctypes.c_int32(), ctypes.c_int32(), ctypes.c_int32()
    _lib.check(_lib.lib.pp_device_info(v._h, ctypes.byref(sm), ctypes.byref(ma), ctypes.byref(mi)))
    return sm.value, ma.value, mi.value


def cache_path(sm, ma, mi):
    return os.path.join(TUNING_DIR, f"sm{sm}_cc{ma}{mi}.json")


def set_tuning(v, t):
    _lib.check(_lib.lib.pp_set_tuning(v._h, ctypes.byref(_lib.PPTuning(*t))))


def get_tuning(v):
    t = _lib.PPTuning()
    _lib.check(_lib.lib.pp_get_tuning(v._h, ctypes.byref(t)))
    return (t.bucket_cap, t.items_per_thread, t.load_div, t.chunk)


def cached(sm, ma, mi, nw):
    """The cached tuning for (device, word count), or None."""
    key = (sm, ma, mi)
    if key not in _cache:
        try:
            with open(cache_path(sm, ma, mi)) as f:
                _cache[key] = json.load(f)
        except (OSError, ValueError):
            _cache[key] = None
    d = _cache[key]
    if not d:
        return None
    e = d.get("nw", {}).get(str(nw))
    return tuple(e["tuning"]) if e else None


def apply_cached(v):
    """Gives vector v the cached tuning of its device and word count (if any)."""
    t = cached(*device_info(v), v.nw)
    if t:
        set_tuning(v, t)
    return t


def _workload(nw):
    """The 8x8-lattice benchmark circuit (3,520 rotations); for two-word keys the
    same terms declared on 100 qubits."""
    w = lattice64()
    return w, (64 if nw == 1 else 100)


def _sequence(nw, layers):
    """Term arrays, generators, angles and truncation of `layers` layers of the workload."""
    from .paulis import PauliBasis, pack_keys
    from .truncation import CoeffTruncation, CompositeTruncation, WeightTruncation
    w, N = _workload(nw)
    z, x = pack_keys(N, [(o[0], o[1]) for o in w.observable])
    c = np.array([o[2] for o in w.observable], dtype=np.float64)
    gens = [PauliBasis(N, p.z, p.x) for p in w.layer] * layers
    return w, N, z, x, c, gens, list(w.angles) * layers, CompositeTruncation(CoeffTruncation(w.thresh),
                                                                              WeightTruncation(w.wmax))


class _Timer:
    """Seconds between two points of a vector's stream (the host time of a call would add its
    own overhead, comparable to the differences between candidates)."""

    def __init__(self, v):
        import torch
        self.stream = torch.cuda.ExternalStream(v.stream())
        self.e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]

    def __enter__(self):
        self.e[0].record(self.stream)
        return self

    def __exit__(self, *exc):
        self.e[1].record(self.stream)
        self.e[1].synchronize()
        self.seconds = self.e[0].elapsed_time(self.e[1]) * 1e-3


def _time_one(nw, t, reps, layers):
    """Live terms rotated per second by an unsharded vector under tuning t."""
    from . import spv
    w, N, z, x, c, gens, angs, strat = _sequence(nw, layers)
    best = 0.0
    for _ in range(reps + 1):     # the first run warms up (allocations)
        v = spv.SparsePauliVector(N, 1 << 16, 1 << 24)
        v.upload(z, x, c, sorted=False)
        set_tuning(v, t)
        st = {}
        with _Timer(v) as tm:
            spv.evolve_(v, gens, angs, truncation=strat, channel=(w.channel[0], w.channel[1], None),
                        channel_every=len(w.layer), stats=st)
        best = max(best, st["terms_in"] / tm.seconds)
        v.close()
    return best


def _time_shard(nw, t, reps, layers):
    """Live terms per second of the rotations alone of a key-sharded run under tuning t: one
    rank, so that no exchange is on its way."""
    from . import shard, spv
    w, N, z, x, c, gens, angs, strat = _sequence(nw, layers)

    class Timed(shard.GpuShard):
        seconds = 0.0

        def rotate(self, r, pref):
            with _Timer(self.v) as tm:
                out = super().rotate(r, pref)
            self.seconds += tm.seconds
            return out

    best = 0.0
    for _ in range(reps + 1):
        v = spv.SparsePauliVector(N, 1 << 16, 16)
        set_tuning(v, t)
        v.upload(z, x, c, sorted=False)
        e = Timed(v, 0, 0)
        _, st = shard.run_sharded([e], shard.LocalGroup(1), N, gens, angs, truncation=strat,
                                  channel=(w.channel[0], w.channel[1], None), channel_every=len(w.layer),
                                  append_capacity=1 << 24)
        best = max(best, st["terms_in"] / e.seconds)
        v.close()
    return best


def _choose(timed, default):
    """The fastest of [(setting, rate)], or the default where it is within MARGIN of it."""
    best = max(timed, key=lambda c: c[1])
    return next((c for c in timed if c[0] == default and c[1] * (1 + MARGIN) >= best[1]), best)


def tune(nws=(1, 2), quick=False, reps=2, layers=None, log=print):
    """Measures the candidates and writes the cache; returns its dict.  layers: of the
    workload, for unsharded and sharded runs (default: all 20, and the first 14)."""
    os.environ["PAULIPROP_WINDOW1_PATH"] = "buckets"
    from . import spv
    probe = spv.SparsePauliVector(8)
    sm, ma, mi = device_info(probe)
    probe.close()
    out = {"sm_count": sm, "cc": [ma, mi], "nw": {}, "candidates": {}, "shard_candidates": {}}
    for nw in nws:
        w, N = _workload(nw)
        full, part = layers or (w.layers, min(w.layers, 14))
        variants = []
        for cap, items in (VARIANTS if not quick else [(256, 4), (512, 4)]):
            variants.append(((cap, items), _time_shard(nw, (cap, items, DEFAULT[2], DEFAULT[3]), reps, part)))
            log(f"nw={nw} sharded {(cap, items)}: {variants[-1][1]:.4g} terms/s")
        variant = _choose(variants, DEFAULT[:2])[0]
        cands = []
        for ld in LOAD_DIVS:
            for ch in (CHUNKS if not quick else (64,)):
                cands.append(((ld, ch), _time_one(nw, (*variant, ld, ch), reps, full)))
                log(f"nw={nw} {(ld, ch)}: {cands[-1][1]:.4g} terms/s")
        best = _choose(cands, DEFAULT[2:])
        out["nw"][str(nw)] = {"tuning": [*variant, *best[0]], "terms_per_s": best[1],
                              "workload": f"{w.name} circuit on N={N} ({full} layers x {len(w.layer)} rotations)"}
        out["candidates"][str(nw)] = [[*t, r] for t, r in cands]
        out["shard_candidates"][str(nw)] = [[*t, r] for t, r in variants]
    os.makedirs(TUNING_DIR, exist_ok=True)
    with open(cache_path(sm, ma, mi), "w") as f:
        json.dump(out, f, indent=1)
    _cache.pop((sm, ma, mi), None)
    return out


if __name__ == "__main__":
    res = tune(quick="--quick" in sys.argv)
    print(json.dumps(res["nw"]))
