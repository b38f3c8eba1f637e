"""The tuner times the one-rotation kernel's variants on key-sharded runs, which launch it."""
import pytest

from pauliprop import shard, tune

pytestmark = pytest.mark.gpu


def test_tuner_times_the_variants_on_sharded_runs(monkeypatch, tmp_path):
    monkeypatch.setenv("PAULIPROP_WINDOW1_PATH", "buckets")       # (tune sets it)
    monkeypatch.setattr(tune, "TUNING_DIR", str(tmp_path))
    monkeypatch.setattr(tune, "LOAD_DIVS", (6,))
    monkeypatch.setattr(tune, "CHUNKS", (128,))
    seen = []
    begin = shard.GpuShard.begin
    monkeypatch.setattr(shard.GpuShard, "begin", lambda self, *a: seen.append(self.tuning()[:2]) or begin(self, *a))
    out = tune.tune(nws=(1,), reps=1, layers=(2, 2), log=lambda *_: None)
    tune._cache.clear()
    assert set(seen) == set(tune.VARIANTS)
    e = out["nw"]["1"]
    timed = {(c[0], c[1]): c[2] for c in out["shard_candidates"]["1"]}
    assert set(timed) == set(tune.VARIANTS) and all(r > 0 for r in timed.values())
    assert timed[tuple(e["tuning"][:2])] * (1 + tune.MARGIN) >= max(timed.values())
