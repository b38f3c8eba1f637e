"""The tuner's choice, on the host with made-up timings: bucket capacity and items per thread
are timed on key-sharded runs, the load divisor and the chunk on unsharded ones, and equal
candidates (to the noise of a run) leave the default."""
import random

import pytest

from pauliprop import spv, tune


@pytest.fixture
def fake(monkeypatch, tmp_path):
    class Vector:
        def __init__(self, *a):
            pass

        def close(self):
            pass

    monkeypatch.setattr(spv, "SparsePauliVector", Vector)
    monkeypatch.setattr(tune, "device_info", lambda v: (148, 10, 0))
    monkeypatch.setattr(tune, "TUNING_DIR", str(tmp_path))
    monkeypatch.setenv("PAULIPROP_WINDOW1_PATH", "buckets")
    rng = random.Random(1)
    rates = {"shard": {}, "one": {}}
    monkeypatch.setattr(tune, "_time_shard",
                        lambda nw, t, *a: rates["shard"].get(t[:2], 1.0) * rng.uniform(0.995, 1.005), raising=False)
    monkeypatch.setattr(tune, "_time_one",
                        lambda nw, t, *a: rates["one"].get(t[2:], 1.0) * rng.uniform(0.995, 1.005))
    yield rates
    tune._cache.clear()


def test_equal_candidates_leave_the_default(fake):
    for _ in range(10):
        out = tune.tune(log=lambda *_: None)
        assert all(out["nw"][k]["tuning"] == list(tune.DEFAULT) for k in ("1", "2"))


def test_each_pair_follows_its_own_runs(fake):
    fake["shard"][(256, 8)] = 1.1
    fake["one"][(5, 32)] = 1.1
    out = tune.tune(nws=(2,), log=lambda *_: None)
    assert out["nw"]["2"]["tuning"] == [256, 8, 5, 32]
    assert tune.cached(148, 10, 0, 2) == (256, 8, 5, 32)
