"""Every compiled (bucket capacity, items per thread) variant of the one-rotation kernel, which
key-sharded runs launch: the union of two ranks' shards is the oracle's vector bit for bit,
with early merges and splits of the layout on the way."""
import random

import numpy as np
import pytest

import orc
import pauliprop as pp
from helpers import filt, rand_terms, strategy
from pauliprop import shard, tune

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant", tune.VARIANTS, ids=str)
@pytest.mark.parametrize("N", [64, 90])
def test_shard_every_variant(variant, N):
    rng = random.Random(sum(variant) + N)
    terms = rand_terms(rng, N, 5000)
    gens, angs = [], []
    for _ in range(28):
        i, j = rng.sample(range(min(N, 14)), 2)
        gens.append(((1 << i) | (1 << j), 0) if rng.random() < 0.6 else (0, 1 << i))
        angs.append(rng.uniform(0.2, 1.2))
    spec = ("coeff", 1e-2)
    v = orc.OracleSPV.from_terms(N, [(k[0], k[1], c) for k, c in terms.items()], append_factor=0.05, min_capacity=4)
    keys = list(terms)
    z, x = pp.pack_keys(N, keys)
    c = np.array([terms[k] for k in keys])
    engines = []
    for r, (pz, px, pc) in enumerate(shard.split(pp.nwords(N), z, x, c, 1)):
        g = pp.SparsePauliVector(N, max(16, 2 * len(pc)), 16)
        tune.set_tuning(g, (*variant, 3, 8))
        g.upload(pz, px, pc, sorted=False)
        engines.append(shard.GpuShard(g, 1, r))
    _, st = shard.run_sharded(engines, shard.LocalGroup(2), N, [pp.PauliBasis(N, a, b) for a, b in gens], angs,
                              truncation=strategy(spec), append_capacity=v.append_cap, load_div=3)
    _, ctr = v.evolve(gens, angs, window=1, strict=filt(spec), nwin=len(gens))
    assert ctr[3].sum() > 0 and st["created"] == ctr[0].sum()
    parts = [e.v.to_arrays() for e in engines]
    nw = pp.nwords(N)
    gz, gx = (np.concatenate([p[k] for p in parts]).reshape(-1, nw) for k in (0, 1))
    gc = np.concatenate([p[2] for p in parts])
    o = np.lexsort(tuple(gx[:, k] for k in range(nw)) + tuple(gz[:, k] for k in range(nw)))
    oz, ox, oc = v.arrays()
    assert gz.shape == oz.shape and np.array_equal(gz[o], oz) and np.array_equal(gx[o], ox), "key sets differ"
    assert np.array_equal(gc[o].view(np.uint64), oc.view(np.uint64)), "coefficients not bit-identical"
    for e in engines:
        e.v.close()
