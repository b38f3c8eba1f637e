"""Blocks of rotations on cosets of buckets (k_bb_block) against the CPU oracle, bit
for bit, where its dispatch changes: the smallest sets it takes, blocks whose deltas
are dependent (a coset of fewer dimensions, or of none), generators that leave every
term alone, a channel inside a layer, growth beyond a coset's room, and the early
merge entering a block."""
import random

import numpy as np
import pytest

import orc
import pauliprop as pp
from helpers import CHANNEL_KIND, filt, rand_terms, strategy

pytestmark = pytest.mark.gpu


def _vectors(N, terms, **kw):
    v = orc.OracleSPV.from_terms(N, [(k[0], k[1], c) for k, c in terms.items()], **kw)
    z, x, c = v.arrays()
    g = pp.SparsePauliVector(N, max(16, 2 * len(c)), v.append_cap)
    g.upload(z, x, c, sorted=True)
    return v, g


def _same(g, v):
    gz, gx, gc = g.to_arrays()
    oz, ox, oc = v.arrays()
    assert gz.shape == oz.shape and np.array_equal(gz, oz) and np.array_equal(gx, ox), "key sets differ"
    assert np.array_equal(gc.view(np.uint64), oc.view(np.uint64)), "coefficients not bit-identical"


def _local(rng, N, L):
    out = []
    for _ in range(L):
        i, j = rng.sample(range(N), 2)
        out.append(((1 << i) | (1 << j), 0) if rng.random() < 0.6 else (0, 1 << i))
    return out


@pytest.mark.parametrize("N,n,kind", [
    (24, 2049, "local"), (24, 2500, "repeated"), (70, 1025, "local"), (70, 1100, "identity"),
    (64, 9000, "local"), (100, 9000, "repeated"), (40, 30011, "dense"), (128, 4097, "local"),
])
def test_block_edges(N, n, kind):
    rng = random.Random(31 * N + n)
    terms = rand_terms(rng, N, n)
    if kind == "repeated":            # dependent deltas: a block of many rotations spans few dimensions
        base = _local(rng, N, 3)
        gens = [base[i % 3] for i in range(40)]
    elif kind == "identity":          # nothing anticommutes with the identity; its delta is zero
        gens = [(0, 0) if i % 3 else g for i, g in enumerate(_local(rng, N, 36))]
    elif kind == "dense":             # half of the terms anticommute: cosets outgrow their room
        m = (1 << N) - 1
        gens = [(rng.getrandbits(N) & m, rng.getrandbits(N) & m) for _ in range(33)]
    else:
        gens = _local(rng, N, 50)
    angs = [rng.uniform(0.03, 0.08) if kind == "dense" else rng.uniform(-1.0, 1.0) for _ in gens]
    spec = ("comp", [("coeff", 2e-2), ("weight", 3 * N // 4 + 2)])
    v, g = _vectors(N, terms)
    v.evolve(gens, angs, window=1, strict=filt(spec))
    pp.evolve_(g, [pp.PauliBasis(N, a, b) for a, b in gens], angs, truncation=strategy(spec))
    _same(g, v)


@pytest.mark.parametrize("N,per", [(30, 1), (30, 6), (90, 33)])
def test_block_channel_and_early_merge(N, per):
    """A channel after every `per` rotations (blocks end there, and the next one filters
    every term), with an append capacity small enough that every rotation starts with
    the early merge; WindowCounters against the oracle's."""
    rng = random.Random(N + per)
    terms = rand_terms(rng, N, 6000)
    for k in list(terms)[:1500]:
        terms[k] = 1e-3 * (rng.random() - 0.5)
    gens = _local(rng, N, 66)
    angs = [rng.uniform(-1.0, 1.0) for _ in gens]
    spec = ("comp", [("coeff", 1e-2), ("weight", 3 * N // 4 + 4)])
    v, g = _vectors(N, terms, append_factor=0.05, min_capacity=4)
    for s in range(0, len(gens), per):
        v.evolve(gens[s:s + per], angs[s:s + per], window=1, strict=filt(spec))
        v.channel(CHANNEL_KIND["depolarizing"], [0.02])
    st = {}
    pp.evolve_(g, [pp.PauliBasis(N, a, b) for a, b in gens], angs, truncation=strategy(spec),
               channel=("depolarizing", 0.02, None), channel_every=per, stats=st)
    assert st["bucket_rot"] > 0 and st["early"] > 0
    _same(g, v)
