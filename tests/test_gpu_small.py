"""The single-CTA rotations (k_small_run) against the CPU oracle, bit for bit: one term,
a thread per slot and more slots than threads, the largest set it takes and one that
outgrows it, enough births and deaths for its slots to run out, channels, and the early
merge with WindowCounters."""
import random

import numpy as np
import pytest

import orc
import pauliprop as pp
from helpers import CHANNEL_KIND, filt, rand_terms, strategy

pytestmark = pytest.mark.gpu


def _run(N, n, L, per, thresh, small_capacity):
    rng = random.Random(1000 * N + n)
    terms = rand_terms(rng, N, n)
    kw = {"append_factor": 0.01, "min_capacity": 4} if small_capacity else {}
    v = orc.OracleSPV.from_terms(N, [(k[0], k[1], c) for k, c in terms.items()], **kw)
    z, x, c = v.arrays()
    g = pp.SparsePauliVector(N, max(16, 2 * len(c)), v.append_cap)
    g.upload(z, x, c, sorted=True)
    gens, angs = [], []
    for _ in range(L):
        i, j = rng.sample(range(min(N, 10)), 2)
        gens.append(((1 << i) | (1 << j), 0) if rng.random() < 0.6 else (0, 1 << i))
        angs.append(rng.uniform(-1.5, 1.5))
    spec = ("comp", [("coeff", thresh), ("weight", 3 * N // 4 + 3)])
    early = 0
    wc = pp.WindowCounters(L)
    ctrs = []
    for s in range(0, L, per):
        _, ctr = v.evolve(gens[s:s + per], angs[s:s + per], window=1, strict=filt(spec), nwin=per)
        ctrs.append(ctr)
        early += int(ctr[3].sum())
        v.channel(CHANNEL_KIND["dephasing"], [0.01])
    _, e = pp.evolve_(g, [pp.PauliBasis(N, a, b) for a, b in gens], angs, truncation=strategy(spec), counters=wc,
                      channel=("dephasing", 0.01, None), channel_every=per, return_expectation=True)
    gz, gx, gc = g.to_arrays()
    oz, ox, oc = v.arrays()
    assert gz.shape == oz.shape and np.array_equal(gz, oz) and np.array_equal(gx, ox), "key sets differ"
    assert np.array_equal(gc.view(np.uint64), oc.view(np.uint64)), "coefficients not bit-identical"
    for got, k in ((wc.terms_created, 0), (wc.merge_in, 1), (wc.merge_out, 2), (wc.early_merges, 3)):
        assert np.array_equal(got, np.concatenate([c[k] for c in ctrs]))
    diag = np.all(ox == 0, axis=1)
    assert abs(e - v.expect(0)) <= 1e-12 * max(1e-300, float(np.abs(oc[diag]).sum()))
    return early


@pytest.mark.parametrize("N,n", [(20, 1), (20, 500), (20, 513), (64, 2047), (64, 2048), (70, 1), (70, 511), (70, 1023),
                                 (128, 1024)])
def test_small_sizes(N, n):
    _run(N, n, 24, 8, 5e-2, False)


@pytest.mark.parametrize("N,n,thresh", [(20, 300, 0.25), (90, 200, 0.3)])
def test_small_slots_run_out(N, n, thresh):
    _run(N, n, 240, 24, thresh, False)


@pytest.mark.parametrize("N,n,per", [(20, 400, 6), (90, 300, 1)])
def test_small_early_merge(N, n, per):
    assert _run(N, n, 36, per, 1e-1, True) > 0
