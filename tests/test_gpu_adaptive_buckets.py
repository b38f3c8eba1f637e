"""AdaptiveTruncation sequences at window 1 (on buckets once the append capacity rules
out early merges) against the CPU oracle, bit for bit: budgets from one term up, sets
below and above the budget, ties at the cut, a minimum threshold that cuts, channels
between layers, and a small capacity (early merges first)."""
import random

import numpy as np
import pytest

import orc
import pauliprop as pp
from helpers import rand_terms

pytestmark = pytest.mark.gpu


def _pair(N, terms, append):
    v = orc.OracleSPV(N, max(16, 2 * len(terms)), append)
    keys = sorted(terms)
    v.upload([k[0] for k in keys], [k[1] for k in keys], [terms[k] for k in keys])
    z, x, c = v.arrays()
    g = pp.SparsePauliVector(N, max(16, 2 * len(c)), append)
    g.upload(z, x, c, sorted=True)
    return g, v


@pytest.mark.parametrize("N,n,budget,min_thresh,append", [
    (12, 1, 1, 1e-12, 1 << 16), (20, 3, 300, 1e-12, 1 << 16), (20, 3, 300, 1e-12, 16), (40, 4000, 1500, 1e-12, 1 << 16),
    (64, 3000, 20000, 3e-2, 1 << 16), (70, 500, 2111, 1e-12, 1 << 16), (128, 6000, 5000, 1e-12, 1 << 16),
])
@pytest.mark.parametrize("channel", [False, True])
def test_adaptive_sequence(N, n, budget, min_thresh, append, channel):
    rng = random.Random(N * 7 + n)
    terms = {(1 << i, 0): 1.0 - 0.25 * (i % 2) for i in range(n)} if n < 10 else rand_terms(rng, N, n)
    if n >= 10:
        for i, k in enumerate(list(terms)[: n // 4]):    # many equal magnitudes
            terms[k] = (1 if i % 2 else -1) * 0.125 * (1 + i % 4)
    gens, angs = [], []
    for _ in range(48):
        i, j = rng.sample(range(min(N, 12)), 2)
        kind = rng.randrange(3)
        gens.append(((1 << i) | (1 << j), 0) if kind == 0 else (0, 1 << i) if kind == 1 else ((1 << i) | (1 << j),) * 2)
        angs.append(rng.choice([0.3, 0.5, -0.7, rng.uniform(-1, 1)]))
    per = 16
    g, v = _pair(N, terms, append)
    for s in range(0, len(gens), per):
        v.evolve(gens[s:s + per], angs[s:s + per], window=1, adaptive=(budget, min_thresh))
        if channel:
            v.channel(0, [0.05])
    kw = {"channel": ("depolarizing", 0.05, None), "channel_every": per} if channel else {}
    st = {}
    _, e = pp.evolve_(g, [pp.PauliBasis(N, a, b) for a, b in gens], angs, truncation=pp.AdaptiveTruncation(budget, min_thresh),
                      return_expectation=True, stats=st, **kw)
    assert (st["bucket_rot"] == 48) == (append > budget) and st["bucket_rot"] > 0
    gz, gx, gc = g.to_arrays()
    oz, ox, oc = v.arrays()
    assert gz.shape == oz.shape and np.array_equal(gz, oz) and np.array_equal(gx, ox), "key sets differ"
    assert np.array_equal(gc.view(np.uint64), oc.view(np.uint64)), "coefficients differ"
    diag = np.all(ox == 0, axis=1)
    assert abs(e - v.expect(0)) <= 1e-12 * max(1e-300, float(np.abs(oc[diag]).sum()))
