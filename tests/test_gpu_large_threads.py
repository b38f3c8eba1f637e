"""Copies evolved and closed on several threads whose buffers are large blocks (64 MiB and
more): a block passes from one handle's stream to another's only when its work has ended."""
import threading

import numpy as np
import pytest

import pauliprop as pp
from pauliprop import circuits

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [64, 100])
def test_large_copies_on_threads(N):
    rng = np.random.default_rng(N)
    n, nw = 700_000, pp.nwords(N)
    z = np.zeros((n, nw), dtype=np.uint64)
    z[:, 0] = np.sort(rng.choice(1 << 40, n, replace=False).astype(np.uint64))
    x = np.zeros((n, nw), dtype=np.uint64)
    x[:, 0] = rng.integers(0, 1 << 40, n, dtype=np.uint64)
    if nw == 2:
        z[:, 1] = np.arange(n) * 5 // n                # the high word orders the keys
    v = pp.SparsePauliVector(N, n, 16)
    v.upload(z, x, rng.uniform(-1, 1, n), sorted=True)
    gens = [circuits.xq(N, q) if q % 2 else circuits.zz(N, q, q + 1) for q in range(1, 29)]
    trunc = pp.CoeffTruncation(0.05)
    lengths = (9, 10, 24)

    def run(L):
        w = pp.evolve(v, gens[:L], [0.2] * L, truncation=trunc)
        out = w.to_arrays()
        w.close()
        return out

    want = {L: run(L) for L in lengths}
    bad = []

    def work(k):
        for i in range(6):
            L = lengths[(k + i) % len(lengths)]
            if not all(np.array_equal(a, b) for a, b in zip(run(L), want[L])):
                bad.append((k, i))

    ts = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad
    v.close()
