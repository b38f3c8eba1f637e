"""Pooled device memory of the handles: copies evolved and closed on several threads at
once give what one thread gives (buffers pass between the handles' streams), and what
the pool keeps of a large vector's memory after it is closed is bounded."""
import gc
import random
import threading

import numpy as np
import pytest

import pauliprop as pp
from helpers import rand_terms

pytestmark = pytest.mark.gpu


def test_copies_on_threads():
    rng = random.Random(4)
    N = 40
    ps = pp.PauliSum(N)
    for k, c in rand_terms(rng, N, 3000).items():
        ps[k] = c
    v = pp.SparsePauliVector.from_paulisum(ps)
    G = [pp.PauliBasis(N, 0, 1 << i) if i % 3 else pp.PauliBasis(N, 3 << i, 0) for i in range(20)]
    angs = [0.1 + 0.02 * i for i in range(20)]
    trunc = pp.CoeffTruncation(1e-3)
    want = [pp.evolve(v, G[k:], angs[k:], truncation=trunc).to_arrays() for k in range(4)]
    bad = []

    def work(k):
        for _ in range(12):
            got = pp.evolve(v, G[k:], angs[k:], truncation=trunc).to_arrays()
            if not all(np.array_equal(a, b) for a, b in zip(got, want[k])):
                bad.append(k)

    ts = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad


def test_memory_given_back():
    import torch
    keepalive = pp.SparsePauliVector(8)      # another handle: the pool is not emptied
    gc.collect()
    before = torch.cuda.mem_get_info()[0]
    v = pp.SparsePauliVector(64, 240_000_000, 16)     # about 14 GiB
    assert torch.cuda.mem_get_info()[0] < before - (10 << 30)
    v.close()
    assert torch.cuda.mem_get_info()[0] > before - (8 << 30) - (64 << 20)
    keepalive.close()
