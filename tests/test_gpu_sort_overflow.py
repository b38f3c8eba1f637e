"""A sample sort that finds a bucket beyond its slots sorts by digits: the same result
where sets of every origin are sorted, and, where an allocation of the call fails on the
way, the vector that entered it."""
import os
import random

import numpy as np
import pytest

import pauliprop as pp
from helpers import rand_terms
from pauliprop import _lib

pytestmark = pytest.mark.gpu


@pytest.fixture
def overflow():
    _lib.check(_lib.lib.pp_debug_sort_overflow(1))
    old = os.environ.get("PAULIPROP_WINDOW1_PATH")
    os.environ["PAULIPROP_WINDOW1_PATH"] = "buckets"
    yield
    _lib.check(_lib.lib.pp_debug_sort_overflow(0))
    if old is None:
        del os.environ["PAULIPROP_WINDOW1_PATH"]
    else:
        os.environ["PAULIPROP_WINDOW1_PATH"] = old


def _case(N):
    rng = random.Random(N)
    terms = rand_terms(rng, N, 5000)
    keys = sorted(terms)
    z, x = pp.pack_keys(N, keys)
    gens, angs = [], []
    for _ in range(24):
        i, j = rng.sample(range(12), 2)
        gens.append(pp.PauliBasis(N, (1 << i) | (1 << j), 0) if rng.random() < 0.6 else pp.PauliBasis(N, 0, 1 << i))
        angs.append(rng.uniform(0.2, 1.2))
    return (z, x, np.array([terms[k] for k in keys])), gens, angs


def _vector(N, obs):
    g = pp.SparsePauliVector(N, 5000, 5000)
    g.upload(*obs, sorted=True)
    return g


def _same(a, b):
    return all(p.shape == q.shape and np.array_equal(p.view(np.uint64), q.view(np.uint64)) for p, q in zip(a, b))


@pytest.mark.parametrize("N", [64, 100])
def test_digits_give_the_same_vector(N, overflow):
    obs, gens, angs = _case(N)
    _lib.check(_lib.lib.pp_debug_sort_overflow(0))
    g = _vector(N, obs)
    pp.evolve_(g, gens, angs, truncation=pp.CoeffTruncation(1e-2))
    want = g.to_arrays()
    assert len(want[2]) > 4096                       # more than one bucket
    _lib.check(_lib.lib.pp_debug_sort_overflow(1))
    g = _vector(N, obs)
    pp.evolve_(g, gens, angs, truncation=pp.CoeffTruncation(1e-2))
    assert _same(g.to_arrays(), want)
    o = np.random.default_rng(N).permutation(len(want[2]))
    g.upload(*(np.ascontiguousarray(a[o]) for a in want), sorted=False)
    assert _same(g.to_arrays(), want)
    g.close()


@pytest.mark.parametrize("N", [64, 100])
def test_failed_allocation_keeps_the_entering_vector(N, overflow):
    obs, gens, angs = _case(N)
    failed = passed = after = 0
    while passed < 8:                                # (up to five in a row only cost the sample sort)
        after += 1
        g = _vector(N, obs)
        _lib.check(_lib.lib.pp_debug_fail_alloc(after))
        try:
            pp.evolve_(g, gens, angs, truncation=pp.CoeffTruncation(1e-2))
            passed += 1
        except MemoryError:
            failed, passed = failed + 1, 0
            assert _same(g.to_arrays(), obs), after
        finally:
            _lib.check(_lib.lib.pp_debug_fail_alloc(0))
            g.close()
    assert failed > 10
