"""EnergyCorrection on buckets adds up what is dropped exactly, whatever its size: values far
below the set's norm, sets whose squares underflow, subnormal values, and values above the
entering norm (which a local truncation can grow).  The generators commute with every term
unless stated, so that the exact sum is the input's."""
import math

import numpy as np
import pytest

import orc
import pauliprop as pp
from helpers import filt, strategy

pytestmark = pytest.mark.gpu

N = 40
KET = 0b1011


def _run(z, x, c, spec, gens=None, angs=None, local=None):
    o = np.lexsort([x, z])
    z, x, c = z[o], x[o], c[o]
    g = pp.SparsePauliVector(N, max(16, 2 * len(c)), 1 << 20)
    g.upload(z.reshape(-1, 1), x.reshape(-1, 1), c, sorted=True)
    gens = gens or [(1 << k, 0) for k in range(8)]
    angs = angs or [0.3] * len(gens)
    corr = pp.EnergyCorrection(KET)
    st = {}
    pp.evolve_(g, [pp.PauliBasis(N, a, b) for a, b in gens], angs, truncation=strategy(spec), correction=corr,
               local_truncation=strategy(local) if local else None, stats=st)
    assert st["bucket_rot"] == len(gens)
    return g, corr.accumulated_energy


def _signs(z):
    return np.where(np.bitwise_count(z & np.uint64(KET)) & 1, -1.0, 1.0)


@pytest.mark.parametrize("scale", [1e-25, 1e-33, 1e-45, 1e-80, 1e-170, 5e-310])
@pytest.mark.parametrize("kept", [0, 3])              # terms of size one that set the norm
@pytest.mark.parametrize("mixed", [False, True])
def test_sum_of_small_values(scale, kept, mixed):
    rng = np.random.default_rng(int(-math.log10(scale)) + 1000 * kept)
    n = 3000
    z = rng.choice(1 << 30, n, replace=False).astype(np.uint64)
    x = np.zeros(n, dtype=np.uint64)
    c = scale * rng.uniform(0.1, 1.0, n)
    if mixed:
        c *= rng.choice([-1.0, 1.0], n) * 10.0 ** rng.uniform(-12, 0, n)
    else:
        c *= _signs(z)                                # every contribution of one sign
    if kept:
        z = np.concatenate([z, (np.uint64(1) << np.uint64(33)) + np.arange(kept, dtype=np.uint64)])
        x = np.concatenate([x, np.zeros(kept, dtype=np.uint64)])
        c = np.concatenate([c, np.ones(kept)])
    g, e = _run(z, x, c, ("coeff", 2 * scale))
    assert len(g) == kept
    v = (c * _signs(z))[:n]
    # the sum is exact up to a few roundings: of its terms' size where they cancel
    want, size = math.fsum(v), math.fsum(np.abs(v)) if mixed else abs(math.fsum(v))
    assert abs(abs(e) - abs(want)) <= 8 * np.finfo(float).eps * size + 16 * 5e-324


def test_values_above_the_entering_norm():
    """A local truncation that drops one of two partners' sin branches: the set grows, and what
    a weight cap drops at the end is larger than what entered."""
    steps = 24
    # X on qubit 0 and 1 .. in turn: pairs (P, P xor M) with one branch too small for the local filter
    z = np.array([1 << 20, (1 << 20) | 1], dtype=np.uint64)
    x = np.zeros(2, dtype=np.uint64)
    c = np.array([1.0, 1e-3])
    gens = [(1 << k, 1 << 20) for k in range(steps)]
    angs = [0.7] * steps
    v = orc.OracleSPV.from_terms(N, [(int(a), int(b), float(d)) for a, b, d in zip(z, x, c)], append_factor=1e6)
    e, _ = v.evolve(gens, angs, window=1, strict=filt(("coeff", 0.05)), energy_ket=KET, local=filt(("coeff", 0.1)))
    g, got = _run(z, x, c, ("coeff", 0.05), gens, angs, ("coeff", 0.1))
    oz, ox, oc = v.arrays()
    gz, gx, gc = g.to_arrays()
    assert np.array_equal(gz, oz) and np.array_equal(gc.view(np.uint64), oc.view(np.uint64))
    assert abs(got - e) <= 4 * steps * np.finfo(float).eps * 2


def test_largest_and_smallest_together():
    # 1e150 is kept (its square is finite), everything below is dropped: exact over 460 decades
    z = np.arange(1, 5001, dtype=np.uint64) << np.uint64(10)
    x = np.zeros(5000, dtype=np.uint64)
    c = 10.0 ** np.linspace(-310, 149, 5000) * _signs(z)
    c[-1] = 1e151
    g, e = _run(z, x, c, ("coeff", 1e150))
    assert len(g) == 1
    want = math.fsum((c * _signs(z))[:-1])
    assert abs(abs(e) - want) <= 8 * np.finfo(float).eps * want
