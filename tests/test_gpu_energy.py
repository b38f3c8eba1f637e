"""EnergyCorrection on buckets against the CPU oracle: the vector bit for bit, the
accumulated energy within the rounding of the oracle's own sum, from the shortest
sequences that take buckets, with early merges, a channel, local truncation, and
coefficients far from one."""
import random

import numpy as np
import pytest

import orc
import pauliprop as pp
from helpers import CHANNEL_KIND, filt, rand_terms, strategy

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,n,L,early,scale", [
    (20, 40, 6, False, 1.0), (30, 5000, 7, False, 1.0), (64, 5000, 40, True, 1e-9), (90, 3000, 24, False, 1e12),
    (128, 1500, 36, True, 1.0),
])
@pytest.mark.parametrize("local", [False, True])
def test_energy_on_buckets(N, n, L, early, scale, local):
    rng = random.Random(N + n + L)
    terms = {k: scale * c for k, c in rand_terms(rng, N, n).items()}
    for i, k in enumerate(list(terms)):
        if i % 3 == 0:                                # diagonal terms, which the energy sees
            terms[(k[0] ^ (i + 1), 0)] = terms.pop(k)
    for i, k in enumerate(list(terms)[: n // 5]):     # below the threshold before any rotation
        terms[k] = scale * 1e-3 * (rng.random() - 0.5)
    kw = {"append_factor": 0.02, "min_capacity": 4} if early else {}
    v = orc.OracleSPV.from_terms(N, [(k[0], k[1], c) for k, c in terms.items()], **kw)
    z, x, c = v.arrays()
    g = pp.SparsePauliVector(N, max(16, 2 * len(c)), v.append_cap)
    g.upload(z, x, c, sorted=True)
    gens, angs = [], []
    for _ in range(L):
        i, j = rng.sample(range(min(N, 14)), 2)
        gens.append(((1 << i) | (1 << j), 0) if rng.random() < 0.6 else (0, 1 << i))
        angs.append(rng.uniform(-1.2, 1.2))
    spec = ("comp", [("coeff", scale * 3e-2), ("weight", max(3, N // 2))])
    lspec = ("coeff", scale * 4e-2) if local else None
    ket = 0b1001101
    lkw = {"local": filt(lspec)} if local else {}
    e, _ = v.evolve(gens, angs, window=1, strict=filt(spec), energy_ket=ket, **lkw)
    corr = pp.EnergyCorrection(ket)
    st = {}
    pp.evolve_(g, [pp.PauliBasis(N, a, b) for a, b in gens], angs, truncation=strategy(spec), correction=corr,
               local_truncation=strategy(lspec) if local else None, stats=st)
    assert st["bucket_rot"] == L
    gz, gx, gc = g.to_arrays()
    oz, ox, oc = v.arrays()
    assert gz.shape == oz.shape and np.array_equal(gz, oz) and np.array_equal(gx, ox), "key sets differ"
    assert np.array_equal(gc.view(np.uint64), oc.view(np.uint64)), "coefficients not bit-identical"
    # the oracle takes differences of <ket|O|ket>, each rounded to the size of the set's diagonal
    tol = 4 * L * np.finfo(float).eps * float(np.abs(c[np.all(x == 0, axis=1)]).sum())
    assert abs(corr.accumulated_energy - e) <= tol


def test_energy_of_many_equal_terms():
    # 2^25 equal diagonal terms, all dropped by one rotation: the parts of the exact sum
    # grow with the number of terms; their rest below the first unit is nearly half of it
    n, N = 1 << 25, 30
    c = (87654 + 0.4999) * 2.0 ** -30
    z = np.arange(n, dtype=np.uint64).reshape(-1, 1)
    g = pp.SparsePauliVector(N, n, 16)
    g.upload(z, np.zeros_like(z), np.full(n, c), sorted=True)
    # <ket|Z-string|ket> = (-1)^popcount(z & ket): with ket 0 every term counts as +c
    corr = pp.EnergyCorrection(0)
    pp.evolve_(g, [pp.PauliBasis(N, 1 << i, 0) for i in range(8)], [0.3] * 8, truncation=pp.CoeffTruncation(1.0),
               correction=corr)
    assert len(g) == 0
    assert abs(abs(corr.accumulated_energy) - n * c) <= 4 * np.finfo(float).eps * n * c
    g.close()

