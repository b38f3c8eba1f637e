"""An AdaptiveTruncation sequence whose bucket overflows where a larger layout does not fit
goes on without buckets, from the rotation it reached and with that rotation's cut and
channel: the oracle's vector bit for bit.  The overflow is made: terms of one bucket, and
generators that keep their partners in it."""
import random

import numpy as np
import pytest

import orc
import pauliprop as pp
from pauliprop import _lib

pytestmark = pytest.mark.gpu

N = 40
CAP = 32                                              # slots of a bucket


def _rows():
    """The hash rows (word k of a row: z, -, x, -), from their generator's seed."""
    s, out, m = 0x5EEDB0C4E7, [], (1 << 64) - 1
    for _ in range(26 * 4):
        s = (s + 0x9E3779B97F4A7C15) & m
        z = s
        z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & m
        z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & m
        out.append(z ^ (z >> 31))
    return [(out[4 * r], out[4 * r + 2]) for r in range(26)]


ROWS = _rows()


def _hash(z, x, bits):
    return sum((((z & a).bit_count() + (x & b).bit_count()) & 1) << r for r, (a, b) in enumerate(ROWS[:bits]))


def _case(seed, bits):
    rng = random.Random(seed)
    masks = []                                        # X strings of hash 0, which commute with each other
    while len(masks) < 4:
        m = rng.getrandbits(36)
        if m and _hash(0, m, bits) == 0:
            masks.append(m)
    want, terms = rng.getrandbits(bits), {}
    while len(terms) < 16:
        z, x = rng.getrandbits(36), rng.getrandbits(36)
        if all((z & m).bit_count() & 1 for m in masks) and _hash(z, x, bits) == want:
            terms[(z, x)] = rng.uniform(0.5, 1.0) * rng.choice([-1, 1])
    idle = [(1 << q, 0) for q in (37, 38, 39)]       # commute with everything here
    more = [(rng.getrandbits(36), rng.getrandbits(36)) for _ in range(9)]
    gens = idle + [(0, m) for m in masks] + more
    return terms, gens, [rng.uniform(0.6, 0.9) for _ in gens]


def test_the_hash_rows():
    from pauliprop import shard
    rng = random.Random(1)
    ks = [(rng.getrandbits(N), rng.getrandbits(N)) for _ in range(64)]
    z, x = pp.pack_keys(N, ks)
    want = [sum((((a & ROWS[25 - k][0]).bit_count() + (b & ROWS[25 - k][1]).bit_count()) & 1) << k for k in range(4))
            for a, b in ks]
    assert list(shard.owners(1, z, x, 4)) == want


@pytest.mark.parametrize("budget", [20, 100])        # cuts before the overflow; none
@pytest.mark.parametrize("channel", [False, True])
@pytest.mark.parametrize("fits", [False, True])
def test_handover(budget, channel, fits):
    most = max(16, 2 * budget)
    bits = 1
    while (CAP << bits) < 6 * most:
        bits += 1
    terms, gens, angs = _case(budget, bits)
    keys = sorted(terms)
    v = orc.OracleSPV(N, 64, 1 << 16)
    v.upload([k[0] for k in keys], [k[1] for k in keys], [terms[k] for k in keys])
    g = pp.SparsePauliVector(N, 64, 1 << 16)
    _lib.check(_lib.lib.pp_set_tuning(g._h, _lib.ctypes.byref(_lib.PPTuning(512, 4, 6, 128))))
    g.upload(*v.arrays(), sorted=True)
    per = 4                                           # a channel behind the rotation before the overflow
    for s in range(0, len(gens), per):
        v.evolve(gens[s:s + per], angs[s:s + per], window=1, adaptive=(budget, 1e-12))
        if channel:
            v.channel(0, [0.05])
    kw = {"channel": ("depolarizing", 0.05, None), "channel_every": per} if channel else {}
    st = {}
    if not fits:
        _lib.check(_lib.lib.pp_debug_bucket_limit(CAP << bits))
    try:
        _, e = pp.evolve_(g, [pp.PauliBasis(N, a, b) for a, b in gens], angs, truncation=pp.AdaptiveTruncation(budget, 1e-12),
                          return_expectation=True, stats=st, **kw)
    finally:
        _lib.check(_lib.lib.pp_debug_bucket_limit(0))
    assert st["bucket_rot"] == len(gens) if fits else 0 < st["bucket_rot"] < 8
    gz, gx, gc = g.to_arrays()
    oz, ox, oc = v.arrays()
    assert gz.shape == oz.shape and np.array_equal(gz, oz) and np.array_equal(gx, ox), "key sets differ"
    assert np.array_equal(gc.view(np.uint64), oc.view(np.uint64)), "coefficients differ"
    diag = np.all(ox == 0, axis=1)
    assert abs(e - v.expect(0)) <= 1e-12 * max(1e-300, float(np.abs(oc[diag]).sum()))
    g.close()
