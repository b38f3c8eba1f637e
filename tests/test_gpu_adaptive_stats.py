"""A profiled AdaptiveTruncation sequence on buckets reports the bytes and the time of its
rotations, so that a rate can be computed from them."""
import numpy as np
import pytest

import pauliprop as pp
from pauliprop import circuits

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [30, 90])
def test_profiled_adaptive_sequence(N):
    gens, angs = circuits.trotterize(circuits.heisenberg_chain_terms(N), 0.2, 2, order=1)
    out = {}
    for profile in (False, True):
        v = pp.SparsePauliVector(N, 1 << 12, 1 << 16)
        z, x = pp.pack_keys(N, [(1 << (N // 2), 0)])
        v.upload(z, x, np.array([1.0]), sorted=True)
        st = {}
        pp.evolve_(v, gens, angs, truncation=pp.AdaptiveTruncation(200, 1e-12), stats=st, profile=profile)
        assert st["bucket_rot"] == len(gens)
        out[profile] = st
        v.close()
    a, b = out[False], out[True]
    # what enters and leaves each rotation: the sets before the cuts
    per_term = 24 if N <= 64 else 40
    assert a["bucket_bytes"] == b["bucket_bytes"]
    assert per_term * len(gens) <= b["bucket_bytes"] <= 2 * per_term * len(gens) * b["peak"]
    assert b["t_merge"] > 0 and a["t_merge"] == 0
    assert 1e6 < b["bucket_bytes"] / b["t_merge"] < 1e13
