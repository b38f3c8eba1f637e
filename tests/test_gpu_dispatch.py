"""Which window-1 sequences run on buckets: short ones where the conversion pays, the longer
the larger the set, and later on a vector whose live sets have room for the sorted merges
than on a copy.  Either way gives the same vector (test_gpu_buckets.py)."""
import random

import numpy as np
import pytest

import pauliprop as pp
from pauliprop import circuits

pytestmark = pytest.mark.gpu

N = 64


def _vector(n, room):
    rng = np.random.default_rng(n)
    z = np.sort(rng.choice(1 << 40, n, replace=False).astype(np.uint64)).reshape(-1, 1)
    v = pp.SparsePauliVector(N, 4 * n + 8192 if room else n, 16)
    v.upload(z, rng.integers(0, 1 << 40, (n, 1), dtype=np.uint64), rng.uniform(-1, 1, n), sorted=True)
    return v


def _gens(L):
    return [circuits.xq(N, 1 + k % 40) if k % 2 else circuits.zz(N, 1 + k % 39, 2 + k % 39) for k in range(L)]


@pytest.mark.parametrize("n,rotations,room,buckets", [
    (200_000, 5, True, False), (200_000, 6, True, True), (200_000, 5, False, False), (200_000, 6, False, True),
    (600_000, 9, True, False), (600_000, 10, True, True), (600_000, 7, False, False), (600_000, 8, False, True),
    (1_500_000, 23, True, False), (1_500_000, 24, True, True), (1_500_000, 23, False, False),
    (3_200_000, 31, True, False), (3_200_000, 32, True, True),
])
def test_line(n, rotations, room, buckets):
    v = _vector(n, room)
    st = {}
    pp.evolve_(v, _gens(rotations), [0.01] * rotations, truncation=pp.CoeffTruncation(0.05), stats=st)
    assert st["bucket_rot"] == (rotations if buckets else 0)
    pp.check_spv(v)
    v.close()


def test_line_of_a_batch_span():
    rng = random.Random(3)
    obs = [[(rng.getrandbits(30), rng.getrandbits(30), 1.0) for _ in range(6200)] for _ in range(50)]
    obs = [[(z, x, c) for (z, x), c in {(t[0], t[1]): t[2] for t in o}.items()] for o in obs]
    gens = [(0, 1 << k) for k in range(16)]
    for rotations, buckets in ((9, False), (10, True)):
        r = pp.evolve_batch(obs, gens[:rotations], [0] * rotations, [[0.01]] * 50, [rotations] * 50, nq=30,
                            truncation=pp.CoeffTruncation(0.05))
        assert r.stats["bucket_rot"] == (rotations if buckets else 0)
        assert r.n_final.sum() > 300_000
