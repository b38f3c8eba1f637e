"""The sample sort against numpy's lexsort, where its plan changes: one bucket (one
CTA), the first size of several, a thousand buckets, and the larger buckets and fewer
samples above; spread keys, keys that differ in their last word only, and few distinct
ones per sample.  Keys and coefficients come back bit for bit."""
import numpy as np
import pytest

import pauliprop as pp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [40, 100])
@pytest.mark.parametrize("n", [1, 2, 33, 1024, 1025, 4096, 4097, 50021, 614401, 1400003, 2200001])
@pytest.mark.parametrize("keys", ["spread", "low", "clustered"])
def test_sort_of_an_upload(N, n, keys):
    rng = np.random.default_rng([N, n])
    nw = 1 if N <= 64 else 2
    z = np.zeros((n, nw), dtype=np.uint64)
    x = np.zeros((n, nw), dtype=np.uint64)
    ids = rng.permutation(n).astype(np.uint64)
    if keys == "spread":
        z[:, -1] = rng.integers(0, 1 << (N - 64 * (nw - 1)), n, dtype=np.uint64)
        x[:, -1] = rng.integers(0, 1 << (N - 64 * (nw - 1)), n, dtype=np.uint64)
    elif keys == "clustered":          # nearly all records share their leading words
        z[:, -1] = (rng.random(n) < 1e-3).astype(np.uint64) << np.uint64(30)
    x[:, 0] ^= ids                     # unique with z, whatever the rest
    z[:, 0] ^= ids if keys == "spread" else np.uint64(0)
    o = np.lexsort([x[:, w] for w in range(nw)] + [z[:, w] for w in range(nw)])
    same = np.all(z[o][1:] == z[o][:-1], axis=1) & np.all(x[o][1:] == x[o][:-1], axis=1)
    keep = np.ones(n, dtype=bool)
    keep[o[1:][same]] = False          # keys must be unique
    z, x = np.ascontiguousarray(z[keep]), np.ascontiguousarray(x[keep])
    c = rng.standard_normal(len(z))
    v = pp.SparsePauliVector(N, max(16, len(c)), 16)
    v.upload(z, x, c, sorted=False)
    o = np.lexsort([x[:, w] for w in range(nw)] + [z[:, w] for w in range(nw)])
    gz, gx, gc = v.to_arrays()
    assert np.array_equal(gz, z[o]) and np.array_equal(gx, x[o])
    assert np.array_equal(gc.view(np.uint64), c[o].view(np.uint64))
    v.close()
