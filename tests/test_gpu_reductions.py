"""Reductions at the sizes where their kernels change: the adaptive threshold in one
CTA (up to 2^18 terms, with ties, few distinct values and more candidates than its
list holds) against numpy, and the variance's long sigma entries."""
import numpy as np
import pytest

import pauliprop as pp

pytestmark = pytest.mark.gpu


def _vector(N, n, c):
    z = np.arange(n, dtype=np.uint64).reshape(-1, 1)
    v = pp.SparsePauliVector(N, max(16, n), 16)
    v.upload(z, np.zeros_like(z), c, sorted=True)
    return v


@pytest.mark.parametrize("n", [2, 1000, 1024, 5000, 1 << 18, (1 << 18) + 1])
@pytest.mark.parametrize("values", ["spread", "ties", "narrow"])
@pytest.mark.parametrize("keep", [0.0, 0.3, 1.0])
def test_adaptive_threshold(n, values, keep):
    rng = np.random.default_rng([n, int(10 * keep)])
    if values == "spread":
        c = 10.0 ** rng.uniform(-8, 1, n) * rng.choice([-1.0, 1.0], n)
    elif values == "ties":
        c = rng.choice([0.5, -0.5, 0.25, 1e-3, 0.0], n)
    else:                                     # the leading 22 bits agree: every value is a candidate
        c = 1.0 + rng.uniform(0, 1e-7, n)
    m = int(keep * n)
    v = _vector(40, n, c)
    pp.truncate_(v, pp.AdaptiveTruncation(m, 1e-3))
    a = np.abs(c)
    thr = np.sort(a)[n - 1 - m] if n > m else 1e-3
    on = a > thr
    z, x, got = v.to_arrays()
    assert np.array_equal(z[:, 0], np.flatnonzero(on).astype(np.uint64))
    assert np.array_equal(got.view(np.uint64), c[on].view(np.uint64))


@pytest.mark.parametrize("cand", [1, 2, 383, 384, 385, 3000])
@pytest.mark.parametrize("tied", [False, True])
@pytest.mark.parametrize("at", [0.0, 0.5, 1.0])
def test_adaptive_threshold_few_candidates(cand, tied, at):
    # the values in [1, 2) share the leading digit, the others are far away on both
    # sides: at most 384 candidates are ranked by counting, more by their digits
    n = 4000
    rng = np.random.default_rng([cand, int(tied), int(10 * at)])
    pool = 1.0 + rng.integers(0, 3, cand) / 4 if tied else 1.0 + (rng.permutation(cand) + 0.5) / cand
    c = np.concatenate([pool, np.full(400, 100.0), np.full(n - 400 - cand, 1e-5)]) * rng.choice([-1.0, 1.0], n)
    c = c[rng.permutation(n)]
    m = 400 + int(at * (cand - 1))            # the threshold is one of the candidates
    v = _vector(40, n, c)
    pp.truncate_(v, pp.AdaptiveTruncation(m, 1e-3))
    a = np.abs(c)
    on = a > np.sort(a)[n - 1 - m]
    z, _, got = v.to_arrays()
    assert np.array_equal(z[:, 0], np.flatnonzero(on).astype(np.uint64))
    assert np.array_equal(got.view(np.uint64), c[on].view(np.uint64))


@pytest.mark.parametrize("group", [1, 64, 65, 66, 127, 1000, 40001])
def test_variance_of_long_entries(group):
    """Var = sum over x of |sigma_x|^2 - sigma_psi^2, `group` terms in each of three
    entries: the z of a term is its position, so signs vary with psi."""
    N = 30
    rng = np.random.default_rng(group)
    z = np.tile(np.arange(group, dtype=np.uint64), 3)
    x = np.repeat(np.array([0, 1 << 20, 1 << 25], dtype=np.uint64), group)
    c = rng.standard_normal(3 * group)
    ket = 0b1011
    o = np.lexsort([x, z])
    v = pp.SparsePauliVector(N, 3 * group, 16)
    v.upload(z[o].reshape(-1, 1), x[o].reshape(-1, 1), c[o], sorted=True)
    sign = 1.0 - 2.0 * (np.bitwise_count(z & (x ^ np.uint64(ket))) & 1)
    s = [np.longdouble(sign[x == k] * c[x == k]).sum() for k in np.unique(x)]
    want = float(sum(t * t for t in s) - s[0] * s[0])
    # each of the terms of sigma_psi^2 and of the two other squares is rounded a few times
    tol = 4 * group * np.finfo(float).eps * float(sum(np.abs(c[x == k]).sum() ** 2 for k in np.unique(x)))
    assert abs(pp.variance(v, ket) - want) <= tol
