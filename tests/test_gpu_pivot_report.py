"""A non-positive pivot is reported for the values that have it: the next factorization of
good values in the same pattern, which reuses the analysis and the factor, is none."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_good_values_after_a_non_positive_pivot(pkg):
    n = 150
    rng = np.random.default_rng(8)
    G = rng.standard_normal((n, n)) / np.sqrt(n)
    A = G @ G.T + np.eye(n)
    iu = np.triu_indices(n)
    ia = np.concatenate([[1], 1 + np.cumsum(np.arange(n, 0, -1))]).astype(np.int64)
    a, ja = np.ascontiguousarray(A[iu]), (iu[1] + 1).astype(np.int64)
    bad = a.copy()
    bad[ia[70] - 1] *= -1.0  # a diagonal entry
    b = rng.standard_normal((2, n))
    x = np.zeros_like(b)
    h = np.zeros(64, dtype=np.int64)
    assert pkg.pardiso_64(h, 12, bad, ia, ja, nrhs=2) == -4
    assert pkg.pardiso_64(h, 12, a, ia, ja, nrhs=2) == 0
    assert pkg.pardiso_64(h, 33, a, ia, ja, nrhs=2, b=b, x=x) == 0
    want = np.linalg.solve(A, b.T).T
    assert np.abs(x - want).max() <= 1e-12 * np.abs(want).max()
    assert pkg.pardiso_64(h, 12, bad, ia, ja, nrhs=2) == -4
    pkg.pardiso_64(h, -1, a, ia, ja)
