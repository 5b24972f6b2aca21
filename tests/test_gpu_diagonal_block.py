"""The diagonal block kernel of the factorization (eight columns at a time, inverse by
16-wide block rows) at the edges of its blocks: one dense front of n pivots, so that its
last diagonal block is n mod 64 wide, and a pivot that is not positive at every place of
the eight columns."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _upper(A):
    n = len(A)
    iu = np.triu_indices(n)
    ia = np.concatenate([[1], 1 + np.cumsum(np.arange(n, 0, -1))]).astype(np.int64)
    return np.ascontiguousarray(A[iu]), ia, (iu[1] + 1).astype(np.int64)


def _spd(n, seed):
    rng = np.random.default_rng(seed)
    G = rng.standard_normal((n, n)) / np.sqrt(n)
    d = 10.0 ** rng.uniform(-4, 4, n)
    A = d[:, None] * (G @ G.T + 0.1 * np.eye(n)) * d
    return (A + A.T) / 2, rng.standard_normal((2, n)) * d


@pytest.mark.parametrize("n", [1, 7, 8, 9, 15, 16, 17, 31, 33, 48, 63, 64, 65, 90])
def test_solution_at_block_edges(pkg, n):
    A, b = _spd(n, n)
    a, ia, ja = _upper(A)
    x = np.zeros_like(b)
    h = np.zeros(64, dtype=np.int64)
    assert pkg.pardiso_64(h, 12, a, ia, ja, nrhs=2) == 0
    assert pkg.pardiso_64(h, 33, a, ia, ja, nrhs=2, b=b, x=x) == 0
    pkg.pardiso_64(h, -1, a, ia, ja)
    # normwise (row-scaled) backward error of a Cholesky solve through inverted blocks:
    # 8 n u covers the factor (n u) and the products with the inverses at the condition
    # number of G G^T + 0.1 I, below 50, of these matrices
    AL = A.astype(np.longdouble)
    res = np.abs(b - (AL @ x.T.astype(np.longdouble)).T)
    s = np.sqrt(np.diag(A))
    scale = s * (np.abs(x) @ s)[:, None] + np.abs(b)
    assert float(np.max(res / scale)) <= 8 * max(n, 8) * 2.0 ** -53


@pytest.mark.parametrize("at", [0, 5, 7, 8, 22, 39, 63, 64, 77])
def test_non_positive_pivot_is_reported(pkg, at):
    A, _ = _spd(80, 3)
    A[at, at] = -A[at, at]
    a, ia, ja = _upper(A)
    h = np.zeros(64, dtype=np.int64)
    assert pkg.pardiso_64(h, 12, a, ia, ja) == -4
    pkg.pardiso_64(h, -1, a, ia, ja)
