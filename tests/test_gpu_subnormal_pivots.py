"""Subnormal positive pivots (whose reciprocals are not finite) at every kind of place in
the diagonal block's eight columns: factored like any other, and the neighbours' values
with them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("at", [[0], [5], [7], [8, 9], [14, 15, 16], [3, 33, 63], [63, 64], [79], list(range(40, 48))])
def test_rows_of_subnormal_diagonal(pkg, at):
    n = 80
    rng = np.random.default_rng(len(at) + 100 * at[0])
    G = rng.standard_normal((n, n)) / np.sqrt(n)
    d = 10.0 ** rng.uniform(-2, 2, n)
    d[at] = 10.0 ** rng.uniform(-155.3, -154.6, len(at))  # squares below 2^-1022 = 2.2e-308, reciprocals above 2^1024
    A = d[:, None] * (G @ G.T + 0.1 * np.eye(n)) * d
    A = np.triu(A) + np.triu(A, 1).T
    assert np.all(np.diag(A)[at] < 2.0 ** -1024) and np.all(np.diag(A)[at] > 1e-311)
    iu = np.triu_indices(n)
    ia = np.concatenate([[1], 1 + np.cumsum(np.arange(n, 0, -1))]).astype(np.int64)
    a, ja = np.ascontiguousarray(A[iu]), (iu[1] + 1).astype(np.int64)
    b = rng.standard_normal((2, n)) * d
    x = np.zeros_like(b)
    h = np.zeros(64, dtype=np.int64)
    assert pkg.pardiso_64(h, 12, a, ia, ja, nrhs=2) == 0
    assert pkg.pardiso_64(h, 33, a, ia, ja, nrhs=2, b=b, x=x) == 0
    pkg.pardiso_64(h, -1, a, ia, ja)
    AL = A.astype(np.longdouble)
    res = np.abs(b - (AL @ x.T.astype(np.longdouble)).T)
    s = np.sqrt(np.diag(AL))
    scale = s * (np.abs(x) @ s)[:, None] + np.abs(b)
    # row-scaled backward error: 8 n u as for normal values, and n roundings to multiples of
    # 2^-1074 in the updates of the smallest diagonal, with the same factor of 8
    tol = 8 * n * (2.0 ** -53 + float(np.longdouble(2.0) ** -1074 / np.diag(AL).min()))
    assert float(np.max(res / scale)) <= tol
