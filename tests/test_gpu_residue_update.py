"""The residue (Chinese remainder) trailing update at the edges of its 256 x 96 tiles: one
dense front of 512 + r pivots whose first trailing update has r rows, every such update
forced onto the integer tensor pipe."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("r", [1, 95, 97, 128, 129, 255, 257, 767, 769, 1100])
def test_trailing_update_at_tile_edges(pkg, monkeypatch, r):
    monkeypatch.setenv("TDEM_OZAKI_ALL", "1")
    n = 512 + r
    rng = np.random.default_rng(r)
    G = rng.standard_normal((n, n)) / np.sqrt(n)
    d = 10.0 ** rng.uniform(-8, 8, n)  # row scales over 16 decades
    A = d[:, None] * (G @ G.T + 0.1 * np.eye(n)) * d
    A = (A + A.T) / 2
    iu = np.triu_indices(n)
    ia = np.concatenate([[1], 1 + np.cumsum(np.arange(n, 0, -1))]).astype(np.int64)
    a, ja = np.ascontiguousarray(A[iu]), (iu[1] + 1).astype(np.int64)
    b = rng.standard_normal((2, n)) * d
    x = np.zeros_like(b)
    h = np.zeros(64, dtype=np.int64)
    assert pkg.pardiso_64(h, 12, a, ia, ja, nrhs=2) == 0
    assert pkg.pardiso_64(h, 33, a, ia, ja, nrhs=2, b=b, x=x) == 0
    pkg.pardiso_64(h, -1, a, ia, ja)
    # componentwise backward error of a Cholesky solve in doubles: at most 3 n u
    # (|L| |L^T| <= diagonal products), with the residual formed in extended precision
    AL = A.astype(np.longdouble)
    res = np.abs(b - (AL @ x.T.astype(np.longdouble)).T)
    scale = np.sqrt(np.diag(A)) * (np.abs(x) @ np.sqrt(np.diag(A)))[:, None] + np.abs(b)
    assert float(np.max(res / scale)) <= 3 * n * 2.0 ** -53
