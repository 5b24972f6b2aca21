"""Factorization of levels with many tiles, whose inner panels take the outer panel's
finished ones in one update just before they are factored: fronts without update rows
(dense blocks of n pivots; the 600 end in a second outer panel with few tiles) and with them (a chain of
coupled blocks), with more tiles than SMs on a level (and, with 100 blocks, fewer).  The
blocks' own levels are followed by levels of fronts without rows, which launch nothing: what
a launch of no blocks leaves behind would fail the next case's set-up."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _blocks(n, count, coupled, seed):
    """Diagonal blocks and, where coupled, the blocks below them."""
    rng = np.random.default_rng(seed)
    G = rng.standard_normal((count, n, n)) / np.sqrt(n)
    d = 10.0 ** rng.uniform(-3, 3, (count, n))
    D = G @ G.transpose(0, 2, 1) + (3.0 if coupled else 0.1) * np.eye(n)
    D = d[:, :, None] * ((D + D.transpose(0, 2, 1)) / 2) * d[:, None, :]
    if not coupled:
        return D, None, d
    E = 0.3 * rng.standard_normal((count - 1, n, n)) / np.sqrt(n)  # norm below 0.7
    return D, d[1:, :, None] * E * d[:-1, None, :], d


@pytest.mark.parametrize("n,count,coupled", [(129, 150, False), (192, 100, False), (200, 80, False), (321, 60, False),
                                             (600, 40, False),
                                             (66, 511, True), (100, 255, True)])
def test_backward_error_of_many_fronts(pkg, n, count, coupled):
    D, E, d = _blocks(n, count, coupled, n)
    # upper triangle, row by row: the rest of the diagonal block, then the transposed block below
    ia, ja, a = [1], [], []
    for c in range(count):
        for i in range(n):
            row, col = D[c, i, i:], np.arange(c * n + i, (c + 1) * n)
            if coupled and c + 1 < count:
                row = np.concatenate([row, E[c][:, i]])
                col = np.concatenate([col, np.arange((c + 1) * n, (c + 2) * n)])
            a.append(row)
            ja.append(col + 1)
            ia.append(ia[-1] + len(row))
    a, ja, ia = np.concatenate(a), np.concatenate(ja).astype(np.int64), np.array(ia, dtype=np.int64)
    b = np.random.default_rng(1).standard_normal((1, n * count)) * d.reshape(1, -1)
    x = np.zeros_like(b)
    h = np.zeros(64, dtype=np.int64)
    assert pkg.pardiso_64(h, 12, a, ia, ja, nrhs=1) == 0
    assert pkg.pardiso_64(h, 33, a, ia, ja, nrhs=1, b=b, x=x) == 0
    pkg.pardiso_64(h, -1, a, ia, ja)
    X = x.reshape(count, n).astype(np.longdouble)
    R = b.reshape(count, n).astype(np.longdouble) - np.einsum("cij,cj->ci", D.astype(np.longdouble), X)
    s = np.sqrt(np.einsum("cii->ci", D))
    norm = np.sum(np.abs(X) * s, axis=1)
    if coupled:
        EL = E.astype(np.longdouble)
        R[1:] -= np.einsum("cij,cj->ci", EL, X[:-1])
        R[:-1] -= np.einsum("cij,ci->cj", EL, X[1:])
        norm = norm + np.concatenate([[0], norm[:-1]]) + np.concatenate([norm[1:], [0]])
    # row-scaled backward error of a Cholesky solve through inverted 64-wide blocks at
    # condition numbers below 50: 8 times the pivots that a row's sums run over
    terms = n if not coupled else 4 * n
    assert float(np.max(np.abs(R) / (s * norm[:, None] + np.abs(b.reshape(count, n))))) <= 8 * terms * 2.0 ** -53
