"""Right-hand sides with NaN (one of them with every bit set, which is what an empty place
of the level solves' mailbox holds) and infinity through the one- and two-column solves:
they end, without an error, with every unknown coupled to the value not finite and the
others as if it were not there."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ALL_ONES = np.frombuffer(b"\xff" * 8, dtype=np.float64)[0]


@pytest.mark.parametrize("nrhs", [1, 2])
@pytest.mark.parametrize("value", [np.nan, ALL_ONES, -np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("at", [0, 300, 699])
def test_non_finite_right_hand_sides(pkg, nrhs, value, at):
    sizes = (700, 200)  # two dense blocks, not coupled
    n, rng = sum(sizes), np.random.default_rng(at)
    a, ja, ia, row = [], [], [1], 0
    for k in sizes:
        G = rng.standard_normal((k, k)) / np.sqrt(k)
        A = G @ G.T + np.eye(k)
        for i in range(k):
            a.append(A[i, i:])
            ja.append(np.arange(row + i, row + k) + 1)
            ia.append(ia[-1] + k - i)
        row += k
    a, ja, ia = np.concatenate(a), np.concatenate(ja).astype(np.int64), np.array(ia, dtype=np.int64)
    b = rng.standard_normal((nrhs, n))
    x, y = np.zeros_like(b), np.zeros_like(b)
    h = np.zeros(64, dtype=np.int64)
    assert pkg.pardiso_64(h, 12, a, ia, ja, nrhs=nrhs) == 0
    assert pkg.pardiso_64(h, 33, a, ia, ja, nrhs=nrhs, b=b, x=x) == 0
    b[0, at] = value
    assert pkg.pardiso_64(h, 33, a, ia, ja, nrhs=nrhs, b=b, x=y) == 0
    assert not np.any(np.isfinite(y[0, :700]))
    assert np.array_equal(y[0, 700:], x[0, 700:]) and np.array_equal(y[1:], x[1:])
    b[0, at] = 0.5  # and nothing of it stays behind
    assert pkg.pardiso_64(h, 33, a, ia, ja, nrhs=nrhs, b=b, x=y) == 0
    assert np.all(np.isfinite(y))
    pkg.pardiso_64(h, -1, a, ia, ja)
