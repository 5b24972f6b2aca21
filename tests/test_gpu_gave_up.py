"""The in-process solver boundary reports a device wait that gave up (the flag is set from
the host, nothing waits): factorization and solve return -5 whichever wait it was, the
factor is gone, and the next factorization is a good one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _system(n=200):
    rng = np.random.default_rng(4)
    G = rng.standard_normal((n, n)) / np.sqrt(n)
    A = G @ G.T + np.eye(n)
    iu = np.triu_indices(n)
    ia = np.concatenate([[1], 1 + np.cumsum(np.arange(n, 0, -1))]).astype(np.int64)
    b = rng.standard_normal((3, n))
    return np.ascontiguousarray(A[iu]), ia, (iu[1] + 1).astype(np.int64), b, np.linalg.solve(A, b.T).T


@pytest.mark.parametrize("which", [1, 2])
@pytest.mark.parametrize("phase", [12, 33])
def test_a_wait_that_gave_up_is_an_error(pkg, which, phase):
    lib = pkg.load_library()
    a, ia, ja, b, want = _system()
    x = np.zeros_like(b)
    h = np.zeros(64, dtype=np.int64)
    assert pkg.pardiso_64(h, 12, a, ia, ja, nrhs=3) == 0
    assert lib.tdem_test_pardiso_gave_up(h.ctypes.data, which) == 0
    if phase == 12:
        assert pkg.pardiso_64(h, 12, a, ia, ja, nrhs=3) == -5
    else:
        assert pkg.pardiso_64(h, 33, a, ia, ja, nrhs=3, b=b, x=x) == -5
    assert pkg.pardiso_64(h, 33, a, ia, ja, nrhs=3, b=b, x=x) == -1  # nothing to solve with
    for nrhs in (3, 1):  # one column: the other level solves
        assert pkg.pardiso_64(h, 12, a, ia, ja, nrhs=nrhs) == 0
        assert pkg.pardiso_64(h, 33, a, ia, ja, nrhs=nrhs, b=b[:nrhs], x=x[:nrhs]) == 0
        assert np.abs(x[:nrhs] - want[:nrhs]).max() <= 1e-12 * np.abs(want).max()
    pkg.pardiso_64(h, -1, a, ia, ja)
