"""Residual norms where a tile's entries do not fit the staging buffers one row a thread:
rows shared by 2 to 32 threads, rows that a warp takes (one dense row among short ones, and
parts that do not fit at all), tiles whose parts and column chunks go to several CTAs, and
more tiles than CTAs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _lengths(kind, n, per_row, rng):
    lens = np.full(n, per_row, dtype=np.int64)
    if kind == "one":  # one row of all columns
        lens[(2 * n) // 3] = n
    elif kind == "some":  # every 50th row is longer than a thread takes, a few are empty
        lens[::50] = rng.integers(129, 400, len(lens[::50]))
        lens[7::60] = 0
    return lens


@pytest.mark.parametrize("ncols", [1, 2, 4, 9, 33, 64])
@pytest.mark.parametrize("kind,n,per_row", [("even", 256, 29), ("even", 255, 57), ("even", 60, 60), ("even", 300, 300),
                                            ("even", 700, 113), ("even", 500, 900), ("even", 76_000, 33),
                                            ("one", 9_000, 27), ("one", 200, 3), ("some", 2_000, 20),
                                            ("some", 500, 60)])
def test_long_rows_against_extended_precision(pkg, kind, n, per_row, ncols):
    if n > 70_000 and ncols not in (1, 9):
        pytest.skip("the large case with two column counts")
    rng = np.random.default_rng(n + per_row + ncols)
    lens = _lengths(kind, n, per_row, rng)
    ptr = np.concatenate([[0], np.cumsum(lens)])
    col = rng.integers(0, n, ptr[-1])
    val = rng.standard_normal(ptr[-1])
    ld = n + 1
    x, b = rng.standard_normal((2, ncols, ld))
    x[:, n:] = b[:, n:] = np.nan  # padding must not be read
    dev = [torch.from_numpy(v).cuda() for v in (ptr.astype(np.int64), col.astype(np.int32), val, x, b)]
    norms = torch.full((2 * ncols,), -1.0, dtype=torch.float64, device="cuda")
    pkg.residual_norms(0, n, *[v.data_ptr() for v in dev], ld, ncols, norms.data_ptr(),
                       torch.cuda.current_stream().cuda_stream)
    got = norms.cpu().numpy()
    u = 2.0 ** -53

    def row_sums(p):  # (a zero behind the last entry, where empty rows at the end begin)
        return np.where(lens > 0, np.add.reduceat(np.append(p, 0), ptr[:-1]), 0)

    for j in range(ncols):
        p = val * x[j, col].astype(np.longdouble)
        r = b[j, :n] - row_sums(p)
        size = np.abs(b[j, :n]) + row_sums(np.abs(p))
        want = np.sqrt(np.sum(r * r))
        # a row's sum of L products errs by (L + 2) u of their sizes, and a sum of n squares,
        # which runs over at most 300 partial sums in a row, by 300 u of itself
        tol = u * (np.sqrt(np.sum(((lens + 2) * size) ** 2)) + 300 * want)
        assert abs(got[2 * j] - want) <= tol
        bn = np.sqrt(np.sum(b[j, :n].astype(np.longdouble) ** 2))
        assert abs(got[2 * j + 1] - bn) <= 300 * u * bn
