"""Residual norms at the edges of the kernel's row tiles (256 rows), column chunks (1, 2, 4
and 8) and staging buffer (tiles of more entries than fit are read directly)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("ncols", [1, 2, 3, 5, 8, 9, 64])
@pytest.mark.parametrize("n,per_row", [(1, 1), (255, 27), (256, 28), (257, 29), (600, 90)])
def test_norms_against_extended_precision(pkg, n, per_row, ncols):
    rng = np.random.default_rng(1000 * n + ncols)
    lens = np.minimum(per_row, n) * np.ones(n, dtype=np.int64)
    if per_row > 1:
        lens[::7] = 0  # empty rows among them
    ptr = np.concatenate([[0], np.cumsum(lens)])
    col = rng.integers(0, n, ptr[-1])
    val = rng.standard_normal(ptr[-1])
    ld = n + 3
    x, b = rng.standard_normal((2, ncols, ld))
    x[:, n:] = b[:, n:] = np.nan  # padding must not be read
    dev = [torch.from_numpy(v).cuda() for v in (ptr.astype(np.int64), col.astype(np.int32), val, x, b)]
    norms = torch.full((2 * ncols,), -1.0, dtype=torch.float64, device="cuda")
    pkg.residual_norms(0, n, *[v.data_ptr() for v in dev], ld, ncols, norms.data_ptr(),
                       torch.cuda.current_stream().cuda_stream)
    rows = np.repeat(np.arange(n), lens)
    want = np.empty(2 * ncols)
    for j in range(ncols):
        r = b[j, :n].astype(np.longdouble)
        np.subtract.at(r, rows, val * x[j, col].astype(np.longdouble))
        want[2 * j] = np.sqrt(np.sum(r * r))
        want[2 * j + 1] = np.sqrt(np.sum(b[j, :n].astype(np.longdouble) ** 2))
    # 90 products a row of unit size and a sum of n squares: (90 + log2 n + 4) u on each
    # row's magnitude, which random signs keep within 10 of the residual's
    assert np.allclose(norms.cpu().numpy(), want, rtol=1000 * 2.0 ** -53, atol=0)
