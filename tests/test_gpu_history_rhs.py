"""The history right-hand side of several sources, both ways it is formed (in one launch and
from a combination made before), at the edges of its lane groups and row tiles, against
extended precision: Dirichlet rows, empty rows, one or two layers, with and without a source."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

SYMBOL = "_ZN4tdem18launch_history_rhsEPKlPKiPKdS5_S5_ddS5_dPKhiiPdS8_P11CUstream_st"


@pytest.mark.parametrize("nsrc", [2, 3, 4, 5, 8, 9, 16, 17, 32, 33, 40])
@pytest.mark.parametrize("n", [1, 7, 33, 1000, 30_000])
def test_right_hand_side_of_several_sources(pkg, n, nsrc):
    launch = getattr(pkg.load_library(), SYMBOL)
    P, D, I = ctypes.c_void_p, ctypes.c_double, ctypes.c_int
    launch.argtypes, launch.restype = [P, P, P, P, P, D, D, P, D, P, I, I, P, P, P], None
    rng = np.random.default_rng(n + nsrc)
    lens = np.minimum(rng.integers(1, 42, n), n)
    lens[rng.random(n) < 0.1] = 0
    lens[0] = min(33, n)
    ptr = np.concatenate([[0], np.cumsum(lens)])
    col, val = rng.integers(0, n, ptr[-1]), rng.standard_normal(ptr[-1])
    u1, u2, src = rng.standard_normal((3, nsrc, n))
    bound = (rng.random(n) < 0.15).astype(np.uint8)
    gpu = [torch.from_numpy(v).cuda() for v in (ptr.astype(np.int64), col.astype(np.int32), val, u1, u2, src, bound)]
    rp, cc, cv, d1, d2, ds, db = [g.data_ptr() for g in gpu]
    gone = torch.full((nsrc, n), float("nan"), dtype=torch.float64, device="cuda")

    def row_sums(p):  # (a zero behind the last entry, where empty rows at the end begin)
        return np.where(lens > 0, np.add.reduceat(np.append(p, 0), ptr[:-1]), 0)

    for m1, m2, coef in ((0.7, -0.2, 0.3), (1.5, 0.0, 0.0)):
        rhs, scratch = torch.full_like(gone, 7.0), torch.full_like(gone, float("nan"))
        # without a second layer, and without a source, what stands there must not be used
        launch(rp, cc, cv, d1, d2 if m2 else gone.data_ptr(), m1, m2, ds if coef else gone.data_ptr(), coef, db, n, nsrc,
               rhs.data_ptr(), scratch.data_ptr(), torch.cuda.current_stream().cuda_stream)
        got = rhs.cpu().numpy()
        for p in range(nsrc):
            v = m1 * u1[p].astype(np.longdouble) + m2 * u2[p].astype(np.longdouble)
            size = abs(m1 * u1[p]) + abs(m2 * u2[p])
            want = row_sums(val * v[col]) + coef * src[p]
            # L products of values combined with two roundings, one more for the source
            tol = 2.0 ** -53 * ((lens + 4) * row_sums(np.abs(val) * size[col])
                        + 4 * np.abs(coef * src[p]))
            assert np.all(np.abs(got[p] - want)[bound == 0] <= tol[bound == 0])
            assert np.all(got[p][bound == 1] == 0.0)
