"""COO / SCOO on each of the kernels their sizes lead to: row blocks below 2^19
triplets, sliced ELL from there on, triplet chunks where there are fewer
triplets than rows between the first and the last one, against the oracle.

Tolerance: the FP64 bar of test_gpu_spmv.py, 1e-13 of |r_i| + sum_j |a_ij x_j|
per entry (rows of at most 3000 triplets, one rounding of 1.1e-16 each)."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu
TOL = 1e-13


def triplets(n, n_col, count, seed):
    """Unsorted, with repeated positions, one row of 3000, rows without any:
    the first 5, the last 7 and others."""
    rng = np.random.default_rng(seed)
    long_row = min(3000, count // 3)
    row = 5 + rng.integers(0, n - 12, count)
    row[:long_row] = 5 + (n - 12) // 2
    row[long_row:long_row + 2] = (5, n - 8)
    col = rng.integers(0, n_col, count)
    val = rng.uniform(-1, 1, count)
    p = rng.permutation(count)
    return row[p].astype(np.int32), col[p].astype(np.int32), val


@pytest.mark.parametrize("prec", ["f64", "f32", "bf16"])
@pytest.mark.parametrize("n,n_col,count", [(13, 5, 3), (400, 90, 390), (2000, 2000, 9000), (40_000, 30_000, (1 << 19) - 1),
                                           (40_000, 30_000, 1 << 19), (300_000, 1000, 700_000), (50_000, 700, 2500)])
@pytest.mark.parametrize("fmt", ["coo", "scoo"])
def test_triplets(gpu, fmt, n, n_col, count, prec):
    T = gpu
    row, col, val = triplets(n, n_col, count, count + n)
    m = T.MatrixCOO.from_arrays(n, n_col, row, col, val)
    if fmt == "scoo":
        m = T.MatrixSCOO(m)
    m.set_precision({"f64": T.F64, "f32": T.F32, "bf16": T.BF16}[prec])
    v = val if prec == "f64" else val.astype(np.float32).astype(np.float64) if prec == "f32" else oracle.bf16_round(val)
    rng = np.random.default_rng(1)
    x = rng.uniform(-1, 1, n_col)
    r0 = rng.uniform(-1, 1, n)
    empty = np.setdiff1d(np.arange(n), row)
    r0[empty[::2]] = -0.0
    scale = oracle.coo_ax(n, row, col, np.abs(v), np.abs(x), np.abs(r0))
    for incr in (0, 7, -5):
        r = r0.copy()
        m.Ax(r, x, incr)
        ref = oracle.coo_ax(n, row, col, v, x, r0.copy(), incr) if incr >= 0 else None
        if incr < 0:  # the same rows, moved down
            ref = oracle.coo_ax(n, row + incr, col, v, x, r0.copy())
        assert oracle.rel_err_normalized(r, ref, np.roll(scale, incr) + np.abs(r0)) <= TOL
        hit = np.zeros(n, bool)
        hit[row + incr] = True
        assert np.array_equal(r[~hit].view(np.int64), r0[~hit].view(np.int64))  # other entries are not touched
        again = r0.copy()
        m.Ax(again, x, incr)
        assert np.array_equal(again, r)
    for incr in (8, -6):
        with pytest.raises(T.TbslaError):
            m.Ax(r0.copy(), x, incr)
    y = m.spmv(x)
    ref = oracle.coo_ax(n, row, col, v, x)
    assert oracle.rel_err_normalized(y, ref, scale) <= TOL
    assert not y[empty].any()
