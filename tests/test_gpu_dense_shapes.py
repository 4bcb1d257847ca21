"""DENSE GEMV over the shapes where its split of rows and columns changes: rows
per warp, column parts, steps that end inside a row, rows that are not
aligned, against the oracle on the values as stored.

Tolerance: the FP64 bar of test_gpu_spmv.py, 1e-13 of sum_j |a_ij x_j| per
entry (double-float: x and FP64 values held to 2^-49, and Dot2 over at most
8192 / 32 columns a lane, 256 roundings of 2^-48 of partial sums at most, in a
random walk)."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu
TOL = 1e-13


@pytest.mark.parametrize("prec", ["f64", "f32", "bf16"])
@pytest.mark.parametrize("shape", [(1, 1), (2, 3), (7, 127), (9, 128), (5, 129), (33, 255), (3, 256), (17, 257),
                                   (1, 8192), (3, 4099), (700, 1024), (5000, 1100), (5001, 1101), (20_003, 130),
                                   (10_000, 520), (4000, 5124), (9800, 5120)])
def test_shapes(gpu, prec, shape):
    T = gpu
    nr, nc = shape
    rng = np.random.default_rng(nr * 10_000 + nc)
    a = rng.uniform(-1, 1, (nr, nc))
    a[rng.random((nr, nc)) < 0.1] = 0.0
    m = T.MatrixDENSE.from_arrays(nr, nc, a)
    m.set_precision({"f64": T.F64, "f32": T.F32, "bf16": T.BF16}[prec])
    v = a if prec == "f64" else a.astype(np.float32).astype(np.float64) if prec == "f32" else oracle.bf16_round(a)
    x = rng.uniform(-1, 1, nc)
    wide = x.copy()  # one entry out of the double-float range: the same launch in FP64
    wide[nc // 2] = 1e15
    for xv in (x, wide):
        ref = oracle.dense_ax(v, nr, nc, xv, np.full(nr, 0.25))
        scale = oracle.dense_ax(np.abs(v), nr, nc, np.abs(xv), np.full(nr, 0.25))
        r = np.full(nr, 0.25)
        m.Ax(r, xv)
        assert oracle.rel_err_normalized(r, ref, scale) <= TOL
        y = m.spmv(xv)
        assert oracle.rel_err_normalized(y, oracle.dense_ax(v, nr, nc, xv), scale) <= TOL
        assert np.array_equal(m.spmv(xv), y)
