"""DENSE GEMV with x outside the double-float range: values on which float pairs
give infinities or zeros, so that only the FP64 rows of the same launch are
right.

One flag per CTA of the kernel that splits x (256 columns each, 64 CTAs at
most, which from 16,384 columns on take several pieces each): the entry that
sets it lies first, last, on either side of a CTA's end, in the second pass of
the flags' loop (columns from 8192 on) and in a later piece.

Tolerance: the FP64 bar of test_gpu_spmv.py, 1e-13 of sum_j |a_ij x_j| per
entry (rows of at most 40,000 columns in at least 256 sums, one rounding of
1.1e-16 each)."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu
TOL = 1e-13


def stored(a, prec):
    return a if prec == "f64" else a.astype(np.float32).astype(np.float64) if prec == "f32" else oracle.bf16_round(a)


@pytest.mark.parametrize("prec", ["f64", "f32", "bf16"])
@pytest.mark.parametrize("shape", [(1, 1), (3, 5), (9, 257), (33, 1000), (700, 1024), (40_003, 130), (3000, 2600), (17, 9000),
                                   (5, 16_384), (5, 16_385), (6, 40_000)])
def test_out_of_range(gpu, prec, shape):
    T = gpu
    nr, nc = shape
    rng = np.random.default_rng(nr + nc)
    a = rng.uniform(-1, 1, (nr, nc))
    m = T.MatrixDENSE.from_arrays(nr, nc, a)
    m.set_precision({"f64": T.F64, "f32": T.F32, "bf16": T.BF16}[prec])
    v = stored(a, prec)
    plain = rng.uniform(-1, 1, nc)
    for at in sorted({k for k in (0, 255, 256, nc // 2, 8191, 8192, 16_383, 16_384, nc - 1) if k < nc}):
        x = plain.copy()
        x[at] = 1e300  # infinite in a float
        check(m, v, nr, nc, x)
    check(m, v, nr, nc, plain * 1e-60)  # zero in a float
    check(m, v, nr, nc, np.where(np.arange(nc) == nc // 2, plain * 1e-60, 0.0))
    check(m, v, nr, nc, plain)  # and back in the range: no flag stays behind


def check(m, v, nr, nc, x):
    ref = oracle.dense_ax(v, nr, nc, x)
    scale = oracle.dense_ax(np.abs(v), nr, nc, np.abs(x))
    y = m.spmv(x)
    assert np.isfinite(y).all() and oracle.rel_err_normalized(y, ref, scale) <= TOL
    r = np.full(nr, scale.max() / 4)
    m.Ax(r, x)
    assert oracle.rel_err_normalized(r, ref + scale.max() / 4, scale + scale.max() / 4) <= TOL
    assert np.array_equal(m.spmv(x), y)
