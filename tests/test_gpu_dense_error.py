"""DENSE GEMV: the error against 64 bits over the widths at which the way a lane
keeps its sums changes.

The bar: no more error in the 2-norm than 256 threads a row leave, each with one
Dot2 sum of every 256th entry (vector of entries), added up in double-float over
the warps and in FP64 over the row; that arithmetic is restated below on the same
rows.  Both errors are sums over thousands of rows (each known to 1 / sqrt(2 rows),
1 to 2%), so 8% above the restated one."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu
f32, f64 = np.float32, np.float64


def two_sum(a, b):
    s = a + b
    t = s - a
    return s, (a - (s - t)) + (b - t)


def fast_two_sum(a, b):
    s = a + b
    return s, b - (s - a)


def fma(a, b, c):  # the product of two floats is exact in FP64
    return (a.astype(f64) * b.astype(f64) + c.astype(f64)).astype(f32)


def split(a):
    h = a.astype(f32)
    return h, (a - h).astype(f32)


def row_sums_256(a, x, fp64):
    """A x with 256 threads a row."""
    rows, cols = a.shape
    (ah, al), (xh, xl) = split(a), split(x)
    vec = 4 if cols % 4 == 0 else 1
    s, c = np.zeros((rows, 256), f32), np.zeros((rows, 256), f32)
    for g in range(0, cols // vec, 256):
        m = min(256, cols // vec - g)
        for k in range(vec):
            j = np.arange(g, g + m) * vec + k
            p = ah[:, j] * xh[j]
            e = fma(ah[:, j], xh[j], -p)
            t, r = two_sum(s[:, :m], p)
            u = fma(ah[:, j], xl[j], c[:, :m] + (e + r))
            s[:, :m], c[:, :m] = t, fma(al[:, j], xh[j], u) if fp64 else u
    h, lo = (v.reshape(rows, 8, 32) for v in two_sum(s, c))
    m = 32
    while m > 1:
        m //= 2
        sh, sl = two_sum(h[..., :m], h[..., m:])
        th, tl = two_sum(lo[..., :m], lo[..., m:])
        sh, sl = fast_two_sum(sh, sl + th)
        h, lo = fast_two_sum(sh, sl + tl)
    return (h[..., 0].astype(f64) + lo[..., 0].astype(f64)).sum(1)


@pytest.mark.parametrize("prec", ["f64", "f32", "bf16"])
@pytest.mark.parametrize("nc", [200, 401, 512, 513, 600, 800, 1000, 1003, 1104, 1301, 1544, 1801, 2000, 2312, 4099, 4104])
def test_error(gpu, nc, prec):
    T = gpu
    nr = min(4000, 5_000_000 // nc)
    rng = np.random.default_rng(nc)
    a, x = rng.uniform(-1, 1, (nr, nc)), rng.uniform(0, 1, nc)
    a = a if prec == "f64" else a.astype(f32).astype(f64) if prec == "f32" else oracle.bf16_round(a)
    m = T.MatrixDENSE.from_arrays(nr, nc, a)
    m.set_precision({"f64": T.F64, "f32": T.F32, "bf16": T.BF16}[prec])
    exact = (a.astype(np.longdouble) * x.astype(np.longdouble)).sum(1)
    err = lambda y: float(np.linalg.norm((y - exact).astype(f64)) / np.linalg.norm(exact.astype(f64)))
    assert err(m.spmv(x)) <= 1.08 * err(row_sums_256(a, x, prec == "f64"))
