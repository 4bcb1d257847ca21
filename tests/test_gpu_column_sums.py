"""PageRank's column weights summed on the device (2^17 entries and more):
columns of 0 and 1 entries, around 64, where a warp takes over from a lane,
and around whole warps of entries, in matrices on either side of that size.

The weights enter every step through the teleport term, so the vector is
compared with the oracle's, which sums them in a loop: both add a column's
values in entry order and agree to the bit; the bar is the SpMV's rounding,
1e-12 in the 1-norm over at most 60 steps."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["f64", "f32", "bf16"])
@pytest.mark.parametrize("n,extra", [(3000, 80_000), (3000, 140_000), (40_000, 300_000)])
def test_weights(gpu, prec, n, extra):
    T = gpu
    rng = np.random.default_rng(n + extra)
    col = [rng.integers(1500, n, extra)]
    for k, length in enumerate((1, 63, 64, 65, 95, 96, 97, 127, 128, 129, 2999, 5000)):
        col.append(np.full(length, 10 * k + 3))
    col = np.concatenate(col)
    row = rng.integers(0, n, len(col))
    order = np.argsort(row, kind="stable")
    col, row = col[order].astype(np.int32), row[order]
    rp = np.concatenate(([0], np.cumsum(np.bincount(row, minlength=n)))).astype(np.int32)
    # columns that sum to about 1/2 .. 1, in values of uneven size
    v = rng.uniform(0.5, 1.0, len(col)) * 2.0 ** -rng.integers(0, 12, len(col))
    v /= np.bincount(col, v, minlength=n)[col] * rng.uniform(1.0, 2.0, n)[col]
    m = T.MatrixCSR.from_arrays(n, n, rp, col, v)
    m.set_precision({"f64": T.F64, "f32": T.F32, "bf16": T.BF16}[prec])
    w = v if prec == "f64" else v.astype(np.float32).astype(np.float64) if prec == "f32" else oracle.bf16_round(v)
    x, *_ = m.page_rank(beta=0.85, epsilon=1e-13, max_iterations=60)
    ref = oracle.pagerank(rp, col, w, beta=0.85, epsilon=1e-13, max_iterations=60)
    assert np.abs(x - ref[0]).sum() <= 1e-12
    again = T.MatrixCSR.from_arrays(n, n, rp, col, v)
    again.set_precision({"f64": T.F64, "f32": T.F32, "bf16": T.BF16}[prec])
    assert np.array_equal(again.page_rank(beta=0.85, epsilon=1e-13, max_iterations=60)[0], x)


@pytest.mark.parametrize("used", ["first", "last", "ends", "one"])
def test_empty_columns(gpu, used):
    """Runs of empty columns before, between and after the others (a column
    per thread looks for its first entry)."""
    T = gpu
    n, count = 70_001, 150_000
    rng = np.random.default_rng(len(used))
    cols = {"first": np.arange(40), "last": np.arange(n - 40, n), "ends": np.r_[:20, n - 20:n], "one": [n // 2]}[used]
    col = rng.choice(cols, count).astype(np.int32)
    row = np.sort(rng.integers(0, n, count))
    rp = np.concatenate(([0], np.cumsum(np.bincount(row, minlength=n)))).astype(np.int32)
    v = rng.uniform(0.5, 1.0, count)
    v /= np.bincount(col, v, minlength=n)[col]
    m = T.MatrixCSR.from_arrays(n, n, rp, col, v)
    x, *_ = m.page_rank(beta=0.85, epsilon=1e-13, max_iterations=60)
    ref = oracle.pagerank(rp, col, v, beta=0.85, epsilon=1e-13, max_iterations=60)
    assert np.abs(x - ref[0]).sum() <= 1e-12


@pytest.mark.parametrize("prec", ["f64", "f32", "bf16"])
@pytest.mark.parametrize("lengths", [[4096], [4097], [200_000], [60_000, 40_000, 40_000, 5000, 4096],
                                     [9000] * 14, [30_000] * 3 + [4097] * 300])
def test_hub_columns(gpu, lengths, prec):
    """Columns next to each other long enough for the host to add some of them
    (4097 entries and more, up to eleven equal ones) or, being many, none."""
    T = gpu
    n, extra = 9000, 150_000
    rng = np.random.default_rng(len(lengths) + lengths[0])
    col = np.concatenate([rng.integers(2000, n, extra)] + [np.full(k, 700 + i) for i, k in enumerate(lengths)])
    row = rng.integers(0, n, len(col))
    order = np.argsort(row, kind="stable")
    col, row = col[order].astype(np.int32), row[order]
    rp = np.concatenate(([0], np.cumsum(np.bincount(row, minlength=n)))).astype(np.int32)
    v = rng.uniform(0.5, 1.0, len(col)) * 2.0 ** -rng.integers(0, 12, len(col))
    v /= np.bincount(col, v, minlength=n)[col] * rng.uniform(1.0, 2.0, n)[col]
    m = T.MatrixCSR.from_arrays(n, n, rp, col, v)
    m.set_precision({"f64": T.F64, "f32": T.F32, "bf16": T.BF16}[prec])
    w = v if prec == "f64" else v.astype(np.float32).astype(np.float64) if prec == "f32" else oracle.bf16_round(v)
    x, *_ = m.page_rank(beta=0.85, epsilon=1e-13, max_iterations=60)
    ref = oracle.pagerank(rp, col, w, beta=0.85, epsilon=1e-13, max_iterations=60)
    assert np.abs(x - ref[0]).sum() <= 1e-12
