"""CSR row blocks under the automatic kernel: rows on either side of the length
at which a row forms a block on its own, among blocks of each lane count,
against the oracle.

Tolerance: the FP64 bar of test_gpu_spmv.py, 1e-13 of sum_j |a_ij x_j| per
entry (rows of at most 1500 entries, one rounding of 1.1e-16 each; the longer
rows of the last test add at most 64 entries a lane, then their pieces)."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu
TOL = 1e-13


# rows of `mean` entries give blocks of 1024 // mean rows (at most 256): 1, 2, 4, 8, 16, 32 lanes a row
@pytest.mark.parametrize("prec", ["f64", "f32", "bf16"])
@pytest.mark.parametrize("mean", [0, 3, 9, 20, 40, 80, 150])
def test_row_blocks(gpu, prec, mean):
    T = gpu
    n = 1201
    rng = np.random.default_rng(mean)
    lens = np.full(n, mean)
    for k, length in enumerate((31, 32, 33, 64, 65, 128, 129, 256, 257, 512, 513, 1023, 1024, 1025, 1500, 0, 1500, 65)):
        lens[37 + 61 * k] = length
    lens[[0, 1, 2, n - 1]] = (700, 40, 700, 1025)
    rp = np.concatenate(([0], np.cumsum(lens)))
    ci = rng.integers(0, n, rp[-1])
    v = rng.uniform(-1, 1, rp[-1])
    m = T.MatrixCSR.from_arrays(n, n, rp, ci, v)
    m.set_precision({"f64": T.F64, "f32": T.F32, "bf16": T.BF16}[prec])
    w = v if prec == "f64" else v.astype(np.float32).astype(np.float64) if prec == "f32" else oracle.bf16_round(v)
    x = rng.uniform(-1, 1, n)
    rp, ci = rp.astype(np.int32), ci.astype(np.int32)
    ref = oracle.csr_ax(rp, ci, w, x)
    scale = oracle.csr_absrow(rp, ci, w, x)
    y = m.spmv(x)
    assert oracle.rel_err_normalized(y, ref, scale) <= TOL
    assert np.array_equal(m.spmv(x), y)
    for tile in (256, 2048, 4096):
        m.set_tile(tile)
        assert oracle.rel_err_normalized(m.spmv(x), ref, scale) <= TOL
    m.set_algorithm(m.SELL)
    assert oracle.rel_err_normalized(m.spmv(x), ref, scale) <= TOL


def test_page_rank(gpu):
    """The PageRank step over such blocks, against the merge path's: 1-norm
    of the difference within 1e-12, as much as the last step's own change."""
    T = gpu
    n = 3000
    rng = np.random.default_rng(5)
    lens = np.minimum(1 + 7 * (200 // (1 + rng.permutation(n))), 1400)
    rp = np.concatenate(([0], np.cumsum(lens)))
    ci = rng.integers(0, n, rp[-1])
    v = 1.0 / np.bincount(ci, minlength=n)[ci]
    out = []
    for algo in (-1, T.MatrixCSR.ROWBLOCK, T.MatrixCSR.MERGE):
        m = T.MatrixCSR.from_arrays(n, n, rp, ci, v)
        if algo >= 0:
            m.set_algorithm(algo)
        out.append(m.page_rank(beta=0.85, epsilon=1e-12, max_iterations=500)[0])
    for x in out[:2]:
        assert np.abs(x - out[2]).sum() <= 1e-12


@pytest.mark.parametrize("count", [(1 << 19) - 1, 1 << 19, (3 << 20) - 1, 3 << 20])
@pytest.mark.parametrize("longest", [64, 65])
def test_kernel_by_size(gpu, count, longest):
    """Either side of the sizes where the automatic kernel changes."""
    T = gpu
    n = 60_000
    rng = np.random.default_rng(count + longest)
    lens = np.full(n, count // n)
    lens[n // 2] = longest
    lens[: count - lens.sum()] += 1
    rp = np.concatenate(([0], np.cumsum(lens)))
    ci = rng.integers(0, n, rp[-1])
    v = rng.uniform(-1, 1, rp[-1])
    m = T.MatrixCSR.from_arrays(n, n, rp, ci, v)
    x = rng.uniform(-1, 1, n)
    a = m.arrays()
    ref = oracle.csr_ax(a["rowptr"], a["colidx"], v, x)
    scale = oracle.csr_absrow(a["rowptr"], a["colidx"], v, x)
    assert oracle.rel_err_normalized(m.spmv(x), ref, scale) <= TOL


def test_page_rank_after_an_update(gpu):
    """PageRank's layout of a small matrix follows a change of the values: the
    vector of a matrix made from the changed arrays, bit for bit."""
    T = gpu
    n = 2000
    rng = np.random.default_rng(9)
    rp = np.concatenate(([0], np.cumsum(rng.integers(0, 12, n))))
    ci = rng.integers(0, n, rp[-1])
    m = T.MatrixCSR.from_arrays(n, n, rp, ci, rng.uniform(0.5, 1.5, rp[-1]))
    first, *_ = m.page_rank(beta=0.5)
    sums = np.zeros(n)
    m.make_stochastic(sums)
    a = m.arrays()
    fresh = T.MatrixCSR.from_arrays(n, n, a["rowptr"], a["colidx"], a["values"])
    x, it, *_ = m.page_rank(beta=0.85)
    y, jt, *_ = fresh.page_rank(beta=0.85)
    assert it == jt and np.array_equal(x, y) and not np.array_equal(x, first)


@pytest.mark.parametrize("prec", ["f64", "f32"])
def test_long_rows_by_size(gpu, prec):
    """2^22 entries and more, where FP64 rows are cut into longer pieces: rows
    around one and two pieces of 32 lanes x 32 and x 64 steps."""
    T = gpu
    n = 600_000
    rng = np.random.default_rng(22)
    lens = np.full(n, 8)
    lens[rng.choice(n, 10, replace=False)] = (1023, 1024, 1025, 2047, 2048, 2049, 4096, 4097, 8193, 70_001)
    rp = np.concatenate(([0], np.cumsum(lens)))
    ci = rng.integers(0, n, rp[-1])
    v = rng.uniform(-1, 1, rp[-1])
    m = T.MatrixCSR.from_arrays(n, n, rp, ci, v)
    m.set_precision({"f64": T.F64, "f32": T.F32}[prec])
    w = v if prec == "f64" else v.astype(np.float32).astype(np.float64)
    x = rng.uniform(-1, 1, n)
    a = m.arrays()
    y = m.spmv(x)
    ref = oracle.csr_ax(a["rowptr"], a["colidx"], w, x)
    assert oracle.rel_err_normalized(y, ref, oracle.csr_absrow(a["rowptr"], a["colidx"], w, x)) <= TOL
    assert np.array_equal(m.spmv(x), y)
