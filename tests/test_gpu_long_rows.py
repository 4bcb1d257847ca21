"""Rows too long for one warp, cut into pieces that several warps sum: CSR
SpMV on the sliced-ELL layout and PageRank.

Tolerance of the SpMV: the FP64 bar of test_gpu_spmv.py, 1e-13 of
sum_j |a_ij x_j| per entry; a cut row adds at most 64 entries per lane, then
up to 3 pieces per lane and two butterflies of 5, under 80 roundings of
2^-53."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu
TOL = 1e-13


def ragged(T, n, lens, seed):
    rng = np.random.default_rng(seed)
    rowptr = np.zeros(n + 1, np.int64)
    full = rng.integers(0, 9, n)
    full[rng.choice(n, len(lens), replace=False)] = lens
    rowptr[1:] = np.cumsum(full)
    nnz = int(rowptr[-1])
    col = rng.integers(0, n, nnz)
    col = col[np.lexsort((col, np.repeat(np.arange(n), full)))]
    m = T.MatrixCSR.from_arrays(n, n, rowptr, col, rng.uniform(-1, 1, nnz))
    return m, full


@pytest.mark.parametrize("prec", ["f64", "f32", "bf16"])
@pytest.mark.parametrize("params", [(0, 0, 16384, 0), (4, 1, 64, 0), (64, 64, 16384, 20_000)])
def test_cut_rows_match_oracle(gpu, prec, params):
    """Row lengths around the cut (32 lanes x 64 steps = 2048 entries; with
    a threshold of one step, 32), one piece more, and a row of more pieces
    than a warp has lanes; one column block and three.  Repeated calls give
    the same bits."""
    T = gpu
    n = 50_000
    lens = [31, 32, 33, 64, 65, 2047, 2048, 2049, 4096, 4097, 70_001]
    m, _ = ragged(T, n, lens, 5)
    m.set_precision({"f64": T.F64, "f32": T.F32, "bf16": T.BF16}[prec])
    m.set_algorithm(m.SELL)
    m.set_sell_params(*params)
    a = m.arrays()
    v = a["values"]
    v = v.astype(np.float32).astype(np.float64) if prec == "f32" else oracle.bf16_round(v) if prec == "bf16" else v
    x = np.random.default_rng(6).uniform(-1, 1, n)
    ref = oracle.csr_ax(a["rowptr"], a["colidx"], v, x)
    scale = oracle.csr_absrow(a["rowptr"], a["colidx"], v, x)
    y = m.spmv(x)
    assert oracle.rel_err_normalized(y, ref, scale) <= TOL
    for _ in range(5):
        assert np.array_equal(m.spmv(x), y)


@pytest.mark.parametrize("prec", ["f64", "f32"])
def test_pagerank_with_hub_rows(gpu, prec):
    """Hub rows of 2049 to 30,000 in-links: the fused step (pieces summed by
    the last warp, their terms added in cut-row order) gives the oracle's
    vector, the separate pass's within 1e-13, and the same bits each time."""
    T = gpu
    n = 40_000
    m, _ = ragged(T, n, [2049, 5000, 30_000], 7)
    a = m.arrays()
    m = T.MatrixCSR.from_arrays(n, n, a["rowptr"], a["colidx"], np.ones(len(a["values"])))
    m.make_stochastic(np.zeros(n))
    m.set_precision(T.F64 if prec == "f64" else T.F32)
    m.set_algorithm(m.SELL)
    out = []
    for fused in (True, True, False):
        m.set_pagerank_fused(fused)
        x, it, _, ok = m.page_rank(0.85, 1e-10, 500)
        assert ok
        out.append((x, it))
    assert np.array_equal(out[0][0], out[1][0]) and out[0][1] == out[1][1] == out[2][1]
    assert np.abs(out[0][0] - out[2][0]).sum() <= 1e-13
    a = m.arrays()
    v = a["values"] if prec == "f64" else a["values"].astype(np.float32).astype(np.float64)
    xr, _, _ = oracle.pagerank(a["rowptr"], a["colidx"], v, 0.85, 1e-10, out[0][1], stop_early=False)
    assert np.abs(out[0][0] - xr).sum() <= 1e-10


@pytest.mark.parametrize("prec,nvec", [("f64", 1), ("f64", 32), ("f32", 32), ("bf16", 5)])
def test_batched_pagerank_with_hub_rows(gpu, prec, nvec):
    """The entry-stream form with rows around and past an item's length (64
    entries at this size) and hub rows of many pieces, empty rows before,
    between and after: each vector within 1e-10 in L1 of the oracle, and the
    double-float forms within 1e-13 of the warp-per-row form."""
    T = gpu
    n = 6000
    m, lens = ragged(T, n, [60, 63, 64, 65, 127, 128, 129, 3000, 20_000, 0, 0, 0], 11)
    a = m.arrays()
    m = T.MatrixCSR.from_arrays(n, n, a["rowptr"], a["colidx"], np.ones(len(a["values"])))
    m.make_stochastic(np.zeros(n))
    m.set_precision({"f64": T.F64, "f32": T.F32, "bf16": T.BF16}[prec])
    rng = np.random.default_rng(12)
    tele = np.zeros((n, nvec))
    for k in range(nvec):
        tele[rng.choice(n, 30, replace=False), k] = 1.0 / 30
    X, it, ok = m.page_rank_batched(tele, 0.85, 1e-10, 500)
    Y, it2, _ = m.page_rank_batched(tele, 0.85, 1e-10, 500)
    assert ok and it == it2 and np.abs(X - Y).sum(axis=0).max() <= 1e-13
    if prec != "f64":
        m.set_pagerank_stream(False)
        Z, it3, _ = m.page_rank_batched(tele, 0.85, 1e-10, 500)
        assert it3 == it and np.abs(X - Z).sum(axis=0).max() <= 1e-13
    a = m.arrays()
    v = a["values"]
    v = v.astype(np.float32).astype(np.float64) if prec == "f32" else oracle.bf16_round(v) if prec == "bf16" else v
    for k in {0, nvec // 2, nvec - 1}:
        xr, _, _ = oracle.pagerank(a["rowptr"], a["colidx"], v, 0.85, 1e-10, it, stop_early=False,
                                   teleport=np.ascontiguousarray(tele[:, k]))
        assert np.abs(X[:, k] - xr).sum() <= 1e-10, k
