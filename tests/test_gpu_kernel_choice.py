"""Which kernel and layout a matrix gets, read off the bytes of its device copy
(the layouts differ by their block and slice arrays) beside the oracle's
values.

Tolerance: the FP64 bar of test_gpu_spmv.py, 1e-13 of sum_j |a_ij x_j|."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu
TOL = 1e-13


def csr(T, n, lens, seed):
    rng = np.random.default_rng(seed)
    rp = np.concatenate(([0], np.cumsum(lens))).astype(np.int32)
    ci = rng.integers(0, n, rp[-1]).astype(np.int32)
    v = rng.uniform(-1, 1, rp[-1])
    x = rng.uniform(-1, 1, n)
    return T.MatrixCSR.from_arrays(n, n, rp, ci, v), x, oracle.csr_ax(rp, ci, v, x), oracle.csr_absrow(rp, ci, v, x)


def test_tile_under_the_automatic_kernel(gpu):
    """A block size that the caller sets holds under the automatic kernel as
    under the row-block one; without one its blocks are smaller."""
    T = gpu
    m, x, ref, scale = csr(T, 20_000, np.full(20_000, 9), 1)
    size = {}
    for algo in (m.AUTO, m.ROWBLOCK):
        m.set_algorithm(algo)
        for tile in (None, 1024, 2048, 4096):
            if tile:
                m.set_tile(tile)
            size[algo, tile] = (m.upload(), m.device_bytes())[1]
            assert oracle.rel_err_normalized(m.spmv(x), ref, scale) <= TOL
    for tile in (1024, 2048, 4096):
        assert size[m.AUTO, tile] == size[m.ROWBLOCK, tile]
    assert size[m.AUTO, None] == size[m.AUTO, 1024] > size[m.AUTO, 2048] > size[m.AUTO, 4096]


@pytest.mark.parametrize("col_block,makes", [(0, True), (3000, True), (2999, False), (100, False)])
def test_page_rank_layout_is_one_column_block(gpu, col_block, makes):
    """PageRank on a small matrix makes its sliced-ELL layout only where that
    is one launch a step, not one per column block."""
    T = gpu
    n = 3000
    rng = np.random.default_rng(2)
    rp = np.concatenate(([0], np.cumsum(rng.integers(0, 16, n)))).astype(np.int32)
    ci = rng.integers(0, n, rp[-1]).astype(np.int32)
    v = 1.0 / np.bincount(ci, minlength=n)[ci]
    m = T.MatrixCSR.from_arrays(n, n, rp, ci, v)
    m.set_sell_params(0, 0, 16384, col_block)
    m.upload()
    before = m.device_bytes()
    x, it, _, ok = m.page_rank(0.85, 1e-10, 500)
    ref = oracle.pagerank(rp, ci, v, 0.85, 1e-10, it, stop_early=False)[0]
    assert ok and np.abs(x - ref).sum() <= 1e-10
    assert (m.device_bytes() > before) == makes
