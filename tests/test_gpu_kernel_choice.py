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


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("fmt", ["coo", "scoo"])
@pytest.mark.parametrize("longest", [10_239, 10_240, 10_241, 60_000])
def test_triplets_with_a_long_row(gpu, longest, fmt, prec):
    """A row of more than 10 2^10 triplets takes a small matrix from the row
    blocks (values, columns, row starts and blocks) to sliced ELL (slices, and
    4.5 bytes a row of descriptors instead of 4 of row starts)."""
    T = gpu
    n, rest = 20_000, 40_000
    rng = np.random.default_rng(longest)
    row = rng.integers(0, n, rest)
    row[row == n // 3] = n // 3 + 1
    row = np.concatenate((row, np.full(longest, n // 3), [0, n - 1])).astype(np.int32)
    col = rng.integers(0, n, len(row)).astype(np.int32)
    v = rng.uniform(-1, 1, len(row))
    m = T.MatrixCOO.from_arrays(n, n, row, col, v)
    if fmt == "scoo":
        m = T.MatrixSCOO(m)
    m.set_precision({"f64": T.F64, "f32": T.F32}[prec])
    w = v if prec == "f64" else v.astype(np.float32).astype(np.float64)
    x, r0 = rng.uniform(-1, 1, n), rng.uniform(-1, 1, n)
    r = r0.copy()
    m.Ax(r, x)
    scale = oracle.coo_ax(n, row, col, np.abs(w), np.abs(x), np.abs(r0))
    assert oracle.rel_err_normalized(r, oracle.coo_ax(n, row, col, w, x, r0.copy()), scale) <= TOL
    assert oracle.rel_err_normalized(m.spmv(x), oracle.coo_ax(n, row, col, w, x), scale) <= TOL
    entry = 12 if prec == "f64" else 8
    assert (m.device_bytes() > entry * len(row) + 4.3 * n) == (longest > 10_240)


@pytest.mark.parametrize("n,mean", [(1000, 10), (50_000, 10), (100_000, 16)])
def test_autotuned_handle(gpu, n, mean, tmp_path):
    """The automatic setting is the first candidate; whichever wins, PageRank
    keeps the layout that an untouched handle gives it, and the cache brings a
    second handle to the same setting."""
    from tbsla_gb300 import autotune as A

    T = gpu
    rng = np.random.default_rng(n)
    rp = np.concatenate(([0], np.cumsum(rng.integers(1, 2 * mean, n)))).astype(np.int32)
    ci = rng.integers(0, n, rp[-1]).astype(np.int32)
    v = 1.0 / np.bincount(ci, minlength=n)[ci]
    make = lambda: T.MatrixCSR.from_arrays(n, n, rp, ci, v)
    m, fresh = make(), make()
    best, trials = m.autotune(reps=3)
    assert trials[0]["algorithm"] == m.ROWBLOCK and trials[0]["tile"] == 1024
    assert best in trials and best["ms"] == min(t["ms"] for t in trials)
    assert {(t["short_thr"], t["long_thr"]) for t in trials if t["algorithm"] == m.SELL} >= {(16, 16), (64, 64)}
    sizes = []
    for h in (m, fresh):
        h.upload()
        before = h.device_bytes()
        x, it, _, ok = h.page_rank(0.85, 1e-10, 500)
        assert ok and np.abs(x - oracle.pagerank(rp, ci, v, 0.85, 1e-10, it, stop_early=False)[0]).sum() <= 1e-10
        sizes.append(h.device_bytes() - before)
    assert sizes[1] > 0 and (sizes[0] == sizes[1] or best["algorithm"] == m.SELL)
    path = str(tmp_path / "tune.json")
    first, second = make(), make()
    e = A.tune_csr(first, T.F64, path=path)
    f = A.tune_csr(second, T.F64, path=path)
    assert f["cached"] and e["settings"] == f["settings"]
    first.upload()
    second.upload()
    assert first.device_bytes() == second.device_bytes()


@pytest.mark.parametrize("count", [(1 << 19) - 1, 1 << 19, (3 << 20) - 1, 3 << 20])
@pytest.mark.parametrize("longest", [64, 65])
def test_automatic_kernel_by_size(gpu, count, longest):
    """Row blocks up to 2^19 entries, up to 3 2^20 where no row is longer than
    64, sliced ELL from there on: told by the bytes (the sliced-ELL copy holds
    the entries twice)."""
    T = gpu
    n = 100_000
    lens = np.full(n, count // n)
    lens[n // 2] = longest
    rest = count - lens.sum()
    others = np.delete(np.arange(n), n // 2)
    lens[others[: abs(rest)]] += np.sign(rest)
    assert lens.sum() == count and lens.max() == longest and lens[n // 2] == longest
    m, x, ref, scale = csr(T, n, lens, count + longest)
    y = m.spmv(x)
    assert oracle.rel_err_normalized(y, ref, scale) <= TOL
    sell = count >= 3 << 20 or (count >= 1 << 19 and longest > 64)
    assert (m.device_bytes() > 24 * count) == sell
    m.set_algorithm(m.SELL if sell else m.ROWBLOCK)
    if not sell:
        m.set_tile(1024)
    assert np.array_equal(m.spmv(x), y)


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("params,steps", [((0, 0, 16384, 0), 16), ((64, 64, 16384, 0), 64), ((8, 32, 16384, 0), 32)])
def test_cuts_at_the_threshold(gpu, params, steps, prec):
    """One column block, rows around one, two and three pieces of 32 lanes x
    `steps` entries (16: the automatic threshold below 2^22 entries).  The
    pieces of a cut row are told by the bytes: 8 a piece for its place, 8 for
    its sum, and a slice of its own."""
    T = gpu
    n, cut = 40_000, 32 * steps
    around = [cut - 1, cut, cut + 1, 2 * cut - 1, 2 * cut, 2 * cut + 1, 3 * cut, 3 * cut + 1]
    size = {}
    for which in ("cut", "one shorter"):
        lens = np.full(n, 6)
        lens[500 * (1 + np.arange(len(around)))] = np.array(around) - (which == "one shorter")
        m, x, _, _ = csr(T, n, lens, steps)
        m.set_precision({"f64": T.F64, "f32": T.F32}[prec])
        m.set_algorithm(m.SELL)
        m.set_sell_params(*params)
        a = m.arrays()
        v = a["values"] if prec == "f64" else a["values"].astype(np.float32).astype(np.float64)
        ref = oracle.csr_ax(a["rowptr"], a["colidx"], v, x)
        scale = oracle.csr_absrow(a["rowptr"], a["colidx"], v, x)
        y = m.spmv(x)
        assert oracle.rel_err_normalized(y, ref, scale) <= TOL
        assert np.array_equal(m.spmv(x), y)
        size[which] = m.device_bytes()
    # lengths one shorter: cut + 1 -> cut, 2 cut + 1 -> 2 cut, 3 cut + 1 -> 3 cut: three pieces and one cut row fewer
    assert size["cut"] - size["one shorter"] > 3 * (8 + 8 + 16 + 8 * 32)
