"""Launches that are set up while the kernel before them still runs: chains of
products in which each reads what the one before wrote, and writes what that
one read, against the same products with a synchronisation after each, and
inside a captured graph behind a copy and a memset.  Bit for bit: the kernels
sum in a fixed order."""
import contextlib
import gc

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def matrix(T, kind, n):
    rng = np.random.default_rng(n)
    if kind == "dense":
        return T.MatrixDENSE.from_arrays(n, n, rng.uniform(-1, 1, (n, n)) / n)
    per = 7
    row = np.repeat(np.arange(n, dtype=np.int32), per)
    row[: per * 3] = 5  # rows 0 .. 2 without triplets
    col = rng.integers(0, n, n * per).astype(np.int32)
    order = np.argsort(row, kind="stable")
    row, col = row[order], col[order]
    val = rng.uniform(-1, 1, n * per) / per
    if kind == "coo":
        return T.MatrixCOO.from_arrays(n, n, row, col, val)
    if kind == "ell":
        return T.MatrixELL(T.MatrixCOO.from_arrays(n, n, row, col, val))
    rp = np.concatenate(([0], np.cumsum(np.bincount(row, minlength=n))))
    m = T.MatrixCSR.from_arrays(n, n, rp, col, val)
    if kind == "sell":
        m.set_algorithm(m.SELL)
    return m


@contextlib.contextmanager
def capture(torch, stream):
    """A graph captured on `stream`; matrices that other tests left to the
    collector are freed before, not during the capture (a free ends it)."""
    gc.collect()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    enabled = gc.isenabled()
    gc.disable()
    try:
        with torch.cuda.stream(stream):
            graph.capture_begin()
            try:
                yield graph
            finally:
                graph.capture_end()
    finally:
        if enabled:
            gc.enable()


CASES = [("csr", 300), ("csr", 40_000), ("sell", 300), ("sell", 40_000), ("sell", 400_000), ("coo", 2000), ("coo", 400_000),
         ("ell", 300), ("ell", 100_000), ("dense", 100), ("dense", 1500)]


@pytest.mark.parametrize("kind,n", CASES)
def test_chain(gpu, kind, n):
    torch = pytest.importorskip("torch")
    m = matrix(gpu, kind, n)
    x0 = torch.linspace(-1, 1, n, dtype=torch.float64, device="cuda")
    st = torch.cuda.Stream()  # (stream 0 would mean the matrix's own)
    torch.cuda.synchronize()

    def chain(steps, wait):
        v = [x0.clone(), torch.empty_like(x0)]
        for k in range(steps):
            m.spmv_device(v[(k + 1) % 2], v[k % 2], stream=st.cuda_stream)
            if k % 10 == 9:
                v[(k + 1) % 2].mul_(1.5).add_(0.25)
            if wait:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        return v[steps % 2]

    with torch.cuda.stream(st):
        want = chain(60, True)
        assert torch.isfinite(want).all() and want.abs().max() > 0
        for _ in range(5):
            assert torch.equal(chain(60, False), want)


@pytest.mark.parametrize("kind,n", CASES)
def test_captured(gpu, kind, n):
    torch = pytest.importorskip("torch")
    m = matrix(gpu, kind, n)
    m.upload()
    x = torch.linspace(-1, 1, n, dtype=torch.float64, device="cuda")
    src, a, b, r = x.clone(), torch.empty_like(x), torch.empty_like(x), torch.empty_like(x)
    side = torch.cuda.Stream()

    def work(stream):
        a.copy_(src)
        m.spmv_device(b, a, stream=stream)
        m.spmv_device(a, b, stream=stream)
        r.zero_()
        m.Ax_device(r, a, stream=stream)
        m.Ax_device(r, b, stream=stream)

    with torch.cuda.stream(side):
        work(side.cuda_stream)
    with capture(torch, side) as graph:
        work(side.cuda_stream)
    for scale in (1.0, -3.0):
        src.copy_(x * scale)
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        got = r.clone()
        with torch.cuda.stream(side):
            work(side.cuda_stream)
        torch.cuda.synchronize()
        assert torch.equal(got, r) and r.abs().max() > 0


@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("kind,n", CASES)
def test_two_streams(gpu, kind, n, captured):
    """Two matrices on two streams that wait for one another by events: each
    product reads what the other stream wrote, behind a slow kernel there."""
    torch = pytest.importorskip("torch")
    m, w = matrix(gpu, kind, n), matrix(gpu, kind, n)
    m.upload()
    w.upload()
    x = torch.linspace(-1, 1, n, dtype=torch.float64, device="cuda")
    src, a, b, c, d = (x.clone() for _ in range(5))
    big = torch.ones(1 << 25, device="cuda")
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()

    def work():
        with torch.cuda.stream(s1):
            for _ in range(4):
                big.mul_(1.0)
            m.spmv_device(a, src, stream=s1.cuda_stream)
            e1 = torch.cuda.Event()
            e1.record(s1)
        with torch.cuda.stream(s2):
            s2.wait_event(e1)
            w.spmv_device(b, a, stream=s2.cuda_stream)  # a: from s1
            for _ in range(4):
                big.mul_(1.0)
            w.spmv_device(c, b, stream=s2.cuda_stream)
            e2 = torch.cuda.Event()
            e2.record(s2)
        with torch.cuda.stream(s1):
            m.spmv_device(d, a, stream=s1.cuda_stream)
            s1.wait_event(e2)
            m.spmv_device(d, c, stream=s1.cuda_stream)  # c: from s2

    torch.cuda.synchronize()
    if captured:
        work()
        with capture(torch, s1) as graph:
            work()
    for scale in (1.0, -3.0, 0.5):
        for t in (a, b, c, d):
            t.fill_(7.0)
        src.copy_(x * scale)
        torch.cuda.synchronize()
        graph.replay() if captured else work()
        torch.cuda.synchronize()
        want = src
        for _ in range(3):
            t = torch.empty_like(x)
            m.spmv_device(t, want, stream=s1.cuda_stream)
            torch.cuda.synchronize()
            want = t
        last = torch.empty_like(x)
        m.spmv_device(last, c, stream=s1.cuda_stream)
        torch.cuda.synchronize()
        assert torch.equal(c, want) and torch.equal(d, last) and d.abs().max() > 0
