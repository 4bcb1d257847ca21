"""Performance cases of tbsla_gb300: the work its users have it do, through its
public entry points -- SpMV in the five formats, PageRank (one vector and
personalised in batches), batched Jacobi-PCG, the learned preconditioner's
gradient and the PCG solve with its factor.

A case is a dict of plain values; prepare() makes its inputs on the GPU from
the seed alone and the handle that a program keeps between calls, run() makes
one pass, exact() restates the result in 64 bits with torch.
"""
import math

import numpy as np
import torch

import tbsla_gb300 as T

PREC = {"f64": T.F64, "f32": T.F32, "bf16": T.BF16}
SIZE = {"f64": 8, "f32": 4, "bf16": 2}
NPARAMS, H = 6467, 32  # the learned preconditioner's parameters and width


# ---- the cases -------------------------------------------------------------------


def listed():
    return [
        # the smallest call: the 10^4-row matrix of the reference's own runs, inside an iterative method
        # that keeps its vectors on the GPU
        spmv("csr_f64_10k", "csr", 10_000, 10, "uniform", "f64"),
        # the benchmark's matrix: 2^24 power-law rows, past L2
        spmv("csr_f64_16M", "csr", 1 << 24, 16, "powerlaw", "f64"),
        # an ordinary ragged matrix with an odd size and narrow values
        spmv("csr_f32_1M", "csr", 1_000_003, 16, "powerlaw", "f32"),
        # a program written for the reference: host vectors in, a new host vector back
        spmv("csr_f64_host_400k", "csr", 400_000, 12, "powerlaw", "f64", host=True),
        # the triplet and ELL formats past L2
        spmv("coo_f64_4M", "coo", 1 << 22, 10, "uniform", "f64"),
        spmv("ell_f64_1.5M", "ell", 1_500_001, 10, "uniform", "f64"),
        # DENSE with bfloat16 values
        {"name": "dense_bf16_24k", "kind": "dense", "rows": 24_576, "cols": 8192, "dtype": "bf16"},
        # PageRank of a web-like graph, then 32 personalised vectors at once
        {"name": "pagerank_f32_4M", "kind": "pagerank", "n": 1 << 22, "mean": 16, "dtype": "f32"},
        {"name": "pagerank_batched_f32_1M", "kind": "ppr", "n": 1 << 20, "mean": 16, "nvec": 32, "dtype": "f32"},
        # many diffusion systems of uneven size solved together
        {"name": "cg_batch_f32", "kind": "cg", "edges": "16 24 32 40 48 56 64 16 24 32 40 48 56 64 80 96",
         "dtype": "f32", "precond": 1, "refresh": 50},
        # training of the learned preconditioner: loss and gradient on one system
        {"name": "mpnn_grad_48", "kind": "grad", "edge": 48, "probes": 8},
        # and its use: the factors of a batch and the PCG solve with them
        {"name": "learned_pcg_96", "kind": "cg", "edges": "96 96 96 96 96 96 96 96", "dtype": "f32", "precond": 2,
         "refresh": 400},
    ]


def spmv(name, fmt, n, mean, rows, dtype, host=False):
    return {"name": name, "kind": "spmv", "format": fmt, "n": n, "mean": mean, "rows": rows, "dtype": dtype,
            "host": host}


def draw(rng):
    """One more case of the same ranges."""

    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    dtype = rng.choice(["f64", "f64", "f32", "bf16"])
    kind = rng.choice(["csr", "csr", "csr", "coo", "scoo", "ell", "dense", "pagerank", "ppr", "cg", "cg", "grad"])
    if kind in ("csr", "coo", "scoo", "ell"):
        n = size(3000, 6_000_000)
        c = spmv("", kind, n, rng.randint(4, 24), "uniform" if kind == "ell" else rng.choice(["uniform", "powerlaw"]),
                 dtype, host=kind == "csr" and rng.random() < 0.25)
        del c["name"]
        return c
    if kind == "dense":
        return {"kind": kind, "rows": size(500, 24_000), "cols": size(500, 8192), "dtype": dtype}
    if kind == "pagerank":
        return {"kind": kind, "n": size(5000, 3_000_000), "mean": rng.randint(6, 20), "dtype": dtype}
    if kind == "ppr":
        return {"kind": kind, "n": size(5000, 800_000), "mean": rng.randint(6, 20), "nvec": rng.randint(2, 32),
                "dtype": dtype}
    if kind == "cg":
        pre = rng.choice([0, 1, 1, 2])
        edges = [size(12, 80) // 4 * 4 if rng.random() < 0.7 else size(12, 80) for _ in range(rng.randint(1, 10))]
        return {"kind": kind, "edges": " ".join(map(str, edges)), "dtype": rng.choice(["f32", "f32", "f64"]),
                "precond": pre, "refresh": rng.choice([50, 400])}
    return {"kind": kind, "edge": size(20, 64), "probes": rng.randint(4, 16)}


# ---- inputs ------------------------------------------------------------------------


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) % (1 << 62))


_streams = {}


def _stream():
    """The program's own stream."""
    dev = torch.cuda.current_device()
    if dev not in _streams:
        _streams[dev] = torch.cuda.Stream()
    return _streams[dev]


def _host(t):
    return t.cpu().numpy()


def _lengths(n, mean, rows, g):
    """Row lengths: constant, or Zipf(2) on [1, 4096] rescaled to the mean and rounded stochastically."""
    if rows == "uniform":
        return torch.full((n,), min(mean, n), dtype=torch.int64, device="cuda")
    u = torch.rand(n, generator=g, device="cuda", dtype=torch.float64)
    z = torch.clamp(1.0 / torch.clamp(u, min=1e-9), max=4096.0).floor()
    z *= mean / (math.log(4096.0) + 0.5772)
    z = (z + torch.rand(n, generator=g, device="cuda", dtype=torch.float64)).floor()
    return torch.clamp(z, 1, min(4096, n)).long()


def _sparse(c, seed):
    """Row pointer, columns (sorted in each row), values of an n x n matrix: 30% of a power-law row's columns
    within 1024 of the diagonal, the others uniform."""
    g = _gen(seed)
    n = c["n"]
    lens = _lengths(n, c["mean"], c["rows"], g)
    rowptr = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(lens, 0, out=rowptr[1:])
    nnz = int(rowptr[-1])
    row = torch.repeat_interleave(torch.arange(n, device="cuda"), lens, output_size=nnz)
    col = torch.randint(0, n, (nnz,), generator=g, device="cuda")
    if c["rows"] == "powerlaw":
        near = torch.randint(-1024, 1025, (nnz,), generator=g, device="cuda").add_(row).clamp_(0, n - 1)
        local = torch.rand(nnz, generator=g, device="cuda") < 0.3
        col = torch.where(local, near, col)
        del near, local
    key = (row << 32) | col
    del row, col
    key = torch.sort(key)[0]
    col = (key & 0xffffffff).int()
    del key
    val = torch.rand(nnz, generator=g, device="cuda", dtype=torch.float64).mul_(2).sub_(1)
    x = torch.rand(n, generator=g, device="cuda", dtype=torch.float64)
    return rowptr, col, val, x, lens


def _graph(c, seed):
    """CSR of the transposed adjacency, column-stochastic: out-degrees Zipf(2) with 5% dangling nodes, targets
    drawn towards a scattered set of popular nodes (the k-th most popular draws in proportion to k^-0.6)."""
    g = _gen(seed)
    n = c["n"]
    deg = _lengths(n, c["mean"], "powerlaw", g)
    deg[torch.rand(n, generator=g, device="cuda") < 0.05] = 0
    m = int(deg.sum())
    src = torch.repeat_interleave(torch.arange(n, device="cuda"), deg, output_size=m)
    u = torch.rand(m, generator=g, device="cuda", dtype=torch.float64)
    pop = torch.randperm(n, generator=g, device="cuda")
    dst = pop[(u.pow_(2.5) * n).long().clamp_(max=n - 1)]
    key = torch.unique((dst << 32) | src)
    del src, dst, u
    dst, src = key >> 32, key & 0xffffffff
    rowptr = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(torch.bincount(dst, minlength=n), 0, out=rowptr[1:])
    val = 1.0 / torch.bincount(src, minlength=n).double()[src]
    return rowptr, src.int(), val


def _teleports(c, seed):
    """n x nvec teleport vectors, each over 100 seed nodes."""
    g = _gen(seed + 1)
    n, k = c["n"], c["nvec"]
    t = torch.zeros(n, k, dtype=torch.float64, device="cuda")
    idx = torch.rand(n, k, generator=g, device="cuda").topk(min(100, n), dim=0)[1]
    return t.scatter_(0, idx, 1.0 / min(100, n))


def _diffusion(n, seed):
    """Slot-major values of the 7-point diffusion matrix on an n^3 grid with Dirichlet boundaries: face
    coefficients exp of a smooth Gaussian field.  Slots: -n^2, -n, -1, 0, 1, n, n^2."""
    g = _gen(seed)
    f = torch.randn(1, 1, n, n, n, generator=g, device="cuda", dtype=torch.float64)
    for _ in range(3):
        f = torch.nn.functional.avg_pool3d(torch.nn.functional.pad(f, (2,) * 6, mode="replicate"), 5, 1)
    f = f[0, 0]
    f = (f - f.mean()) / f.std()
    a = torch.zeros(7, n, n, n, dtype=torch.float64, device="cuda")
    diag = a[3]
    for d, (lo, hi) in enumerate(((0, 6), (1, 5), (2, 4))):
        face = torch.exp(0.5 * (f.narrow(d, 0, n - 1) + f.narrow(d, 1, n - 1)))
        a[hi].narrow(d, 0, n - 1).copy_(-face)
        a[lo].narrow(d, 1, n - 1).copy_(-face)
        diag.narrow(d, 0, n - 1).add_(face)
        diag.narrow(d, 1, n - 1).add_(face)
        for side in (0, n - 1):
            diag.select(d, side).add_(torch.exp(f.select(d, side)))
    return a.reshape(7, -1)


def _deltas(n):
    return torch.tensor([-n * n, -n, -1, 0, 1, n, n * n], device="cuda")


def _diffusion_csr(n, seed):
    a = _diffusion(n, seed).t().contiguous()
    live = a != 0
    rowptr = torch.zeros(n ** 3 + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(live.sum(1), 0, out=rowptr[1:])
    col = (torch.arange(n ** 3, device="cuda")[:, None] + _deltas(n))[live].int()
    return rowptr, col, a[live]


def _csr(n, rowptr, col, val):
    return T.MatrixCSR.from_arrays(n, n, _host(rowptr.int()), _host(col), _host(val))


def _edges(c):
    return [int(e) for e in c["edges"].split()]


def _rhs(c, seed):
    n = sum(e ** 3 for e in _edges(c))
    return torch.rand(n, generator=_gen(seed + 7), device="cuda", dtype=torch.float64).mul_(2).sub_(1)


def _theta(seed):
    """Parameters near those that training reaches: random message layers, a head close to the truncated
    Neumann series of the scaled matrix."""
    r = np.random.RandomState(seed % (1 << 31))
    th = np.zeros(NPARAMS, np.float32)
    th[:4 * H] = r.randn(4 * H) * 0.7
    o = 4 * H + H
    for _ in range(3):
        th[o:o + 2 * H * H] = r.randn(2 * H * H) * 0.09
        o += 2 * H * H + H
    th[o:o + H] = r.randn(H) * 2e-3   # w_e
    th[o + H] = -0.9                  # c_e
    th[o + H + 2:o + 2 * H + 2] = r.randn(H) * 2e-3  # w_d
    th[NPARAMS - 1] = math.log(math.e - 1)
    return th


def prepare(case, seed):
    c = case
    kind = c["kind"]
    s = {"case": c, "stream": _stream()}
    if kind == "spmv":
        n = c["n"]
        rowptr, col, val, x, lens = _sparse(c, seed)
        f = c["format"]
        if f == "csr":
            m = _csr(n, rowptr, col, val)
        elif f == "ell":
            k = int(lens[0])
            m = T.MatrixELL.from_arrays(dict(n_row=n, n_col=n, ln_row=n, ln_col=n, nnz=n * k, max_col=k),
                                        _host(col), _host(val))
        else:
            row = _host(torch.repeat_interleave(torch.arange(n, device="cuda", dtype=torch.int32), lens))
            if f == "coo":
                m = T.MatrixCOO.from_arrays(n, n, row, _host(col), _host(val))
            else:
                m = T.MatrixSCOO.from_arrays(dict(n_row=n, n_col=n, ln_row=n, ln_col=n, nnz=len(row)), row,
                                             _host(col), _host(val))
        s["v"] = _host(x) if c["host"] else x
        s["r"] = None if c["host"] else torch.zeros(n, dtype=torch.float64, device="cuda")
    elif kind == "dense":
        a, x = _dense(c, seed)
        m = T.MatrixDENSE.from_arrays(c["rows"], c["cols"], _host(a))
        s["v"], s["r"] = x, torch.zeros(c["rows"], dtype=torch.float64, device="cuda")
    elif kind in ("pagerank", "ppr"):
        m = _csr(c["n"], *_graph(c, seed))
        if kind == "ppr":
            s["t"] = _host(_teleports(c, seed))
            s["out"] = np.zeros_like(s["t"])
        else:
            s["out"] = np.zeros(c["n"])
    elif kind == "cg":
        systems = [_csr(e ** 3, *_diffusion_csr(e, seed + 31 * i)) for i, e in enumerate(_edges(c))]
        s["batch"] = T.Batch(systems, PREC[c["dtype"]])
        s["rhs"] = _host(_rhs(c, seed))
        s["x"] = np.zeros_like(s["rhs"])
        if c["precond"] == 2:
            s["net"] = T.MPNN(0)
            s["net"].set_params(_theta(seed))
        m = None
    else:
        m = None
        s["m"] = _csr(c["edge"] ** 3, *_diffusion_csr(c["edge"], seed))
        s["net"] = T.MPNN(0)
        s["net"].set_params(_theta(seed))
        s["z"] = _host(_probes(c, seed))
    if m is not None:
        m.set_precision(PREC[c["dtype"]])
        m.upload()
        s["m"] = m
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return s


def _dense(c, seed):
    g = _gen(seed)
    a = torch.rand(c["rows"], c["cols"], generator=g, device="cuda", dtype=torch.float64).mul_(2).sub_(1)
    return a, torch.rand(c["cols"], generator=g, device="cuda", dtype=torch.float64)


def _probes(c, seed):
    z = torch.randn(c["edge"] ** 3, c["probes"], generator=_gen(seed + 3), device="cuda", dtype=torch.float32)
    return z.double()


# ---- one pass ------------------------------------------------------------------------


def run(s):
    c = s["case"]
    kind = c["kind"]
    if kind == "spmv":
        if c["host"]:
            return s["m"].spmv(s["v"])
        if c["format"] in ("csr", "ell"):
            s["m"].Ax_device(s["r"], s["v"], stream=s["stream"])
        else:  # Ax of the triplet formats and of DENSE adds to r
            s["m"].spmv_device(s["r"], s["v"], stream=s["stream"])
        return s["r"]
    if kind == "dense":
        s["m"].spmv_device(s["r"], s["v"], stream=s["stream"])
        return s["r"]
    if kind == "pagerank":
        x, iterations, _, _ = s["m"].page_rank(beta=0.85, epsilon=1e-10, max_iterations=1000, out=s["out"])
        return {"x": x, "iterations": iterations}
    if kind == "ppr":
        x, iterations, _ = s["m"].page_rank_batched(s["t"], beta=0.85, epsilon=1e-10, max_iterations=1000,
                                                    out=s["out"])
        return {"x": x, "iterations": iterations}
    if kind == "cg":
        if c["precond"] == 2:
            s["batch"].factor_mpnn(s["net"])
        s["x"].fill(0.0)
        # a tolerance at which x is settled to about 1e-10 whatever the order of the sums; the iteration counts
        # follow that order, by one now and then: x is the result
        x, _, _, _ = s["batch"].cg(s["rhs"], s["x"], max_iterations=20000, rel_tol=1e-11, precond=c["precond"],
                                   refresh=c["refresh"])
        return x
    loss, grad = s["net"].loss_grad(s["m"], s["z"])
    return {"loss": loss, "grad": grad}


# ---- the work ------------------------------------------------------------------------


def work(case):
    c = case
    kind = c["kind"]
    if kind == "spmv":
        n, sv = c["n"], SIZE[c["dtype"]]
        nnz = n * min(c["mean"], n)
        idx = {"csr": 4 * nnz + 4 * (n + 1), "ell": 4 * nnz}.get(c["format"], 8 * nnz)
        return {"bytes": nnz * sv + idx + 16 * n, "flops": 2 * nnz}
    if kind == "dense":
        k = c["rows"] * c["cols"]
        return {"bytes": k * SIZE[c["dtype"]] + 8 * (c["rows"] + c["cols"]), "flops": 2 * k}
    if kind in ("pagerank", "ppr"):
        n, v = c["n"], c.get("nvec", 1)
        nnz = 0.95 * n * c["mean"]
        # an iteration reads the matrix and the iterate and writes the next one; about 25 of them
        it = nnz * (SIZE[c["dtype"]] + 4) + 4 * (n + 1) + 8 * n * (1 + 2 * v) + (8 * n * v if v > 1 else 0)
        return {"bytes": 25 * it + 8 * n * v * (2 if v > 1 else 1), "flops": 25 * (2 * nnz * v + 8 * n * v)}
    if kind == "cg":
        # per row and iteration: the 7 values, and p, q, r, z, x read and written where the method needs it
        s = 4 if c["dtype"] == "f32" else 8
        per = {0: 15 * s, 1: 19 * s, 2: 21 * s + 8}[c["precond"]]
        b = f = 0
        for e in _edges(c):
            its = {0: 12.0, 1: 6.0, 2: 3.5}[c["precond"]] * e
            b += e ** 3 * (its * per + 16)
            f += e ** 3 * its * (24 if c["precond"] < 2 else 40)
        return {"bytes": b, "flops": f}
    n = c["edge"] ** 3
    # the activations of the four levels written once and read once by the backward pass, the probe blocks,
    # the matrix; multiply-adds of the three dense layers forward and twice backward
    return {"bytes": n * (4 * 4 * H * 4 + 7 * 12 + c["probes"] * 4 * 8), "flops": n * (3 * 3 * 2 * 2 * H * H)}


# ---- the results in 64 bits ------------------------------------------------------------


def _stored(val, dtype):
    if dtype != "bf16":
        return val if dtype == "f64" else val.float().double()
    b = val.view(torch.int64)  # rounded to 8 significant bits, ties to even, in one step
    return (b + (1 << 44) - 1 + ((b >> 45) & 1)).bitwise_and_(-(1 << 45)).view(torch.float64)


def _row_sums(row, prod, n):
    return torch.zeros(n, dtype=torch.float64, device="cuda").index_add_(0, row, prod)


def _rows(rowptr):
    n = rowptr.numel() - 1
    return torch.repeat_interleave(torch.arange(n, device="cuda"), rowptr[1:] - rowptr[:-1])


def exact(case, seed):
    c = case
    kind = c["kind"]
    if kind == "spmv":
        rowptr, col, val, x, _ = _sparse(c, seed)
        y = _row_sums(_rows(rowptr), _stored(val, c["dtype"]) * x[col.long()], c["n"])
        return _host(y) if c["host"] else y
    if kind == "dense":
        a, x = _dense(c, seed)
        return _stored(a, c["dtype"]) @ x
    if kind == "pagerank":
        x, it = _pagerank(c, seed, torch.full((c["n"], 1), 1.0 / c["n"], dtype=torch.float64, device="cuda"))
        return {"x": _host(x[:, 0]), "iterations": it}
    if kind == "ppr":
        x, it = _pagerank(c, seed, _teleports(c, seed))
        return {"x": _host(x), "iterations": it}
    if kind == "cg":
        rhs, out, o = _rhs(c, seed), [], 0
        for i, e in enumerate(_edges(c)):
            out.append(_solve(e, seed + 31 * i, rhs[o:o + e ** 3]))
            o += e ** 3
        return _host(torch.cat(out))
    return _loss_grad(c, seed)


def _pagerank(c, seed, tele):
    rowptr, col, val = _graph(c, seed)
    n, row, col, val = c["n"], _rows(rowptr), col.long(), _stored(val, c["dtype"])
    A = torch.sparse_csr_tensor(rowptr, col, val, (n, n))
    w = _row_sums(col, val, n)
    x = torch.full_like(tele, 1.0 / n)
    for it in range(1, 1001):
        sums = x.sum(0)
        y = 0.85 * (A @ x) / sums + (1 - 0.85 * (w @ x) / sums) * tele
        err = (y - x / sums).abs().sum(0).max()
        x = y
        if err < 1e-10:
            break
    return x / x.sum(0), it


def _apply(a, n, x):
    y = a[3] * x
    for k, d in enumerate((-n * n, -n, -1, 0, 1, n, n * n)):
        if d < 0:
            y[-d:] += a[k][-d:] * x[:d]
        elif d > 0:
            y[:-d] += a[k][:-d] * x[d:]
    return y


def _solve(n, seed, b):
    """A^-1 b by Jacobi-PCG in 64 bits."""
    a = _diffusion(n, seed)
    x, r = torch.zeros_like(b), b.clone()
    z = r / a[3]
    p, rz = z.clone(), r @ z
    for k in range(20 * n + 500):
        q = _apply(a, n, p)
        alpha = rz / (p @ q)
        x += alpha * p
        r -= alpha * q
        z = r / a[3]
        new = r @ z
        p = z + (new / rz) * p
        rz = new
        if k % 50 == 49 and float(r.norm() / b.norm()) < 1e-14:
            break
    return x


def _loss_grad(c, seed):
    """The network's loss and gradient by automatic differentiation, weights rounded to bfloat16."""
    n = c["edge"]
    a = _diffusion(n, seed)
    N = n ** 3
    th = torch.from_numpy(_theta(seed)).cuda().bfloat16().double().requires_grad_()
    z = _probes(c, seed)
    s = a[3].rsqrt()
    deltas = (-n * n, -n, -1, 0, 1, n, n * n)

    def shift(v, d):  # row i of the result is row i + d of v
        out = torch.zeros_like(v)
        if d < 0:
            out[-d:] = v[:d]
        else:
            out[:N - d] = v[d:]
        return out

    e = torch.stack([a[k] * s * shift(s, d) for k, d in enumerate(deltas)])
    off = [0, 1, 2, 4, 5, 6]
    x = torch.stack([torch.ones_like(s), e[off].sum(0), e[off].square().sum(0), (e[off] != 0).sum(0) / 8.0], 1)
    h = torch.relu(x @ th[:4 * H].view(H, 4).t() + th[4 * H:5 * H])
    o = 5 * H
    for _ in range(3):
        w, b = th[o:o + 2 * H * H].view(H, 2 * H), th[o + 2 * H * H:o + 2 * H * H + H]
        m = sum(e[k][:, None] * shift(h, deltas[k]) for k in off)
        h = h + torch.relu(torch.cat([h, m], 1) @ w.t() + b)
        o += 2 * H * H + H
    we, ce, be, wd, bd = th[o:o + H], th[o + H], th[o + H + 1], th[o + H + 2:o + 2 * H + 2], th[o + 2 * H + 2]
    lower = [(s * ((h * shift(h, deltas[k])) @ we + ce * e[k] + be) * (a[k] != 0), deltas[k]) for k in (0, 1, 2)]
    lower.append((s * torch.nn.functional.softplus(h @ wd + bd), 0))
    u = sum(a[k][:, None] * shift(z, d) for k, d in enumerate(deltas))
    v = sum(shift(l[:, None] * u, -d) for l, d in lower)
    r = sum(l[:, None] * shift(v, d) for l, d in lower) - z
    loss = r.square().sum() / r.numel()
    loss.backward()
    return {"loss": float(loss.detach()), "grad": _host(th.grad)}
