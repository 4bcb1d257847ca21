"""Learned preconditioner on other graphs than stencils: the device-built
lists (rows of more than 8 entries take the long path, columns of L of more
than 32 entries the sorted one) and remainders of the four nodes that a warp
takes together, against the float64 restatement (oracle/mpnn.py) with its
bars: loss 1e-4, gradient 1e-3 in norm (FP32 kernels), L 1e-5 of max |L|."""
import numpy as np
import pytest

import oracle.mpnn as M

pytestmark = pytest.mark.gpu


def spd(T, n, kind, seed):
    """Symmetric diagonally dominant: a line, an arrow (row and column 0
    full: one column of L holds n entries) or random rows of about 12."""
    rng = np.random.default_rng(seed)
    a = np.zeros((n, n))
    if kind != "random":
        i = np.arange(n - 1)
        a[i, i + 1] = a[i + 1, i] = -rng.uniform(0.2, 1.0, n - 1)
    if kind == "arrow" and n > 2:
        a[0, 2:] = a[2:, 0] = -rng.uniform(0.2, 1.0, n - 2)
    if kind == "random":
        m = np.triu(rng.random((n, n)) < min(1.0, 12.0 / n), 1)
        a = np.where(m, -rng.uniform(0.2, 1.0, (n, n)), 0.0)
        a = a + a.T
    np.fill_diagonal(a, -a.sum(1) + rng.uniform(0.5, 1.0, n))
    r, c = np.nonzero(a)
    rowptr = np.concatenate([[0], np.cumsum(np.bincount(r, minlength=n))])
    return T.MatrixCSR.from_arrays(n, n, rowptr, c, a[r, c])


@pytest.mark.parametrize("kind", ["line", "arrow", "random"])
@pytest.mark.parametrize("n,probes", [(1, 1), (2, 16), (7, 3), (33, 8), (130, 5), (1025, 8)])
def test_gradient_on_general_graphs(gpu, kind, n, probes):
    T = gpu
    A = spd(T, n, kind, n)
    a = A.arrays()
    rng = np.random.default_rng(5)
    th = M.unpack(M.init_params(3))
    th["we"] = rng.normal(0, 0.2, M.H)
    th["wd"] = rng.normal(0, 0.2, M.H)
    th["ce"], th["be"] = -0.3, 0.02
    theta = M.bf16(M.pack(th)).astype(np.float32)
    Z = rng.normal(size=(n, probes))
    net = T.MPNN(0)
    net.set_params(theta)
    loss, g = net.loss_grad(A, Z)
    ref, gr = M.loss_and_grad(theta.astype(np.float64), a["rowptr"], a["colidx"], a["values"], Z)
    assert abs(loss - ref) <= 1e-4 * ref
    assert np.linalg.norm(g - gr) <= 1e-3 * np.linalg.norm(gr)
    la = net.factor(A).arrays()
    r, c, v = M.factor(theta.astype(np.float64), a["rowptr"], a["colidx"], a["values"])
    rows = np.repeat(np.arange(n), np.diff(la["rowptr"]))
    got = {(i, j): x for i, j, x in zip(rows, la["colidx"], la["values"])}
    assert len(got) == len(v)
    assert max(abs(got[i, j] - x) for i, j, x in zip(r, c, v)) <= 1e-5 * np.abs(v).max()


def test_bad_graphs_are_refused(gpu):
    """A row without a positive diagonal entry, a column outside the matrix, a
    row pointer that falls: TBSLA_ERR_BAD_MATRIX, parameters untouched."""
    T = gpu
    net = T.MPNN(0)
    before = net.params()
    eye = [0, 1, 2, 3]
    for rowptr, col, val in ((eye, [0, 1, 2], [1.0, 0.0, 1.0]), (eye, [0, 1, 1], [1.0, 1.0, 1.0]),
                             (eye, [0, 1, 7], [1.0, 1.0, 1.0]), (eye, [0, -1, 2], [1.0, 1.0, 1.0]),
                             ([0, 2, 1, 3], [0, 1, 2], [1.0, 1.0, 1.0])):
        A = T.MatrixCSR.from_arrays(3, 3, rowptr, col, val)
        for call in (lambda: net.train_step(A, probes=2, seed=1, lr=1e-2), lambda: net.factor(A),
                     lambda: net.loss_grad(A, np.ones((3, 2)))):
            with pytest.raises(T.TbslaError) as e:
                call()
            assert e.value.status == T._lib.ERR_BAD_MATRIX
    assert np.array_equal(net.params(), before)
