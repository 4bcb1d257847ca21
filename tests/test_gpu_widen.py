"""FP32 / BF16 values widened to FP64 on the integer pipes: every class of
stored value comes out exactly, A = diag(v) times ones in each format."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

SPECIAL = np.array([0.0, -0.0, 1.0, -1.5, np.inf, -np.inf, np.nan, 1e-45, -1e-45, 1.1754942e-38, 1.17549435e-38,
                    -1.17549435e-38, 3.4028235e38, -3.4028235e38, 2.0 ** -126, 2.0 ** -127, 2.0 ** 127, 1 + 2.0 ** -7,
                    1 + 2.0 ** -23, 9.1835e-41, 6.1e-39])


@pytest.mark.parametrize("prec", ["f32", "bf16"])
@pytest.mark.parametrize("fmt", ["csr", "sell", "merge", "coo", "ell"])
def test_special_values(gpu, prec, fmt):
    T = gpu
    rng = np.random.default_rng(3)
    v = np.concatenate([SPECIAL, rng.uniform(-2, 2, 300) * 2.0 ** rng.integers(-130, 127, 300)])
    n = len(v)
    i = np.arange(n)
    if fmt == "coo":
        m = T.MatrixCOO.from_arrays(n, n, i, i, v)
    elif fmt == "ell":
        m = T.MatrixELL.from_arrays(dict(n_row=n, n_col=n, ln_row=n, ln_col=n, nnz=n, max_col=1), i, v)
    else:
        m = T.MatrixCSR.from_arrays(n, n, np.arange(n + 1), i, v)
        m.set_algorithm({"csr": m.ROWBLOCK, "sell": m.SELL, "merge": m.MERGE}[fmt])
    m.set_precision(T.F32 if prec == "f32" else T.BF16)
    with np.errstate(over="ignore"):
        ref = v.astype(np.float32)
        if prec == "bf16":  # as stored: the high 16 bits of the float (they hold all but subnormals exactly)
            ref = (oracle.bf16_round(v).astype(np.float32).view(np.uint32) & np.uint32(0xFFFF0000)).view(np.float32)
    y = m.spmv(np.ones(n))
    assert np.array_equal(y, ref.astype(np.float64) + 0.0, equal_nan=True)
