"""Persistent batched CG: how the rows are dealt out.  A warp takes the unit of
its index and claims further ones; a small batch runs on fewer CTAs.

Every system has to end at its FP64 true residual, recomputed here by the
oracle: ||b - A x|| <= 1e-8 ||b|| (1 + 1e-4), the slack covering the order of
the sums of the two residuals (1e-13 of ||A|| ||x|| against 1e-8 ||b||)."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu
TOL = 1e-8


def solve(T, edges, prec, precond, ctas=0):
    systems = []
    for i, e in enumerate(edges):
        m = T.MatrixCSR()
        m.fill_diffusion7(e, 1.0, 8.0, 40 + i)
        systems.append(m)
    rhs = np.concatenate([T.fill_uniform(e ** 3, -1.0, 1.0, 70 + i) for i, e in enumerate(edges)])
    b = T.Batch(systems, prec)
    b.set_ctas_per_sm(ctas)
    x, its, rr, ok = b.cg(rhs, max_iterations=5000, rel_tol=TOL, precond=precond, refresh=50)
    assert ok and b.engine()["persistent"]
    o = 0
    for m, e in zip(systems, edges):
        a, n = m.arrays(), e ** 3
        r = rhs[o:o + n] - oracle.csr_ax(a["rowptr"], a["colidx"], a["values"], x[o:o + n])
        assert np.linalg.norm(r) <= TOL * (1 + 1e-4) * np.linalg.norm(rhs[o:o + n]), e
        o += n
    return its


@pytest.mark.parametrize("prec", ["f32", "bf16", "f64"])
@pytest.mark.parametrize("edges", [
    [4],                      # half a unit: one CTA
    [8, 3, 5],                # systems below a unit, odd sizes (one row per thread)
    [10] * 16,                # a CTA's warps on several systems
    [76, 4, 44],              # past one unit per warp of the GPU: claims, and systems that end early
])
def test_units_and_claims(gpu, prec, edges):
    T = gpu
    p = {"f32": T.F32, "bf16": T.BF16, "f64": T.F64}[prec]
    its = solve(T, edges, p, 1)
    # one CTA per SM: other warps take the units, the same sums up to their order
    one = solve(T, edges, p, 1, ctas=1)
    assert (np.abs(its - one) <= np.maximum(1, its // 50)).all()


def test_many_systems(gpu):
    """As many systems as the persistent engine takes, plain and Jacobi."""
    T = gpu
    edges = [3 + k % 6 for k in range(256)]
    for precond in (0, 1):
        solve(T, edges, T.F32, precond)
