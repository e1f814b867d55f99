"""Diagonal blocks of 65 to 192 columns on the one-CTA kernel: eight columns at a
time while no column needs an interchange, a column at a time from there on.
Widths around the step, pivots from the start, from the middle, and none."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
sp = pytest.importorskip("scipy.sparse")


@pytest.mark.parametrize("fp32", [False, True])
@pytest.mark.parametrize("kind", ["none", "all", "half"])
@pytest.mark.parametrize("n", [65, 71, 72, 73, 130, 161, 192])
def test_block(n, kind, fp32):
    import nasoq_gb300 as nq

    rng = np.random.default_rng(n)
    r = rng.standard_normal((n, n))
    if kind == "all":
        a = r + r.T
        np.fill_diagonal(a, 0.0)
    else:
        a = r @ r.T / n + 4 * np.eye(n)
        if kind == "half":
            h = n // 2 + 3
            s = rng.standard_normal((n - h, n - h))
            a[h:, h:] = s + s.T
            a[h:, :h] *= 0.1
            a[:h, h:] *= 0.1
    low = sp.csc_matrix(np.tril(np.ones_like(a)))
    low.sort_indices()
    low.data = a[low.indices, np.repeat(np.arange(n), np.diff(low.indptr))]
    rhs = rng.standard_normal(n)
    plan = nq.Plan(n, low.indptr, low.indices, low.data, precision=nq.NQG_FP32 if fp32 else nq.NQG_FP64,
                   req_ref_iter=4, max_inner_iter=8)
    plan.factor()
    x = plan.solve(rhs)
    res = np.abs(a @ x - rhs).max()
    if fp32:  # FP32 factor with a diagonal floor, refined in FP64: the bound of the other FP32 checks
        assert res <= 1e-10 * (np.abs(a) @ np.abs(x) + np.abs(rhs)).max()
    else:  # backward stable with refinement
        assert res <= n * np.finfo(float).eps * (np.abs(a) @ np.abs(x) + np.abs(rhs)).max()
