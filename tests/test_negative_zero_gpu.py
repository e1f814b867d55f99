"""The Bunch-Kaufman search among explicit negative zeros: they are the smallest
magnitudes of a column, not the largest.  Diagonal blocks of every kernel
(warp, CTA up to 64 columns, up to 192, beyond), beside a zero and a tiny
diagonal; for FP32 also values that become -0.0f."""
import numpy as np
import pytest

import nasoq_gb300 as nq
from nasoq_gb300 import problems as P

pytestmark = pytest.mark.gpu


def _pairs(n, diag, zero):
    """Dense lower CSC of 2 x 2 blocks [[diag, c], [c, 1/4]], `zero` everywhere else."""
    a = np.full((n, n), zero)
    k = np.arange(0, n, 2)
    a[k, k], a[k + 1, k], a[k + 1, k + 1] = diag, 1.0 + k / n, 0.25
    rows, cols = np.tril_indices(n)
    order = np.lexsort((rows, cols))
    rows, cols = rows[order], cols[order]
    ptr = np.concatenate([[0], np.cumsum(np.bincount(cols, minlength=n))]).astype(np.int32)
    low = np.tril(a)
    return ptr, rows.astype(np.int32), a[rows, cols], low + np.tril(low, -1).T


@pytest.mark.parametrize("precision,zero", [(nq.NQG_FP64, -0.0), (nq.NQG_FP32, -0.0), (nq.NQG_FP32, -1e-60)])
@pytest.mark.parametrize("diag", [0.0, 1e-9])
@pytest.mark.parametrize("n", [2, 4, 34, 64, 66, 130, 192, 200])
def test_block(n, diag, precision, zero):
    rhs = np.random.default_rng(n).standard_normal(n)
    pivots = []
    for z in (zero, 0.0):
        p, i, x, full = _pairs(n, diag, z)
        # no perturbation of small diagonals (FP32: a floor of 1e-30), no refinement to hide a bad factor
        plan = nq.Plan(n, p, i, x, settings=nq.default_settings(precision=precision, reg_diag=0.0, req_ref_iter=0,
                                                                reg_diag_fp32=1e-30))
        assert plan.factor() == nq.NQG_OK
        sol = plan.solve(rhs)
        pivots.append(plan.timings().num_2x2)
        # 2 x 2 blocks apart from one another, each of condition below 4: a few roundings per entry
        unit = 2.0 ** -24 if precision == nq.NQG_FP32 else 2.0 ** -53
        assert np.abs(full @ sol - rhs).max() <= 64 * unit * np.abs(rhs).max()
    assert pivots[0] == pivots[1] > 0


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("n", [3, 20, 40, 90])
def test_batch(n, mixed):
    rng = np.random.default_rng(n)
    G = rng.standard_normal((n, n))
    q, b, d = rng.standard_normal(n), rng.standard_normal(2), np.full(2 * n, 0.7)
    row, col = np.tril_indices(n)
    probs = []
    for z in (-0.0, 0.0):
        H = np.where(np.eye(n, dtype=bool), np.diag(np.linspace(1e-6, 2.0, n)), z)
        A = np.where(np.arange(2)[:, None] == np.arange(n)[None, :] % 2, G[:2], z)
        C = np.full((2 * n, n), z)
        C[0::2][np.arange(n), np.arange(n)], C[1::2][np.arange(n), np.arange(n)] = 1.0, -1.0
        cr, cc = np.nonzero(np.abs(C) + (np.arange(2 * n)[:, None] % n < 3))
        probs.append((P.csc_from_coo(n, n, row, col, H[row, col]), q,
                      P.csc_from_coo(2, n, np.repeat([0, 1], n), np.tile(np.arange(n), 2), A.ravel()), 0.1 * b,
                      P.csc_from_coo(2 * n, n, cr, cc, C[cr, cc]), d))
    eps = 1e-8
    s = dict(precision=nq.NQG_FP32, refine=1, refine_tol=1e-12) if mixed else {}
    batch = nq.QPBatch(probs, settings=nq.batch_settings(eps_abs=eps, **s))
    batch.solve()
    x, _, z, st = batch.results()
    assert st[0].status == st[1].status == 1 and st[0].num_iter == st[1].num_iter
    assert (z[:2 * n] != 0).tolist() == (z[2 * n:] != 0).tolist()
    batch.close()
