"""The one-launch refined solve of small FP64 plans against the level kernels on
every path of its refinement: several Krylov steps and restarts (the factor
belongs to other values than the refinement matrix, so that they are needed),
refinement alone, early ends, and hidden constraint columns.  Both do the same
steps in the same arithmetic up to the order of sums."""
import numpy as np
import pytest

import nasoq_gb300 as nq

pytestmark = pytest.mark.gpu


def _kkt(n, m, k, rng, dense):
    """Lower CSC of [H A' C'; A 0 0; C 0 0] with k constraint rows at the end, well conditioned; entry positions of C."""
    N = n + m + k
    a = np.zeros((N, N))
    h = rng.standard_normal((n, n)) / np.sqrt(n)
    a[:n, :n] = (h @ h.T if dense else np.diag(rng.uniform(0.5, 1.5, n))) + 2.0 * np.eye(n)
    if not dense:
        i = np.arange(n - 1)
        a[i + 1, i] = a[i, i + 1] = 0.4
    for r in range(m + k):
        cols = rng.choice(n, 3, replace=False) if r >= m else np.arange(r, n, m)
        a[n + r, cols] = rng.choice([-1.0, 1.0], len(cols)) / np.sqrt(len(cols)) * rng.uniform(0.7, 1.0, len(cols))
    low = np.tril(a)
    rows, cols = np.nonzero((low != 0) | np.eye(N, dtype=bool))
    order = np.lexsort((rows, cols))
    rows, cols = rows[order], cols[order]
    ptr = np.concatenate([[0], np.cumsum(np.bincount(cols, minlength=N))]).astype(np.int32)
    extra = np.zeros(N, np.int32)
    extra[n + m:] = 1
    return N, ptr, rows.astype(np.int32), cols, low[rows, cols], extra


def _both(monkeypatch, make):
    """make() with the one-launch solve, then with the level kernels; and the factor's element growth."""
    out = []
    for general in (False, True):
        if general:
            monkeypatch.setenv("NASOQ_GB300_SOLVE_SMALL", "64,256")
        plan, run = make()
        before = plan.launch_count()
        x = run()
        assert (plan.launch_count() - before == 1) != general
        out.append((x, plan.timings().num_ref_iter))
    return out, np.abs(plan.factor_arrays()[0]).max()


def _agree(out, growth, kappa):
    x, xg = out[0][0], out[1][0]
    # the bar of the comparisons with the reference's solutions: pivots of 1e-9 (the regularization) are taken
    # inside their supernode, the growth of up to 1e9 amplifies the rounding of either solve
    tol = max(1e-9, 1e-14 * kappa, 1e-15 * growth)
    assert np.isfinite(x).all() and np.linalg.norm(x - xg) <= tol * np.linalg.norm(xg)


@pytest.mark.parametrize("dense", [False, True])
@pytest.mark.parametrize("refine_only", [False, True])
@pytest.mark.parametrize("restarts,steps,tol", [(1, 1, 1e-15), (2, 2, 1e-15), (1, 7, 1e-15), (3, 5, 1e-15), (1, 16, 1e-6),
                                                (4, 3, 1e-6), (3, 16, 1e6), (0, 4, 1e-15), (2, 0, 1e-15)])
def test_refinement(restarts, steps, tol, refine_only, dense, monkeypatch):
    rng = np.random.default_rng([restarts, steps, dense])
    N, p, i, cols, v, extra = _kkt(90 if dense else 300, 12, 40, rng, dense)
    off = i != cols
    other = v.copy()
    other[off] *= 1.0 + 0.2 * rng.uniform(-1.0, 1.0, off.sum())  # what the refinement sees
    rhs = rng.standard_normal(N)

    def make():
        plan = nq.Plan(N, p, i, v, extra_cols=extra, settings=nq.default_settings(
            req_ref_iter=restarts, max_inner_iter=steps, tol_abs=tol, tol_rel=tol, reg_diag=1e-9))
        assert plan.factor() == nq.NQG_OK
        for part in np.array_split(np.nonzero(off)[0], 1 + off.sum() // N):  # at most N entries a call
            plan.edit_values(part, other[part])
        return plan, lambda: (plan.refine_only if refine_only else plan.solve)(rhs)

    out, growth = _both(monkeypatch, make)
    full = np.zeros((N, N))
    full[i, cols] = v
    full = full + np.tril(full, -1).T
    _agree(out, growth, np.linalg.cond(full))
    # with hidden constraints the last step's residual is at rounding level, here it is not
    assert out[0][1] == out[1][1]
    if tol == 1e6:  # the first residual is below it
        assert out[0][1] == 0
    elif tol == 1e-15:
        assert out[0][1] == restarts * steps


@pytest.mark.parametrize("dense", [False, True])
@pytest.mark.parametrize("share", [0.0, 0.3, 1.0])
def test_hidden_constraints(share, dense, monkeypatch):
    rng = np.random.default_rng([int(10 * share), dense])
    n, m, k = 90 if dense else 300, 12, 60
    N, p, i, cols, v, extra = _kkt(n, m, k, rng, dense)
    hidden = np.zeros(N, bool)
    hidden[n + m:] = rng.random(k) < share
    v = np.where(hidden[i] & (i != cols), 0.0, v)
    rhs = np.where(hidden, 0.0, rng.standard_normal(N))

    def make():
        plan = nq.Plan(N, p, i, v, extra_cols=extra, settings=nq.default_settings(
            req_ref_iter=2, max_inner_iter=3, reg_diag=1e-9))
        s = plan.symbolic
        col = hidden[np.asarray(s.perm)[:N]]
        sup = np.asarray(s.super)
        single = np.diff(sup) == 1
        visible = ~(col[sup[:-1]] & single)
        assert (~visible).sum() == hidden.sum()  # constraint columns are supernodes of their own
        assert plan.factor() == nq.NQG_OK
        plan.set_visibility(visible.astype(np.uint8), col.astype(np.uint8))
        return plan, lambda: plan.solve(rhs)

    out, growth = _both(monkeypatch, make)
    x = out[0][0]
    full = np.zeros((N, N))
    full[i, cols] = v
    full = full + np.tril(full, -1).T
    see = ~hidden
    _agree(out, growth, np.linalg.cond(full[np.ix_(see, see)]))
    assert (x[hidden] == 0.0).all()
    bound = N * np.finfo(float).eps * (np.abs(full) @ np.abs(x) + np.abs(rhs)).max()
    assert np.abs(full @ x - rhs)[see].max() <= bound
