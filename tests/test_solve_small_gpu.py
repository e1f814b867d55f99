"""Refined solve of small FP64 plans in one launch against the level and block
kernels, at the edges of its block classes: 32-column chunks, rows that take a
thread or a warp, columns that merge into one block, levels with more large
blocks than CTAs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
sp = pytest.importorskip("scipy.sparse")


def _dense(n, rng):
    a = rng.standard_normal((n, n))
    return a + a.T


def _bordered(nblk, w, border, rng):
    """nblk dense blocks of w columns, each coupled to all `border` last columns."""
    n = nblk * w + border
    a = np.zeros((n, n))
    for b in range(nblk):
        q = slice(b * w, (b + 1) * w)
        a[q, q] = _dense(w, rng)
        a[nblk * w :, q] = rng.standard_normal((border, w))
    a[nblk * w :, nblk * w :] = _dense(border, rng)
    return np.tril(a) + np.tril(a, -1).T


CASES = {f"dense{n}": (lambda r, n=n: _dense(n, r)) for n in (1, 2, 31, 32, 33, 64, 65, 95, 97, 128, 161)}
CASES |= {f"singles_border{m}": (lambda r, m=m: _bordered(300, 1, m, r)) for m in (1, 14, 15, 16, 17, 40)}
CASES |= {
    "blocks17x24": lambda r: _bordered(17, 24, 30, r),
    "blocks15x33": lambda r: _bordered(15, 33, 20, r),
    "blocks3x70": lambda r: _bordered(3, 70, 130, r),
    "chain": lambda r: np.diag(np.full(700, 0.1)) + np.diag(np.ones(699), 1) + np.diag(np.ones(699), -1),
}


@pytest.mark.parametrize("name", CASES)
def test_matches_level_kernels(name, monkeypatch):
    import nasoq_gb300 as nq

    rng = np.random.default_rng(5)
    full = CASES[name](rng)
    n = full.shape[0]
    low = sp.csc_matrix(np.tril(full))
    low.sort_indices()
    rhs = rng.standard_normal(n)
    xs = []
    for general in (None, "64,256", "0,0"):  # 0,0: every supernode on the block kernels' 64-column tiles
        if general:
            monkeypatch.setenv("NASOQ_GB300_SOLVE_SMALL", general)
        plan = nq.Plan(n, low.indptr, low.indices, low.data)
        plan.factor()
        before = plan.launch_count()
        xs.append(plan.solve(rhs))
        assert (plan.launch_count() - before == 1) != bool(general)
    # a refined solve is backward stable: |b - Ax| <= n eps (|A||x| + |b|), row by row at most n products
    eps = np.finfo(float).eps
    for x in xs:
        bound = n * eps * (np.abs(full) @ np.abs(x) + np.abs(rhs)).max() + 4 * eps * np.abs(rhs).max()
        assert np.abs(full @ x - rhs).max() <= bound
