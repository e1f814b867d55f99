"""FP64 block-first panels against the column-by-column kernel: the same
multiply-adds in the same order, so the same factor, at widths around the panel,
the 8-column step and the 32 rows of a CTA; and systems whose pivots stop them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
sp = pytest.importorskip("scipy.sparse")


def _factor(monkeypatch, a, general, nb):
    import nasoq_gb300 as nq

    monkeypatch.setenv("NASOQ_GB300_WIDE_MIN", "12")
    monkeypatch.setenv("NASOQ_GB300_WIDE_NB", str(nb))
    if general:
        monkeypatch.setenv("NASOQ_GB300_PANEL", "general")
    else:
        monkeypatch.delenv("NASOQ_GB300_PANEL", raising=False)
    low = sp.csc_matrix(np.tril(np.ones_like(a)))  # full lower pattern: zeros on the diagonal stay entries
    low.sort_indices()
    low.data = a[low.indices, np.repeat(np.arange(a.shape[0]), np.diff(low.indptr))]
    plan = nq.Plan(a.shape[0], low.indptr, low.indices, low.data)
    plan.factor()
    return plan


@pytest.mark.parametrize("nb", [5, 8, 13, 64])
@pytest.mark.parametrize("n", [13, 63, 64, 65, 96, 97, 161, 200])
def test_same_factor_without_pivoting(n, nb, monkeypatch):
    rng = np.random.default_rng(n)
    r = rng.standard_normal((n, n))
    a = r @ r.T / n + 4 * np.eye(n)
    h = n // 2
    a[h:, h:] *= -1.0  # quasi-definite; the diagonal dominates enough for 1 x 1 pivots
    a[h:, :h] *= 0.1
    a[:h, h:] *= 0.1
    got = _factor(monkeypatch, a, False, nb).factor_arrays()
    want = _factor(monkeypatch, a, True, nb).factor_arrays()
    got, want = (list(f.values()) if isinstance(f, dict) else list(f) for f in (got, want))
    for g, w in zip(got, want):
        assert np.array_equal(np.asarray(g), np.asarray(w))


@pytest.mark.parametrize("nb", [8, 64])
@pytest.mark.parametrize("n", [64, 129, 200])
def test_pivots_stop_the_panel(n, nb, monkeypatch):
    rng = np.random.default_rng(n)
    r = rng.standard_normal((n, n))
    a = r + r.T
    np.fill_diagonal(a, 0.0)
    rhs = rng.standard_normal(n)
    x = _factor(monkeypatch, a, False, nb).solve(rhs)
    eps = np.finfo(float).eps
    assert np.abs(a @ x - rhs).max() <= n * eps * (np.abs(a) @ np.abs(x) + np.abs(rhs)).max()
