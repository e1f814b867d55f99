"""The batched solver at the edges of its block shapes: dense Hessians around
the widths where a supernode changes hands (a thread, a warp, the CTA, two
rows per lane, the general block), and arrow Hessians around the number of
single columns from which their targets gather and the rows from which a
column counts as long.  Checked by the KKT conditions of the given data."""
import numpy as np
import pytest

import nasoq_gb300 as nq
from nasoq_gb300 import problems as P


def _csc(M, lower=False):
    r, c = np.nonzero(np.tril(M) if lower else M)
    return P.csc_from_coo(M.shape[0], M.shape[1], r, c, M[r, c])


def _dense(n, rng):
    G = rng.standard_normal((n, n))
    return G @ G.T / n + np.eye(n)


def _arrow(cols, hub, rng):
    """`cols` variables of their own, each coupled to all of the `hub` ones."""
    n = cols + hub
    H = np.zeros((n, n))
    H[np.arange(cols), np.arange(cols)] = rng.uniform(2.0, 4.0, cols)
    H[cols:, :cols] = rng.uniform(-1.0, 1.0, (hub, cols)) / np.sqrt(cols)
    H[:cols, cols:] = H[cols:, :cols].T
    H[cols:, cols:] = _dense(hub, rng) + 2.0 * np.eye(hub)
    return H


def _box(n):
    C = np.zeros((2 * n, n))
    C[0::2][np.arange(n), np.arange(n)] = 1.0
    C[1::2][np.arange(n), np.arange(n)] = -1.0
    return C


SHAPES = [("dense", n, 0) for n in (2, 3, 4, 5, 15, 16, 17, 31, 32, 33, 63, 64, 65, 90)] + \
         [("arrow", k, 6) for k in (8, 31, 32, 33, 63, 64, 65, 200)] + [("arrow", 40, h) for h in (30, 31, 32, 40)]


@pytest.mark.gpu
@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("kind,size,hub", SHAPES)
def test_block_shapes(kind, size, hub, mixed):
    rng = np.random.default_rng([size, hub])
    H = _dense(size, rng) if kind == "dense" else _arrow(size, hub, rng)
    n = H.shape[0]
    A = rng.standard_normal((1, n)) / np.sqrt(n)
    C = _box(n)
    eps = 1e-8
    Hs, As, Cs = _csc(H, lower=True), _csc(A), _csc(C)
    # two problems over the same matrices (one shared factorization) and one over others
    H3 = H + np.diag(rng.uniform(0.0, 0.1, n))
    probs, dense = [], []
    for k, (Hk, Mk) in enumerate([(Hs, H), (Hs, H), (_csc(H3, lower=True), H3)]):
        q = 3.0 * rng.standard_normal(n)
        x0 = rng.uniform(-0.3, 0.3, n)
        b, d = A @ x0, np.full(2 * n, 0.5)
        probs.append((Hk, q, As, b, Cs, d))
        dense.append((Mk, q, b, d))
    s = dict(precision=nq.NQG_FP32, refine=1, refine_tol=1e-12) if mixed else {}
    batch = nq.QPBatch(probs, settings=nq.batch_settings(eps_abs=eps, **s))
    batch.solve()
    for i, (M, q, b, d) in enumerate(dense):
        x, y, z, act, res = batch.result(i)
        assert res.status == 1, f"problem {i}: status {res.status}"
        # the solver's own bounds (eps_abs on each norm), with room for the rounding of the products formed here
        tol = 2 * eps
        assert np.abs(M @ x + q + A.T @ y + C.T @ z).max() <= tol
        assert np.abs(A @ x - b).max() <= tol and (C @ x - d).max() <= tol
        assert z.min() >= -tol and np.abs(z * (C @ x - d)).max() <= tol * (1.0 + z.max())
    batch.close()
