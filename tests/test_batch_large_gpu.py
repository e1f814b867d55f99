"""Batches whose patterns have too many columns for shared memory to hold both
vectors of the solves: they keep part of their state in global memory.  The
same problems through both kernels, and long horizons."""
import numpy as np
import pytest

import nasoq_gb300 as nq
from nasoq_gb300 import problems as P

pytestmark = pytest.mark.gpu


def _solve(qps, mixed, **kw):
    s = dict(precision=nq.NQG_FP32, refine=1, refine_tol=1e-12) if mixed else {}
    b = nq.QPBatch([(p.H, p.q, p.A, p.b, p.C, p.d) for p in qps], settings=nq.batch_settings(eps_abs=1e-8, **s, **kw))
    b.solve()
    x, y, z, st = b.results()
    smem = b.info().smem_bytes
    b.close()
    return x, y, z, st, smem


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("share", [0, 1])
def test_same_as_in_shared_memory(mixed, share, monkeypatch):
    qps = [P.qp_mpc(3, h) for h in (10, 25, 50)] + [P.qp_random_convex(5, grid=8, meq=9, mineq=53)]
    qps += [qps[1]] * 2  # two more over the same matrices
    near = _solve(qps, mixed, share_factor=share)
    monkeypatch.setenv("NASOQ_GB300_BATCH_LARGE", "1")
    far = _solve(qps, mixed, share_factor=share)
    assert far[4] < near[4]
    assert [(s.status, s.num_iter) for s in far[3]] == [(s.status, s.num_iter) for s in near[3]]
    # the bars of the reference comparison for x and z: 1e-7, FP32 factor 1e-6
    tol = 1e-6 if mixed else 1e-7
    for u, v in zip(far[:3], near[:3]):
        assert np.linalg.norm(u - v) <= tol * max(np.linalg.norm(v), 1.0)


@pytest.mark.parametrize("horizon,mixed", [(400, False), (470, False), (700, True)])
def test_long_horizons(horizon, mixed):
    qp = P.qp_mpc(1, horizon, q_scale=0.5)
    eps = 1e-8
    x, y, z, st, _ = _solve([qp], mixed)
    assert st[0].status == 1
    H = np.asarray(qp.H.x)  # diagonal
    col = np.repeat(np.arange(qp.n), np.diff(qp.A.p))
    aty = np.zeros(qp.n)
    np.add.at(aty, col, qp.A.x * y[qp.A.i])
    ax = np.zeros(qp.A.nrow)
    np.add.at(ax, qp.A.i, qp.A.x * x[col])
    tol = 2 * eps  # the solver's own bounds, with room for the rounding of the products formed here
    assert np.abs(H * x + qp.q + aty + z[0::2] - z[1::2]).max() <= tol
    assert np.abs(ax - qp.b).max() <= tol
    assert max((x - qp.d[0::2]).max(), (-x - qp.d[1::2]).max()) <= tol and z.min() >= -tol
