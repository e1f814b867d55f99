"""MPC problems whose active sets bring an eigenvalue of the constraints' Schur
complement near the diagonal floor of the FP32 factor: with a floor of the
wrong sign the preconditioner is close to singular there and the refinement
stops short.  Many copies of each, since the factorization's sums (and with
them which copy fails) vary between runs."""
import numpy as np
import pytest

import nasoq_gb300 as nq
from nasoq_gb300 import problems as P

# plant, horizon, and where its linear term's noise lies in the stream of its seed
HARD = [(2700309, 31, 27, 110313), (5300616, 76, 53, 223911), (6600736, 85, 66, 264834), (5901102, 47, 59, 450648)]


@pytest.mark.gpu
@pytest.mark.parametrize("plant,horizon,seed,offset", HARD)
def test_every_copy_is_solved(plant, horizon, seed, offset):
    qp = P.qp_mpc(plant, horizon)
    noise = np.random.default_rng([seed, 5]).standard_normal(offset + qp.n)[offset:]
    prob = (qp.H, qp.q * (1.0 + 0.05 * noise), qp.A, qp.b, qp.C, qp.d)
    eps = 1e-8
    exact = nq.QPBatch([prob], settings=nq.batch_settings(eps_abs=eps))
    exact.solve()
    xr, _, _, st = exact.results()
    assert st[0].status == 1
    copies = 64
    batch = nq.QPBatch([prob] * copies, settings=nq.batch_settings(eps_abs=eps, precision=nq.NQG_FP32, refine=1,
                                                                   refine_tol=1e-10, share_factor=0))
    batch.solve()
    x, _, _, st = batch.results()
    assert [s.status for s in st] == [1] * copies
    # two points on the same active set whose Lagrangian residuals are within eps in each entry:
    # |dx| <= |residuals' difference| / lambda_min(H), and H is diagonal, 0.1 at least
    assert np.linalg.norm(x.reshape(copies, -1) - xr, axis=1).max() <= 2 * eps * np.sqrt(qp.n) / 0.1
    batch.close()
    exact.close()
