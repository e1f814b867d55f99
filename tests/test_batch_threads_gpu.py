"""The batched solver's CTA sizes: every multiple of 32 up to 256 is accepted, the
ones that are no power of two included (lanes to rows and columns of a block
have to divide the CTA evenly).  H >= I, so that points whose KKT residuals are
below 1e-8 lie within 1e-8 times a few row sums of each other."""
import numpy as np
import pytest

import nasoq_gb300 as nq

from test_batch_blocks_gpu import _arrow, _box, _csc, _dense

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("threads", [32, 64, 96, 160, 192, 224, 256])
@pytest.mark.parametrize("kind", ["dense40", "dense90", "arrow"])
def test_cta_sizes_agree(kind, threads):
    rng = np.random.default_rng(7)
    H = {"dense40": lambda: _dense(40, rng), "dense90": lambda: _dense(90, rng),
         "arrow": lambda: _arrow(150, 40, rng)}[kind]()
    n = H.shape[0]
    A = rng.standard_normal((1, n)) / np.sqrt(n)
    C = _box(n)
    Hs, As, Cs = _csc(H, lower=True), _csc(A), _csc(C)
    probs = [(Hs, 3.0 * rng.standard_normal(n), As, np.zeros(1), Cs, np.full(2 * n, 0.5)) for _ in range(3)]
    xs = []
    for t in (128, threads):
        batch = nq.QPBatch(probs, eps_abs=1e-8, threads=t)
        batch.solve()
        x, _, _, st = batch.results()
        assert [s.status for s in st] == [1, 1, 1]
        xs.append(x)
    assert np.abs(xs[0] - xs[1]).max() <= 1e-6
