"""Two batches alive at once, the second with less shared memory than the first:
both still launch, in either order, through the graph and without it."""
import numpy as np
import pytest

import nasoq_gb300 as nq

from test_batch_blocks_gpu import _box, _csc, _dense

pytestmark = pytest.mark.gpu


def _batch(n, graph):
    rng = np.random.default_rng(n)
    H, C = _dense(n, rng), _box(n)
    A = rng.standard_normal((1, n)) / np.sqrt(n)
    prob = (_csc(H, lower=True), 3.0 * rng.standard_normal(n), _csc(A), np.zeros(1), _csc(C), np.full(2 * n, 0.5))
    return nq.QPBatch([prob], eps_abs=1e-8, use_graph=graph)


@pytest.mark.parametrize("graph", [0, 1])
def test_larger_batch_still_launches(graph):
    large, small = _batch(90, graph), _batch(5, graph)
    for b in (small, large, small, large):
        b.solve()
        assert b.results()[3][0].status == 1
