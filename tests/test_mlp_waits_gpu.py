"""A tensor-core wait of the active-set model that gives up (the limit set so
that every one does): the call that waits returns NQG_ERR_TIMEOUT, a forward on
a caller's stream reports to nqg_mlp_stream_status and to no other call, its
tiles are NaN, and the model works again with the default limit."""
import numpy as np
import pytest

import nasoq_gb300 as nq

pytestmark = pytest.mark.gpu


def _timeout():
    return pytest.raises(nq.NasoqError, match=r"\(-5\)")


@pytest.mark.parametrize("sizes,rows", [((32, 70), 130), ((200, 64, 900), 2000)])
def test_reports(sizes, rows):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(rows)
    m = nq.MLP(sizes, seed=2)
    x = rng.standard_normal((rows, sizes[0])).astype(np.float32)
    y = np.zeros((rows, sizes[-1]), np.float32)
    want = m.forward(x)
    stream = torch.cuda.Stream()
    dx, dz = torch.from_numpy(x).cuda(), torch.zeros(want.shape, device="cuda")
    torch.cuda.synchronize()

    def on_stream():
        m.forward_device(rows, dx.data_ptr(), dz.data_ptr(), stream.cuda_stream)
        stream.synchronize()
        return dz.cpu().numpy()

    m.set_wait_limit(-1)
    with _timeout():
        m.forward(x)
    with _timeout():
        m.loss_grad(x, y)
    assert np.isnan(on_stream()).all()
    m.set_wait_limit(0)
    assert np.array_equal(m.forward(x), want)  # not this call's failure
    with _timeout():
        m.check_stream()
    m.check_stream()  # reported once
    assert np.array_equal(on_stream(), want)
    m.check_stream()
    m.loss_grad(x, y)
    m.close()
