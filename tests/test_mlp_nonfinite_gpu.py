"""Infinities and NaN through the active-set model's products: what is not
finite in plain floating-point arithmetic comes out the same."""
import numpy as np
import pytest

import nasoq_gb300 as nq

pytestmark = pytest.mark.gpu


def _nan(bits):
    return np.array([bits], np.uint32).view(np.float32)[0]


@pytest.mark.parametrize("bits", [0x7F800001, 0xFF80ABCD, 0x7FC00000, 0x7FFFFFFF, 0xFFFFFFFF])
def test_nan_of_any_payload_stays(bits):
    m = nq.MLP((32, 70), seed=1)
    x = np.ones((3, 32), np.float32)
    x[1, 4] = _nan(bits)
    assert x.view(np.uint32)[1, 4] == bits
    z = m.forward(x)
    assert np.isfinite(z[[0, 2]]).all() and np.isnan(z[1]).all()
    _, gw, _ = m.loss_grad(x, np.zeros((3, 70), np.float32))
    assert np.isnan(gw).all()  # the row's logits, and with them its share of every gradient
    m.close()
