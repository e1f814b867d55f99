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


@pytest.mark.parametrize("rows", [4, 300])
def test_infinite_input_in_gradients(rows):
    """dL/dW of a single layer is a sum over rows of d x, an FP32 sum in which
    an infinite x gives an infinity for d != 0 and NaN for d = 0, also where d
    has few bits (labels and saturated outputs give d = +-1 / rows)."""
    sizes = (33, 66)
    rng = np.random.default_rng(rows)
    m = nq.MLP(sizes, seed=1)
    m.set_weights(np.where(rng.random(33 * 66) < 0.5, 1.0, -1.0).astype(np.float32), np.zeros(66, np.float32))
    x = rng.standard_normal((rows, 33)).astype(np.float32)
    x[1, 7], x[2, 9] = np.inf, -np.inf
    y = (rng.random((rows, 66)) < 0.5).astype(np.float32)
    w = m.get_weights()[0].reshape(66, 33).astype(np.float64)
    z = np.zeros((rows, 66))
    for k in range(33):
        z += x[:, k, None].astype(np.float64) * w[None, :, k]
    assert (m.forward(x)[1:3] == z[1:3]).all()  # +-inf
    with np.errstate(over="ignore", invalid="ignore"):
        s = 1.0 / (1.0 + np.exp(-z))
        d = (s * (2.0 * y + 1.0 - y) - 2.0 * y) / rows
        want = np.zeros((66, 33))
        for r in range(rows):
            want += d[r][:, None] * x[r].astype(np.float64)[None, :]
    _, gw, gb = m.loss_grad(x, y, pos_weight=2.0)
    gw = gw.reshape(66, 33)
    odd = ~np.isfinite(want)
    assert odd[:, [7, 9]].any() and np.isinf(want).any()
    assert np.array_equal(gw[odd], want[odd].astype(np.float32), equal_nan=True)
    # sums of `rows` FP32 terms
    assert np.abs(gw[~odd] - want[~odd]).max() <= 2.0 ** -23 * (rows + 33) * np.linalg.norm(want[~odd])
    m.close()


def test_infinite_weight():
    """A weight of infinity times an activation of few bits is an infinity (NaN
    for 0), in the logits and in the gradient of the layer below."""
    m = nq.MLP((32, 70), seed=1)
    w = np.ones((70, 32), np.float32)
    w[5, 3] = np.inf
    m.set_weights(w.ravel(), np.zeros(70, np.float32))
    x = np.ones((5, 32), np.float32)
    x[:, 3] = [1.0, -2.0, 0.0, 0.1, -np.inf]
    z = m.forward(x)
    assert np.array_equal(z[:, 5], np.array([np.inf, -np.inf, np.nan, np.inf, -np.inf], np.float32), equal_nan=True)
    assert np.isfinite(np.delete(z[:4], 5, axis=1)).all()
    m.close()

    inp, hid, out, rows = 16, 24, 70, 4
    m = nq.MLP((inp, hid, out), seed=1)
    w2 = np.ones((out, hid), np.float32)
    w2[6, 2] = w2[65, 11] = np.inf
    m.set_weights(np.concatenate([np.ones(hid * inp, np.float32), w2.ravel()]), np.zeros(hid + out, np.float32))
    x = np.full((rows, inp), 0.5, np.float32)  # every hidden unit is 8
    y = np.ones((rows, out), np.float32)
    y[:, 6] = 0.0
    assert (m.forward(x)[:, [6, 65]] == np.inf).all()
    _, gw, _ = m.loss_grad(x, y)
    g1 = gw[:hid * inp].reshape(hid, inp)
    assert (g1[2] == np.inf).all()  # dlogit 1 / rows there
    assert np.isnan(g1[11]).all()   # dlogit 0
    assert np.isfinite(np.delete(g1, [2, 11], axis=0)).all()
    m.close()
