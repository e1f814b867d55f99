"""The active-set model's tensor-core products at the edges of their tiles
(128 rows, 64 columns, 64 entries of K, rows that cannot be read 16 bytes at a
time): logits and gradients against FP64 numpy."""
import numpy as np
import pytest

import nasoq_gb300 as nq

SHAPES = [((32, 256, 256, 900), 130), ((1, 1), 1), ((7, 5, 3), 2), ((33, 63, 65), 127), ((64, 64, 64), 128),
          ((65, 129, 1), 129), ((100, 62, 130), 300), ((8, 200, 61), 513)]


def _bf16(w):
    b = np.ascontiguousarray(w, np.float32).view(np.uint32)
    return ((b + 0x7FFF + ((b >> 16) & 1)) & 0xFFFF0000).view(np.float32).astype(np.float64)


def _forward(layers, x):
    acts, bound = [x.astype(np.float64)], None
    for l, (w, b) in enumerate(layers):
        z = acts[-1] @ w.T + b
        # a chain of fan-in + 1 FP32 roundings of partial sums, each at most 2^-23 of the sum of magnitudes, and
        # what the layer before was off by
        mag = np.abs(acts[-1]) @ np.abs(w).T + np.abs(b)
        bound = (w.shape[1] + 2) * 2.0 ** -23 * mag + (0.0 if bound is None else bound @ np.abs(w).T)
        acts.append(np.maximum(z, 0.0) if l + 1 < len(layers) else z)
    return acts, bound


@pytest.mark.gpu
@pytest.mark.parametrize("sizes,rows", SHAPES)
def test_products(sizes, rows):
    rng = np.random.default_rng([rows, len(sizes)])
    m = nq.MLP(sizes, seed=5)
    w, b = m.get_weights()
    b = (0.1 * rng.standard_normal(b.shape)).astype(np.float32)
    m.set_weights(w, b)
    layers = [(_bf16(W), B.astype(np.float64)) for W, B in m.layers()]
    x = rng.standard_normal((rows, sizes[0])).astype(np.float32)
    x[0, 0] = 1e-30  # parts below the range of a BF16 one's neighbours
    y = (rng.random((rows, sizes[-1])) < 0.3).astype(np.float32)
    acts, bound = _forward(layers, x)
    z = m.forward(x)
    assert (np.abs(z - acts[-1]) <= bound).all()
    loss, gw, gb = m.loss_grad(x, y, pos_weight=3.0)
    s = 1.0 / (1.0 + np.exp(-acts[-1]))
    d = (s * (3.0 * y + 1.0 - y) - 3.0 * y) / rows
    want_w, want_b = [], []
    for l in range(len(layers) - 1, -1, -1):
        want_w.insert(0, (d.T @ acts[l]).ravel())
        want_b.insert(0, d.sum(axis=0))
        if l:
            d = (d @ layers[l][0]) * (acts[l] > 0.0)
    # sums of `rows` FP32 terms per entry, through at most three layers: 2^-23 (rows + fan) relative to the norm
    tol = 2.0 ** -23 * (rows + sum(sizes))
    want_w, want_b = np.concatenate(want_w), np.concatenate(want_b)
    assert np.linalg.norm(gw - want_w) <= tol * np.linalg.norm(want_w)
    assert np.linalg.norm(gb - want_b) <= tol * np.linalg.norm(want_b)
    m.close()


@pytest.mark.gpu
def test_infinities_and_nan_stay():
    m = nq.MLP((32, 70), seed=1)
    W, b = m.layers()[0]
    x = np.ones((3, 32), np.float32)
    x[1, 4], x[2, 5] = np.inf, np.nan
    z = m.forward(x)
    assert np.isfinite(z[0]).all()
    assert (np.isinf(z[1]) == (_bf16(W)[:, 4] != 0.0)).all() and np.isnan(z[2]).all()
    m.close()
