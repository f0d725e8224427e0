"""The rows at the edges of a training step: the first and last row of every split and the rows of
the last tile carry nearly all of the loss and its gradient, so that one of them lost, taken twice
or taken from the wrong place moves both past the bounds."""
import numpy as np
import pytest

import rfdem
from oracle import mlp_ref

pytestmark = pytest.mark.gpu


def edge_rows(rows):
    """First and last row of every split (whole 64-row chunks, one split per 2048 rows up to 64)
    and the rows of the last 128-row tile."""
    chunks = (rows + 127) // 128 * 2
    splits = max(1, min(64, chunks // 32))
    size = (chunks + splits - 1) // splits * 64
    first = np.arange(0, rows, size)
    last = np.minimum(first + size, rows) - 1
    tail = np.arange((rows - 1) // 128 * 128, rows)
    return np.unique(np.concatenate([first, last, tail]))


def heavy_data(rows):
    """Features, and targets of which the edge rows' are about 1e3, the others' 0.5."""
    rng = np.random.default_rng(rows + 23)
    X = mlp_ref.bf16(rng.standard_normal((rows, 64)))
    T = (0.5 * np.tanh(X[:, :6] + 0.3 * X[:, 6:12])).astype(np.float32)
    edge = edge_rows(rows)
    T[edge] = (1e3 * rng.choice([-1.0, 1.0], (edge.size, 6)) * rng.uniform(0.8, 1.2, (edge.size, 6))).astype(np.float32)
    return X, T


# One edge row is at least 5e-3 of the loss and 3.6 % of the norm of every gradient. The bound of the
# loss is 1e-3 (the outputs' BF16 error is 1e-5 of such a target), of the gradients the 2 % of the
# other MLP tests.
@pytest.mark.parametrize("rows", [129, 2049, 148 * 128 + 1, 2 * 148 * 128 + 65, 133000, 133057])
def test_mlp_training_edge_rows(cuda, rows):
    X, T = heavy_data(rows)
    m = rfdem.MLP(seed=rows)
    ws = m.weights()
    loss = m.train_step(cuda.from_numpy(X).to(cuda.bfloat16).cuda(), cuda.from_numpy(T).cuda(), rows, 0.0)
    loss_ref, g_ref = mlp_ref.backward(ws, X, T)
    assert abs(loss - loss_ref) <= 1e-3 * loss_ref, (loss, loss_ref)
    for l, (a, b) in enumerate(zip(m.grads(), g_ref)):
        for u, v in zip(a, b):
            n = np.linalg.norm(v)
            assert np.linalg.norm(u - v) <= 2e-2 * n, (l, np.linalg.norm(u - v) / n)
    m.close()
