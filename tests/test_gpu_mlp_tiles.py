"""The fused MLP kernels at the edges of their tiling (128-row tiles, up to 64 splits): row
counts around a tile and a split (133000: the last split would be padding alone), unaligned features, every output
stride and column count, the residual mode; against the CPU restatement (oracle/mlp_ref.py)
with the bound of the existing MLP test (BF16 roundings: 2 % of the largest output, 2 %
relative norm of the gradients)."""
import numpy as np
import pytest

import rfdem
from oracle import mlp_ref

pytestmark = pytest.mark.gpu


def _data(torch, rows, offset=0):
    rng = np.random.default_rng(rows + 17)
    X = rng.standard_normal((rows, 64)).astype(np.float32)
    T = (0.5 * np.tanh(X[:, :6] + 0.3 * X[:, 6:12]) + 0.1 * X[:, 12:18]).astype(np.float32)
    buf = torch.zeros(rows * 64 + offset, dtype=torch.bfloat16, device="cuda")
    Xb = buf[offset:].view(rows, 64)
    Xb.copy_(torch.from_numpy(X))
    return buf, Xb, torch.from_numpy(T).cuda(), Xb.float().cpu().numpy().astype(np.float64), T


def _check(torch, rows, offset=0, residual=False):
    m = rfdem.MLP(seed=rows)
    m.set_residual(residual)
    ws = m.weights()
    keep, Xb, Td, X, T = _data(torch, rows, offset)
    loss = m.train_step(Xb, Td, rows, 0.0)
    loss_ref, g_ref = mlp_ref.backward(ws, X, T - X[:, :6] if residual else T)
    assert abs(loss - loss_ref) <= 1e-2 * loss_ref
    for l, (a, b) in enumerate(zip(m.grads(), g_ref)):
        for u, v in zip(a, b):
            n = np.linalg.norm(v)
            assert np.linalg.norm(u - v) <= 2e-2 * n, (rows, l, np.linalg.norm(u - v) / max(n, 1e-300))
    if offset == 0:
        Y = torch.full((rows + 1, 16), 7.0, device="cuda")
        m.forward(Xb, rows, Y)
        torch.cuda.synchronize()
        y_ref, _ = mlp_ref.forward(ws, X)
        if residual:
            y_ref[:, :6] += X[:, :6]
        y = Y[:rows].cpu().numpy()
        assert np.max(np.abs(y[:, :6] - y_ref[:, :6])) <= 2e-2 * (np.abs(y_ref[:, :6]).max() + 1e-6)
        assert np.all(Y[rows].cpu().numpy() == 7.0)
    m.close()


@pytest.mark.parametrize("rows", [1, 127, 128, 129, 148 * 128, 148 * 128 + 1, 2 * 148 * 128 + 65, 4 * 148 * 128 + 3,
                                  133000, 133057])
def test_mlp_row_counts(cuda, rows):
    _check(cuda, rows)


def test_mlp_residual_and_unaligned_features(cuda):
    _check(cuda, 700, residual=True)
    _check(cuda, 700, offset=3)
    with pytest.raises(rfdem.RFError):
        m = rfdem.MLP()
        buf, Xb, _, _, _ = _data(cuda, 10, 3)
        m.forward(Xb, 10, cuda.zeros(10, 16, device="cuda"))


@pytest.mark.parametrize("ldy,ncols,offset", [(6, 6, 0), (16, 6, 0), (17, 16, 0), (16, 16, 1), (1, 1, 0), (20, 16, 0)])
def test_mlp_output_strides(cuda, ldy, ncols, offset):
    rows = 333
    m = rfdem.MLP(seed=5)
    _, Xb, _, _, _ = _data(cuda, rows)
    ref = cuda.zeros(rows, 16, device="cuda")
    m.forward(Xb, rows, ref)
    buf = cuda.full((rows * ldy + offset + 32,), 7.0, device="cuda")
    m.forward(Xb, rows, buf[offset:], ldy=ldy, ncols=ncols)
    cuda.cuda.synchronize()
    want = cuda.full_like(buf, 7.0)
    want[offset:offset + rows * ldy].view(rows, ldy)[:, :ncols] = ref[:, :ncols]
    assert cuda.equal(buf, want)
    m.close()
