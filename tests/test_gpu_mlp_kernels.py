"""The closure network's forward, backpropagation and gradient kernels at the sizes where their tiles
(32 samples), summation blocks (64) and stages (256) end, against the CPU oracle.

Tolerance: the oracle has the kernels' bf16 roundings, so what differs is FP32 summation (2^-24 a term,
a few hundred terms: 1e-5) and activations that this moves over a bf16 rounding boundary (2^-9 of one
activation, about one in 2^9 of them: 2^-9 2^-4.5 = 1e-4 of a norm); 1e-3 keeps a tenfold margin."""
import numpy as np
import pytest
import torch

from oracle import mlp_oracle as mo
from test_gpu_closure import _weights

pytestmark = pytest.mark.gpu


def _data(n, nout):
    rng = np.random.default_rng(n)
    X = rng.normal(size=(n, mo.IN)).astype(np.float32)
    T = rng.normal(size=(n, nout)).astype(np.float32)
    return X, T


@pytest.mark.parametrize("nout", [36, 48, 1])
@pytest.mark.parametrize("n", [1, 31, 33, 64, 65, 255, 257, 1000])
def test_edges_against_oracle(cuda, n, nout):
    from vlasov1d2v_b200.closure import MLP

    mlp = MLP(seed=n)
    X, T = _data(n, nout)
    Xd, Td = torch.as_tensor(X, device="cuda"), torch.as_tensor(T, device="cuda")
    buf = mlp.buffers(n, Xd.device)
    Y = mlp.gradients(Xd, Td, buf)
    assert torch.equal(Y, mlp.forward(Xd))   # the inference form
    W, b = _weights(mlp)
    Yo, H, Z = mo.forward(X, W, b)
    Y = Y.cpu().numpy().astype(np.float64)
    assert np.linalg.norm(Y - Yo) < 1e-3 * np.linalg.norm(Yo)
    dW, db = mo.backward(Y, T.astype(np.float64), W, H, Z, nout)
    off = 0
    for l, (_, m) in enumerate(mlp.LAYERS):
        g = mlp.layer_views(mlp.grad_w)[l].cpu().numpy()
        gb = mlp.grad_b[off:off + m].cpu().numpy()
        off += m
        assert np.linalg.norm(g - dW[l]) < 1e-3 * np.linalg.norm(dW[l]), l
        assert np.linalg.norm(gb - db[l]) < 1e-3 * np.linalg.norm(db[l]), l


def test_buffers_off_16_byte_boundaries(cuda):
    """Layer inputs and scratch 4 bytes past a 16-byte boundary: the same bits."""
    from vlasov1d2v_b200.closure import MLP

    n, nout = 129, 36
    X, T = (torch.as_tensor(a, device="cuda") for a in _data(n, nout))
    got = []
    for shift in (0, 1):
        mlp = MLP(seed=5)
        buf = mlp.buffers(n, X.device)
        for key in ("H0", "Hh", "parts"):
            t = buf[key]
            per = 2 * shift if t.dtype == torch.bfloat16 else shift
            big = torch.empty(t.numel() + 8, dtype=t.dtype, device="cuda")
            buf[key] = big[per:per + t.numel()].view(t.shape)
        mlp.gradients(X, T, buf)
        got.append((mlp.grad_w.clone(), mlp.grad_b.clone()))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
