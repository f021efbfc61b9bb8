"""vl_mlp_backward on FP32 arrays that start on any float, as its interface takes them: the same bits as on
arrays of the allocator's alignment."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _shifted(t):
    """The values of ``t`` 4 bytes past an 8-byte boundary."""
    big = torch.empty(t.numel() + 4, dtype=t.dtype, device=t.device)
    out = big[1:1 + t.numel()].view(t.shape)
    assert out.data_ptr() % 8 == 4
    out.copy_(t)
    return out


def _inputs(n, nout):
    from vlasov1d2v_b200.closure import IN, MLP

    rng = np.random.default_rng(n)
    X = torch.as_tensor(rng.normal(size=(n, IN)).astype(np.float32), device="cuda")
    T = torch.as_tensor(rng.normal(size=(n, nout)).astype(np.float32), device="cuda")
    return MLP(seed=3), X, T


@pytest.mark.parametrize("n,nout", [(65, 36), (257, 48)])
def test_gradients_on_any_float(cuda, n, nout):
    mlp, X, T = _inputs(n, nout)
    buf = mlp.buffers(n, X.device)
    mlp.gradients(X, T, buf)
    want = mlp.grad_w.clone(), mlp.grad_b.clone()
    mlp.grad_w, mlp.grad_b = _shifted(torch.zeros_like(mlp.grad_w)), _shifted(torch.zeros_like(mlp.grad_b))
    mlp.gradients(X, T, buf)
    assert torch.equal(mlp.grad_w, want[0]) and torch.equal(mlp.grad_b, want[1])


@pytest.mark.parametrize("n,nout", [(65, 36), (257, 48)])
def test_pre_activations_on_any_float(cuda, n, nout):
    """Z of a caller's own copy (vl_mlp_forward writes pairs; only the backward pass reads it here)."""
    from vlasov1d2v_b200 import _lib
    from vlasov1d2v_b200.closure import _stream, _vp

    mlp, X, T = _inputs(n, nout)
    buf = mlp.buffers(n, X.device)
    mlp.gradients(X, T, buf)
    want = mlp.grad_w.clone(), mlp.grad_b.clone()
    mlp.grad_w.zero_()
    mlp.grad_b.zero_()
    Z = _shifted(buf["Z"])
    _lib.call("vl_mlp_backward", _vp(buf["Y"]), _vp(T), n, nout, _vp(mlp.wf), _vp(mlp.wb), _vp(mlp.master_b),
              _vp(buf["H0"]), _vp(buf["Hh"]), _vp(Z), _vp(buf["parts"]), _vp(mlp.grad_w), _vp(mlp.grad_b), _stream())
    assert torch.equal(mlp.grad_w, want[0]) and torch.equal(mlp.grad_b, want[1])
