"""The moment and the scalar kernels at the edges of their splits: shares of a velocity plane that are
empty, ragged or one column, one x element, and the most nodes the field takes.

Tolerance: a thread adds n^2 terms a column over at most nu nv n / 8 columns in working order, the rest is
compensated: 300 eps of the sum of magnitudes covers the sizes here.  The energy sums at most three terms a
thread: 16 eps."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
EPS = 2.3e-16


def _axis(res, n, spectrum=False, low=-2.0, high=3.0):
    from vlasov1d2v_b200.basis import Basis1D
    from vlasov1d2v_b200.grid import Grid1D

    return Grid1D(low=low, high=high, res=res, basis=Basis1D(n), spectrum=spectrum)


@pytest.mark.parametrize("res,n", [((1, 1, 1), 2), ((1, 1, 1), 10), ((3, 1, 7), 5), ((2, 5, 1), 9), ((1, 9, 11), 8),
                                   ((60, 2, 3), 3), ((5, 13, 17), 7), ((4, 40, 3), 6), ((2, 33, 31), 2)])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_moment(cuda, res, n, precision):
    from vlasov1d2v_b200.context import NativeContext

    x, u, v = _axis(res[0], n, True), _axis(res[1], n), _axis(res[2], n)
    ctx = NativeContext(x=x, u=u, v=v, precision=precision)
    rng = np.random.default_rng(n + res[1])
    shape = (res[0] + 2, n, res[1] + 2, n, res[2] + 2, n)
    f = rng.standard_normal(shape).astype(np.float64 if precision == "fp64" else np.float32)
    rho = torch.empty((res[0], n), dtype=torch.float64, device="cuda")
    ctx.moment(torch.as_tensor(f, device="cuda"), rho)
    w = _weights(n)
    inner = f[1:-1, :, 1:-1, :, 1:-1, :].astype(np.longdouble)
    scale = np.longdouble(u.dx) * np.longdouble(v.dx) / 4
    want = np.einsum("eiajbk,j,k->ei", inner, w, w) * scale
    size = np.einsum("eiajbk,j,k->ei", np.abs(inner), w, w) * scale
    assert np.all(np.abs(rho.cpu().numpy() - want) <= 300 * EPS * size)


def _weights(n):
    """Lobatto weights from the Legendre polynomial at the nodes."""
    from vlasov1d2v_b200.basis import Basis1D

    return np.asarray(Basis1D(n).weights, dtype=np.longdouble)


@pytest.mark.parametrize("nx,n", [(1, 2), (1, 3), (7, 5), (29, 9), (64, 10), (64, 4)])
def test_field_energy(cuda, nx, n):
    from vlasov1d2v_b200.context import NativeContext

    x = _axis(nx, n, True)
    ctx = NativeContext(x=x, accel=-0.7, bfield=1.3, courant=0.1)
    rng = np.random.default_rng(nx)
    E = rng.standard_normal((nx + 2, n))
    out = torch.empty(1, dtype=torch.float64, device="cuda")
    dE = torch.as_tensor(E, device="cuda")
    ctx.field_energy(dE, out)
    want = 0.5 * np.sum(_weights(n) * E[1:-1].astype(np.longdouble) ** 2)
    assert abs(out.item() - float(want)) <= 16 * EPS * float(want)
    first = out.item()
    E[0, 0] = 1e6    # ghost rows do not count
    ctx.field_energy(torch.as_tensor(E, device="cuda"), out)
    assert out.item() == first
    for bad in (np.inf, np.nan):
        E[1, 0] = bad
        ctx.field_energy(torch.as_tensor(E, device="cuda"), out)
        assert not np.isfinite(out.item())
