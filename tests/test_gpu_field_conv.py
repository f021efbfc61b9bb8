"""The field solve in its convolution form against the transform form (VLASOV1D2V_FIELD=dft, read when
a context is created) and against the oracle.

Tolerance: the two forms round the phases k x differently, by up to 2.5 pi nx eps = 6e-14 a factor at
64 elements, three factors to a term: 2e-13 of the result, ten times that as the bar."""
import numpy as np
import pytest
import torch

from helpers import rel_err
from oracle import vlasov_oracle as vo

pytestmark = pytest.mark.gpu
TOL = 2e-12


def _solve(ctx, charge):
    E = torch.empty((ctx.nx + 2, ctx.n), dtype=torch.float64, device="cuda")
    phi = torch.empty((ctx.nx, ctx.n), dtype=torch.float64, device="cuda")
    ctx.poisson(charge, E, phi)
    E1 = torch.empty_like(E)
    ctx.poisson(charge, E1)   # without phi
    assert torch.equal(E, E1)
    return E.cpu().numpy(), phi.cpu().numpy()


def _context(x, form, monkeypatch):
    from vlasov1d2v_b200.context import NativeContext

    monkeypatch.setenv("VLASOV1D2V_FIELD", form)
    return NativeContext(x=x, kappa=1.7)


@pytest.mark.parametrize("nx,n", [(1, 4), (2, 8), (3, 5), (7, 3), (16, 8), (32, 8), (33, 9), (64, 9), (64, 10), (64, 2)])
def test_convolution_matches_transform(cuda, nx, n, monkeypatch):
    from vlasov1d2v_b200.basis import Basis1D
    from vlasov1d2v_b200.grid import Grid1D

    x = Grid1D(low=-3.0, high=5.0, res=nx, basis=Basis1D(n), spectrum=True)
    rng = np.random.default_rng(nx + n)
    charge = rng.standard_normal((nx, n))
    charge -= charge.mean()
    d = torch.as_tensor(charge, device="cuda")
    E, phi = _solve(_context(x, "conv", monkeypatch), d)
    E0, phi0 = _solve(_context(x, "dft", monkeypatch), d)
    assert rel_err(E, E0) < TOL and rel_err(phi, phi0) < TOL
    c = vo.make_axis(-3.0, 5.0, nx, vo.make_basis(n), spectrum=True)
    case = vo.Case(n=n, basis=c.basis, x=c, u=None, v=None, accel=0.0, B=0.0, kappa=1.7)
    Eo, phio = vo.poisson2(charge, case)
    assert rel_err(E, Eo) < TOL and rel_err(phi, phio) < TOL


def test_other_phases_keep_the_transform(cuda, monkeypatch):
    """Phases that are not those of a uniform periodic grid take the transform form: the same bits."""
    from vlasov1d2v_b200.basis import Basis1D
    from vlasov1d2v_b200.grid import Grid1D

    x = Grid1D(low=0.0, high=2.0, res=6, basis=Basis1D(4), spectrum=True)
    x.np_dft_phase[2] *= np.exp(1e-9j)
    d = torch.as_tensor(np.random.default_rng(0).standard_normal((6, 4)), device="cuda")
    for a, b in zip(_solve(_context(x, "conv", monkeypatch), d), _solve(_context(x, "dft", monkeypatch), d)):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_steps_and_histories(cuda, precision, monkeypatch):
    """Steps with energy, dt and time histories, a final time inside a batch, and an ensemble: the two
    forms of the solve agree."""
    from vlasov1d2v_b200 import problem
    from vlasov1d2v_b200.ensemble import Ensemble

    got = {}
    for form in ("conv", "dft"):
        monkeypatch.setenv("VLASOV1D2V_FIELD", form)
        ps = [problem.build(r, n, perturbation="cos", amp=0.1, precision=precision, background_split=False,
                            batch_steps=4) for r, n in (((5, 4, 6), 5), ((9, 5, 5), 4), ((5, 4, 6), 5))]
        p = ps[0]
        p.stepper.run_steps(p.f, p.basis, p.elliptic, p.grids, p.flux, p.refs, 6)
        q = ps[1]
        q.stepper.final_time = 5.5 * float(p.stepper.dt)
        q.stepper.main_loop(q.f, q.basis, q.elliptic, q.grids, q.flux, q.refs, None)
        Ensemble(ps[2:], batch_steps=3).run_steps(6)
        got[form] = [np.concatenate([np.asarray(s.stepper.field_energy), np.asarray(s.stepper.time_array),
                                     s.elliptic.potential.get().ravel() * 1e3]) for s in ps]
    for a, b in zip(got["conv"], got["dft"]):
        assert len(a) == len(b)
        # rounding of the density (FP32 states: of the state) over the perturbation, over the steps
        assert rel_err(a, b) < (1e-11 if precision == "fp64" else 1e-5)
