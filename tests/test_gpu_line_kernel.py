"""The line-form stage kernel: every order, both precisions, odd sizes (rows of any alignment, ragged
last v tiles, one element per axis), all stage kinds, direction weights, both x halos, the background
split and the moment partials, against the oracle and the generic forms.

Tolerance: a value is a sum of about 3 n + 9 products of size |D| |f| with an error of eps each; the
results are compared with their largest value, which is at least the largest |D| |f|: 3 n + 9 < 40
eps, 1e-14 in FP64 and 5e-6 in FP32."""
import numpy as np
import pytest
import torch

from helpers import INNER, rel_err
from oracle import vlasov_oracle as vo

pytestmark = pytest.mark.gpu
TOL = {"fp64": 1e-14, "fp32": 5e-6}
DT = {"fp64": torch.float64, "fp32": torch.float32}


def _context(p, precision, courant=0.05):
    from vlasov1d2v_b200.context import get_context

    return get_context(p.grids, precision=precision, accel=p.refs.electron_acceleration_multiplier,
                       bfield=p.elliptic.magnetic_field, kappa=p.elliptic.poisson_coefficient, courant=courant)


def _inputs(shape, n, res, precision):
    rng = np.random.default_rng(n + 31 * res[2])
    npd = np.float64 if precision == "fp64" else np.float32
    f, fn = (rng.standard_normal(shape).astype(npd).astype(np.float64) for _ in range(2))
    E = rng.standard_normal((res[0] + 2, n))
    dev = [torch.as_tensor(a, dtype=DT[precision], device="cuda") for a in (f, fn)]
    return f, fn, E, dev[0], dev[1], torch.as_tensor(E, device="cuda")


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("res", [(1, 1, 1), (2, 3, 5), (3, 2, 33)])
@pytest.mark.parametrize("n", range(2, 11))
def test_stages_and_rhs(cuda, n, res, precision, monkeypatch):
    from vlasov1d2v_b200 import _lib, problem

    monkeypatch.setenv("VLASOV1D2V_STAGE_KERNEL", "line")
    p = problem.build(res, n, perturbation=None, precision=precision, background_split=False)
    ctx = _context(p, precision)
    c = vo.make_case(*res, n)
    f, fn, E, tf, tfn, tE = _inputs(c.shape, n, res, precision)
    out = torch.zeros_like(tf)
    ctx.rhs(tf, tE, out, xhalo=_lib.VL_XHALO_GHOST)
    got = out.cpu().numpy().astype(np.float64)
    assert rel_err(got[INNER], vo.rhs(f, E, c)[INNER]) < TOL[precision]
    got[INNER] = 0.0
    assert not got.any()   # the interior only
    f[0], f[-1] = f[-2], f[1]
    R = vo.rhs(f, E, c)
    dt = 0.0071
    tdt = torch.tensor([dt], dtype=torch.float64, device="cuda")
    for stage, want in ((0, f + dt * R), (1, 0.75 * fn + 0.25 * f + (0.25 * dt) * R),
                        (2, fn / 3 + (2 / 3) * f + ((2 / 3) * dt) * R)):
        parts = torch.zeros_like(ctx.workspace)
        o = torch.zeros_like(tf) if stage < 2 else tfn.clone()   # the last stage writes over f^n
        ctx.rk_stage(stage, tf, (o if stage == 2 else tfn) if stage else None, o, tE, tdt,
                     xhalo=_lib.VL_XHALO_PERIODIC, partials=parts)
        got = o.cpu().numpy().astype(np.float64)
        assert rel_err(got[INNER], want[INNER]) < TOL[precision], stage
        # the partials of all CTAs add up to the moment of what was stored
        rho = np.tensordot(got[INNER], c.qw, axes=([2, 3, 4, 5], [0, 1, 2, 3]))
        size = np.tensordot(np.abs(got[INNER]), c.qw, axes=([2, 3, 4, 5], [0, 1, 2, 3]))
        total = parts.view(torch.float64).cpu().numpy()
        total = total[:total.size // (res[0] * n) * (res[0] * n)].sum()
        assert abs(total - rho.sum()) < (1e-13 if precision == "fp64" else 1e-6) * size.sum()


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("n", [2, 3, 5, 7, 9])
def test_default_route_matches_the_generic_forms(cuda, n, precision, monkeypatch):
    """Where the line form is the default: direction weights and both halos against the generic
    (FP64) and register-pencil (FP32) kernels."""
    from vlasov1d2v_b200 import _lib, problem

    res = (2, 3, 5)
    got = []
    for form in (None, "gen" if precision == "fp64" else "pencil"):
        monkeypatch.delenv("VLASOV1D2V_STAGE_KERNEL", raising=False)
        if form:
            monkeypatch.setenv("VLASOV1D2V_STAGE_KERNEL", form)
        p = problem.build(res, n, perturbation=None, precision=precision, background_split=False)
        ctx = _context(p, precision)
        _, _, _, tf, _, tE = _inputs(tuple(ctx.state_shape), n, res, precision)
        for w in ((1.0, 0.0, 0.0), (0.0, 1.0, 0.0), (0.0, 0.0, 1.0), (0.5, -2.0, 3.0)):
            for halo in (_lib.VL_XHALO_GHOST, _lib.VL_XHALO_PERIODIC):
                out = torch.zeros_like(tf)
                ctx.rhs_weighted(tf, tE, out, w, xhalo=halo)
                got.append(out.double().cpu().numpy())
    half = len(got) // 2
    for a, b in zip(got[:half], got[half:]):
        assert rel_err(a, b) < TOL[precision]


@pytest.mark.parametrize("n,res", [(3, (2, 3, 4)), (5, (3, 2, 7)), (7, (2, 5, 6)), (9, (2, 4, 3))])
def test_background_split_steps(cuda, n, res, monkeypatch):
    """Steps of the FP32 mixed form (background tables) against the register-pencil kernel."""
    from vlasov1d2v_b200 import problem

    got = []
    for form in (None, "pencil"):
        monkeypatch.delenv("VLASOV1D2V_STAGE_KERNEL", raising=False)
        if form:
            monkeypatch.setenv("VLASOV1D2V_STAGE_KERNEL", form)
        p = problem.build(res, n, perturbation="cos", amp=0.02, precision="fp32", batch_steps=3)
        p.stepper.run_steps(p.f, p.basis, p.elliptic, p.grids, p.flux, p.refs, 4)
        got.append((p.f.full_array().get(), p.f.arr.get()))
    assert rel_err(got[0][0], got[1][0]) < 4 * TOL["fp32"]
    # the x-ghost slabs follow the interior (stage 1 refreshes them)
    assert rel_err(got[0][1][0], got[1][1][0]) < 1e-4 and rel_err(got[0][1][-1], got[1][1][-1]) < 1e-4


@pytest.mark.parametrize("precision,n,nv", [("fp64", 5, 4), ("fp32", 4, 6), ("fp32", 7, 4)])
def test_alignment_rules_stay(cuda, precision, n, nv):
    """Buffers that the tensor-copy forms refused (not on a 16-byte boundary) are still refused."""
    from vlasov1d2v_b200 import _lib, problem
    from vlasov1d2v_b200._lib import VlasovError

    p = problem.build((1, 2, nv), n, perturbation=None, precision=precision, background_split=False)
    ctx = _context(p, precision)
    t = torch.zeros(ctx.state_elems + 4, dtype=DT[precision], device="cuda")
    off = t[1:1 + ctx.state_elems].view(ctx.state_shape)
    out = torch.zeros(ctx.state_shape, dtype=DT[precision], device="cuda")
    E = torch.zeros((3, n), dtype=torch.float64, device="cuda")
    with pytest.raises(VlasovError):
        ctx.rhs(off, E, out, xhalo=_lib.VL_XHALO_GHOST)
