"""The stage forms that serve x slabs of 4 GiB and more (past the line form's 32-bit offsets) at small sizes, by
switch: the generic kernel's cp.async form (FP64 rows of an odd number of values) and the register-pencil
kernel (FP32), every stage kind and the moment partials of each element and node, against the oracle.

Tolerances as for the line form (40 eps of the largest value; test_gpu_line_kernel.py) and the FP64
partials (test_gpu_moment_partials.py)."""
import numpy as np
import pytest
import torch

from helpers import INNER, rel_err
from oracle import vlasov_oracle as vo
from test_gpu_line_kernel import TOL, _context, _inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,form", [("fp64", "gen"), ("fp32", "pencil")])
@pytest.mark.parametrize("n,res", [(3, (2, 3, 5)), (5, (1, 4, 9)), (7, (3, 2, 5)), (9, (2, 3, 5))])
def test_stages(cuda, n, res, precision, form, monkeypatch):
    from vlasov1d2v_b200 import _lib, problem

    monkeypatch.setenv("VLASOV1D2V_STAGE_KERNEL", form)
    p = problem.build(res, n, perturbation=None, precision=precision, background_split=False)
    ctx = _context(p, precision)
    assert ctx.stage_form == {"gen": "generic", "pencil": "pencil"}[form]
    c = vo.make_case(*res, n)
    f, fn, E, tf, tfn, tE = _inputs(c.shape, n, res, precision)
    f[0], f[-1] = f[-2], f[1]
    R = vo.rhs(f, E, c)
    dt = 0.0071
    tdt = torch.tensor([dt], dtype=torch.float64, device="cuda")
    for stage, want in ((0, f + dt * R), (1, 0.75 * fn + 0.25 * f + (0.25 * dt) * R),
                        (2, fn / 3 + (2 / 3) * f + ((2 / 3) * dt) * R)):
        parts = torch.zeros(ctx.workspace.numel() // 8, dtype=torch.float64, device="cuda")
        out = torch.zeros_like(tf)
        ctx.rk_stage(stage, tf, tfn if stage else None, out, tE, tdt, xhalo=_lib.VL_XHALO_PERIODIC,
                     partials=parts.view(torch.uint8))
        got = out.cpu().numpy().astype(np.float64)[INNER]
        assert rel_err(got, want[INNER]) < TOL[precision], stage
        part = parts.cpu().numpy()
        used = int(np.flatnonzero(part)[-1]) + 1
        assert used % (res[0] * n) == 0
        rho = part[:used].reshape(res[0], -1, n).sum(axis=1)
        size = np.tensordot(np.abs(got), np.abs(c.qw), axes=([2, 3, 4, 5], [0, 1, 2, 3]))
        assert np.all(np.abs(rho - np.tensordot(got, c.qw, axes=([2, 3, 4, 5], [0, 1, 2, 3]))) < 1e-12 * size), stage
