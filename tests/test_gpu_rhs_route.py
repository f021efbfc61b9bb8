"""FP32 order 3 on rows that no tensor copy takes: a right-hand side alone runs on the register-pencil kernel
where the line form's tiles would be too empty (rows of 29 elements in tiles of 28) and not all resident at
once, on the line form elsewhere; the stages always on the line form.  Told apart by their rounding: the
same bits as the forced kernel, and other bits than the other one."""
import pytest
import torch

from helpers import rel_err
from test_gpu_line_kernel import TOL, _context, _inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("res,pencil", [((64, 40, 29), True), ((48, 50, 31), True), ((64, 40, 57), True),
                                        ((64, 80, 1), True), ((64, 40, 67), True), ((64, 30, 89), True),
                                        ((64, 40, 25), False), ((48, 50, 27), False), ((64, 40, 83), False),
                                        ((64, 40, 45), False), ((64, 20, 117), False),
                                        ((2, 5, 29), False), ((1, 5, 1), False)])
def test_order_3(cuda, res, pencil, monkeypatch):
    from vlasov1d2v_b200 import _lib, problem

    got = {}
    for form in (None, "line", "pencil"):
        monkeypatch.delenv("VLASOV1D2V_STAGE_KERNEL", raising=False)
        if form:
            monkeypatch.setenv("VLASOV1D2V_STAGE_KERNEL", form)
        p = problem.build(res, 3, perturbation=None, precision="fp32", background_split=False)
        ctx = _context(p, "fp32")
        assert ctx.stage_form == (form or "line")
        _, _, _, tf, _, tE = _inputs(tuple(ctx.state_shape), 3, res, "fp32")
        rhs, weighted, stage = (torch.zeros_like(tf) for _ in range(3))
        ctx.rhs(tf, tE, rhs, xhalo=_lib.VL_XHALO_GHOST)
        ctx.rhs_weighted(tf, tE, weighted, (0.5, -2.0, 3.0), xhalo=_lib.VL_XHALO_PERIODIC)
        tdt = torch.tensor([0.0071], dtype=torch.float64, device="cuda")
        ctx.rk_stage(0, tf, None, stage, tE, tdt, partials=ctx.workspace)
        got[form] = rhs, weighted, stage
    same, other = ("pencil", "line") if pencil else ("line", "pencil")
    for k in range(2):
        assert torch.equal(got[None][k], got[same][k])
        assert not torch.equal(got[None][k], got[other][k])
        assert rel_err(got[None][k].cpu().numpy(), got[other][k].cpu().numpy()) < TOL["fp32"]
    assert torch.equal(got[None][2], got["line"][2])
