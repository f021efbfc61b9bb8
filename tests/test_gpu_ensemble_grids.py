"""Grids of an ensemble member's stage launches: a member that has most of the work takes the ones that its
context has for the device alone (read from a profile), the others their share; and such members
step as the same problem alone, whose stages have different grids by kind."""
import json
import os
import tempfile

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _build(res, n, precision, batch=4):
    from vlasov1d2v_b200 import problem

    return problem.build(res, n, perturbation="cos", amp=0.05, precision=precision, background_split=False,
                         batch_steps=batch)


def _grids(body, nx):
    """x grid sizes of the kernels with nx rows of CTAs that body launches."""
    from torch.profiler import ProfilerActivity, profile

    body()
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        body()
        torch.cuda.synchronize()
    out = set()
    with tempfile.TemporaryDirectory() as d:
        path = os.path.join(d, "trace.json")
        prof.export_chrome_trace(path)
        with open(path) as fh:
            events = json.load(fh)["traceEvents"]
    if not any(e.get("cat") == "kernel" for e in events):
        pytest.skip("kernel profiles are not available")
    for e in events:
        grid = e.get("args", {}).get("grid")
        if e.get("cat") == "kernel" and grid and grid[1] == nx and "stage_" in e["name"]:
            out.add(grid[0])
    return out


@pytest.mark.parametrize("res,n,precision", [((16, 24, 24), 8, "fp64"), ((16, 20, 20), 6, "fp64"), ((20, 27, 29), 7, "fp32")])
@pytest.mark.parametrize("others", [0, 2])
def test_grids_of_a_member_with_most_of_the_work(cuda, res, n, precision, others, monkeypatch):
    from vlasov1d2v_b200.ensemble import Ensemble

    monkeypatch.setenv("VLASOV1D2V_FIELD", "solve")
    alone = _build(res, n, precision)
    st = alone.stepper
    st.run_steps(alone.f, alone.basis, alone.elliptic, alone.grids, alone.flux, alone.refs, 1)
    run = st._run(alone.f, alone.elliptic, alone.grids, alone.refs)

    def stages():
        dt = torch.full((1,), 1e-4, dtype=torch.float64, device="cuda")
        run.ctx.rk_stage(0, run.f, None, run.sa, run.E, dt, partials=run.ctx.workspace)
        run.ctx.rk_stage(1, run.sa, run.f, run.sb, run.E, dt, partials=run.ctx.workspace)

    want = _grids(stages, res[0])
    assert want
    ens = Ensemble([_build(res, n, precision)] + [_build((3, 4, 6), 4 + k, precision) for k in range(others)],
                   batch_steps=4)
    ens.launch(4, False)
    assert _grids(lambda: ens._steps(1), res[0]) >= want
    # one of many members of its size: not sized for the device
    ens = Ensemble([_build(res, n, precision) for _ in range(12)], batch_steps=4)
    ens.launch(4, False)
    assert not _grids(lambda: ens._steps(1), res[0]) & want


@pytest.mark.parametrize("res,n,precision", [((8, 16, 16), 8, "fp64"), ((6, 9, 11), 5, "fp64"), ((6, 9, 11), 7, "fp32")])
def test_steps_as_alone(cuda, res, n, precision):
    from vlasov1d2v_b200.ensemble import Ensemble

    alone, member, small = _build(res, n, precision), _build(res, n, precision), _build((3, 4, 6), 4, precision)
    alone.stepper.run_steps(alone.f, alone.basis, alone.elliptic, alone.grids, alone.flux, alone.refs, 7)
    Ensemble([member, small], batch_steps=4).run_steps(7)
    a, b = member.f.arr.get().astype(np.float64), alone.f.arr.get().astype(np.float64)
    assert np.max(np.abs(a - b)) < (1e-12 if precision == "fp64" else 2e-5) * np.max(np.abs(b))
    np.testing.assert_allclose(member.stepper.field_energy, alone.stepper.field_energy,
                               rtol=1e-9 if precision == "fp64" else 1e-3)
