"""Steps of a batch after the end of the loop: the loop state they leave, and their time, with the field solve
inside the stage kernels against separate solves."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _loop(res, n, precision, form, batch, monkeypatch):
    from vlasov1d2v_b200 import problem

    monkeypatch.setenv("VLASOV1D2V_FIELD", form)
    p = problem.build(res, n, perturbation="cos", amp=0.1, precision=precision, background_split=False,
                      batch_steps=batch)
    st = p.stepper
    st.run_steps(p.f, p.basis, p.elliptic, p.grids, p.flux, p.refs, 1)
    run = st._run(p.f, p.elliptic, p.grids, p.refs)
    assert run.ctx.loop_launches(1) == (5 if form == "conv" else 7)
    return st, run


@pytest.mark.parametrize("taken", [0, 1, 2, 4])
@pytest.mark.parametrize("res,n,precision", [((5, 6, 6), 8, "fp64"), ((5, 6, 7), 7, "fp32"), ((6, 5, 6), 6, "fp64"),
                                             ((4, 6, 6), 8, "fp32"), ((4, 5, 6), 3, "fp32")])
def test_state_after_the_end(cuda, res, n, precision, taken, monkeypatch):
    """A batch of 9 whose loop ends after `taken` steps, then another: nothing moves after the end."""
    got = []
    for form in ("conv", "solve"):
        st, run = _loop(res, n, precision, form, 9, monkeypatch)
        run.upload_state(st._host_state(run, float("inf"), taken))
        run.launch(9, False)
        one = bytes(run.read_state()), run.f.clone(), run.E.clone(), run.phi.clone()
        run.launch(9, True)
        run.graph = None
        two = bytes(run.read_state()), run.f.clone(), run.E.clone(), run.phi.clone()
        assert all(torch.equal(a, b) for a, b in zip(one[1:], two[1:]))
        a = run.read_state()
        assert a.steps == taken and a.active == 0 and a.active_next == 0 and a.status == 0
        assert one[0] == two[0]
        got.append((a.time, a.dt, a.dt_next, run.f.cpu().numpy().astype(np.float64)))
    tol = 4e-12 if precision == "fp64" else 1.2e-5
    for a, b in zip(*got):
        assert np.max(np.abs(a - b)) <= tol * np.max(np.abs(b))


def test_steps_after_the_end_are_cheap(cuda, monkeypatch):
    """They take no longer with the solve inside than with separate solves, whose kernels return at once
    (1.25 times as long when every such step repeated the solve, 0.6 as it is; best of ten replays)."""
    best = {}
    for form in ("conv", "solve"):
        st, run = _loop((20, 27, 29), 7, "fp32", form, 32, monkeypatch)
        run.upload_state(st._host_state(run, float("inf"), 0))
        for _ in range(2):
            run.launch(32, True)
        for _ in range(10):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            run.launch(32, True)
            b.record()
            torch.cuda.synchronize()
            best[form] = min(best.get(form, 1e9), a.elapsed_time(b))
        run.graph = None
    assert best["conv"] < 1.1 * best["solve"], best
