"""The loop whose stage kernels solve for the field against the loop with separate solves
(VLASOV1D2V_FIELD=solve) and with the transform (dft), read when a context is created.

Tolerance: the solves sum the density in the same precision and differ in the order of the dot products,
nx n eps = 1.4e-13 at 640 nodes, against the transform 2e-13 more; through a few steps ten times that.
FP32 states: one rounding of the state (6e-8) a stage where E differs in the last bits, 18 stages; the
field is formed from the perturbation, 0.1 of the state, so ten times that."""
import numpy as np
import pytest
import torch

from helpers import rel_err

pytestmark = pytest.mark.gpu


def _run(res, n, precision, split, form, monkeypatch, part):
    from vlasov1d2v_b200 import problem

    monkeypatch.setenv("VLASOV1D2V_FIELD", form)
    p = problem.build(res, n, perturbation="cos", amp=0.1, precision=precision, background_split=split, batch_steps=4)
    st = p.stepper
    if part == "final":      # ends inside a batch
        st.run_steps(p.f, p.basis, p.elliptic, p.grids, p.flux, p.refs, 1)
        st.final_time = float(st.time) + 5.5 * float(st.dt)
        st.main_loop(p.f, p.basis, p.elliptic, p.grids, p.flux, p.refs, None)
    else:
        st.run_steps(p.f, p.basis, p.elliptic, p.grids, p.flux, p.refs, 6)
    torch.cuda.synchronize()
    return {"f": p.f.arr.get().astype(np.float64), "E": p.elliptic.electric_field.get(),
            "phi": p.elliptic.potential.get(), "energy": np.asarray(st.field_energy),
            "time": np.asarray(st.time_array), "dt": np.asarray([float(st.dt)]), "steps": st.steps_counter}


# every kernel with the prologue: fragment, packed FP32, line (odd rows, high orders), generic TMA and
# paired rows; one x element, one tile, an element count that no lane split divides
CASES = [((1, 5, 4), 8, "fp64", False), ((9, 6, 6), 8, "fp64", False), ((7, 8, 6), 8, "fp32", True),
         ((5, 7, 9), 8, "fp32", False), ((6, 5, 7), 5, "fp64", False), ((3, 4, 5), 9, "fp64", False),
         ((1, 4, 6), 6, "fp64", False), ((12, 8, 8), 4, "fp64", False), ((4, 5, 6), 9, "fp64", False),
         ((5, 6, 7), 7, "fp32", True), ((2, 4, 4), 9, "fp32", False), ((10, 6, 6), 6, "fp32", True),
         ((7, 5, 5), 6, "fp32", True), ((6, 6, 6), 4, "fp32", False), ((5, 7, 6), 3, "fp32", True),
         ((64, 2, 1), 9, "fp64", False), ((3, 5, 6), 2, "fp32", False)]


@pytest.mark.parametrize("res,n,precision,split", CASES)
def test_matches_separate_solves(cuda, res, n, precision, split, monkeypatch):
    got = {form: _run(res, n, precision, split, form, monkeypatch, "steps") for form in ("conv", "solve", "dft")}
    tol = 4e-12 if precision == "fp64" else 1.2e-5
    for form in ("solve", "dft"):
        a, b = got["conv"], got[form]
        assert a["steps"] == b["steps"] == 6
        for key in ("f", "E", "phi", "energy", "time", "dt"):
            assert a[key].shape == b[key].shape and rel_err(a[key], b[key]) < tol, (form, key)


@pytest.mark.parametrize("res,n,precision", [((5, 6, 6), 8, "fp64"), ((5, 6, 7), 7, "fp32"), ((6, 5, 6), 6, "fp64")])
def test_final_time_inside_a_batch(cuda, res, n, precision, monkeypatch):
    got = {form: _run(res, n, precision, False, form, monkeypatch, "final") for form in ("conv", "solve")}
    a, b = got["conv"], got["solve"]
    assert a["steps"] == b["steps"]
    for key in ("f", "E", "phi", "energy", "time", "dt"):
        assert a[key].shape == b[key].shape and rel_err(a[key], b[key]) < (4e-12 if precision == "fp64" else 1.2e-5), key


def test_stopped_loop_changes_nothing(cuda, monkeypatch):
    """A batch launched on a loop that has ended leaves the state, the field and the histories alone."""
    from vlasov1d2v_b200 import problem

    monkeypatch.setenv("VLASOV1D2V_FIELD", "conv")
    p = problem.build((4, 6, 6), 6, perturbation="cos", amp=0.1, precision="fp64", batch_steps=4)
    st = p.stepper
    st.run_steps(p.f, p.basis, p.elliptic, p.grids, p.flux, p.refs, 2)
    run = st._run(p.f, p.elliptic, p.grids, p.refs)
    assert run.ctx.workspace_bytes > 0
    run.upload_state(st._host_state(run, float(st.time) * 0.5, 1 << 40))   # the final time has passed
    before = [t.clone() for t in (run.f, run.E, run.phi)]
    for graph in (False, True):
        run.launch(4, graph)
    torch.cuda.synchronize()
    assert all(torch.equal(x, y) for x, y in zip(before, (run.f, run.E, run.phi)))
    assert run.read_state().steps == 0
