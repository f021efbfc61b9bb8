"""The loop state and the histories in one transfer: what a caller sees of a batch is what the device holds."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _build(res, n, batch, precision="fp64"):
    from vlasov1d2v_b200 import problem

    return problem.build(res, n, perturbation="cos", amp=0.1, precision=precision, background_split=False,
                         batch_steps=batch)


@pytest.mark.parametrize("batch,steps", [(1, 3), (4, 4), (4, 6), (7, 0)])
def test_state_and_histories(cuda, batch, steps):
    """run_steps against the same batches launched by hand, their state and history rows read one by one."""
    p, q = _build((3, 5, 4), 5, batch), _build((3, 5, 4), 5, batch)
    for s in (p, q):   # the initial energy and dt
        s.stepper.run_steps(s.f, s.basis, s.elliptic, s.grids, s.flux, s.refs, 0)
    p.stepper.run_steps(p.f, p.basis, p.elliptic, p.grids, p.flux, p.refs, steps)
    st = q.stepper
    run = st._run(q.f, q.elliptic, q.grids, q.refs)
    energy, times, dt, left = [], [], st.dt, steps
    while left:
        k = min(batch, left)
        st.time, st.dt = (times[-1] if times else 0), dt
        run.upload_state(st._host_state(run, float("inf"), k))
        run.launch(k, False)
        h = run.hist[:, :k].cpu().numpy()
        assert run.read_state().steps == k
        energy, times, dt, left = energy + list(h[0]), times + list(h[1]), float(h[2, -1]), left - k
    assert p.stepper.steps_counter == steps and p.stepper.dt == dt
    assert np.array_equal(p.stepper.time_array[1:], times) and np.array_equal(p.stepper.field_energy[1:], energy)
    assert torch.equal(p.elliptic.potential, run.phi) and torch.equal(p.elliptic.electric_field, run.E)
    run = p.stepper._run(p.f, p.elliptic, p.grids, p.refs)
    state, h = run.read_batch()
    assert bytes(state) == bytes(run.read_state()) and np.array_equal(h, run.hist.cpu().numpy())
    assert run.hist.data_ptr() % 64 == 0 and run.state.data_ptr() % 64 == 0
    assert p.elliptic.electric_field.data_ptr() != run.E.data_ptr()


@pytest.mark.parametrize("batch,steps,graph", [(3, 7, True), (4, 4, False), (2, 0, True)])
def test_ensemble_batches(cuda, batch, steps, graph):
    """An ensemble against its members run alone, one of which reaches its final time inside a batch."""
    from vlasov1d2v_b200.ensemble import Ensemble

    shapes = (((4, 5, 6), 5), ((3, 6, 6), 4), ((4, 4, 4), 6))
    alone = [_build(r, n, 1) for r, n in shapes]
    for s in alone:
        s.stepper.run_steps(s.f, s.basis, s.elliptic, s.grids, s.flux, s.refs, max(steps, 1))
    final = [float("inf"), float(alone[1].stepper.time_array[-1]) * 0.5, float("inf")]
    members = [_build(r, n, 1) for r, n in shapes]
    ens = Ensemble(members, final_time=final, batch_steps=batch)
    ens.run_steps(steps, use_graph=graph)
    for i, (m, s) in enumerate(zip(members, alone)):
        times = s.stepper.time_array
        want = steps if i != 1 else int(np.sum(times[1:-1] < final[1])) + 1 if steps else 0
        assert m.stepper.steps_counter == want == len(m.stepper.time_array) - 1
        # the same kernels' sums in another grouping: rounding of the density through the steps
        np.testing.assert_allclose(m.stepper.time_array, times[:want + 1], rtol=1e-11)
        np.testing.assert_allclose(m.stepper.field_energy, s.stepper.field_energy[:want + 1], rtol=1e-11)
        assert torch.equal(m.elliptic.electric_field, ens.runs[i].E)


def test_ensemble_reports_a_failed_member(cuda):
    from vlasov1d2v_b200.ensemble import Ensemble
    from vlasov1d2v_b200.timestep import NonFiniteError

    members = [_build((3, 4, 4), 4, 2), _build((2, 4, 4), 5, 2)]
    ens = Ensemble(members, batch_steps=2)
    members[1].f.arr[1] = float("nan")
    for _ in range(2):   # and stays reported
        with pytest.raises(NonFiniteError):
            ens.run_steps(2)
    assert members[0].stepper.steps_counter == 4
