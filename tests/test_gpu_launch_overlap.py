"""Stage kernels launched as the one before ends (the loop with the field solves inside): back to back in one
stream, in a captured graph and on two streams at once, the same bits as a launch at a time."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _loop(res, n, precision):
    from vlasov1d2v_b200 import problem

    p = problem.build(res, n, perturbation="cos", amp=0.1, precision=precision, background_split=False, batch_steps=6)
    st = p.stepper
    st.run_steps(p.f, p.basis, p.elliptic, p.grids, p.flux, p.refs, 0)   # initial energy and dt
    run = st._run(p.f, p.elliptic, p.grids, p.refs)
    run.upload_state(st._host_state(run, float("inf"), 1 << 40))
    return run


def _result(run):
    torch.cuda.synchronize()
    return run.f.clone(), run.E.clone(), run.phi.clone(), bytes(run.read_state())[:40]


# one CTA; fragment, packed FP32, line and generic kernels, small and with every slot taken
@pytest.mark.parametrize("res,n,precision", [((1, 1, 1), 6, "fp64"), ((16, 16, 16), 8, "fp64"), ((16, 16, 16), 8, "fp32"),
                                             ((8, 9, 9), 7, "fp32"), ((5, 7, 9), 5, "fp64"), ((16, 20, 20), 6, "fp64"),
                                             ((12, 24, 24), 5, "fp32"), ((4, 40, 40), 9, "fp64")])
def test_same_bits_however_launched(cuda, res, n, precision):
    runs = [_loop(res, n, precision) for _ in range(4)]
    first = runs[0]
    first.launch(6, False)
    first.launch(6, False)
    want = _result(first)
    runs[1].launch(6, False)
    runs[1].launch(6, True)    # captured: the graph's edges carry the same order
    streams = [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()
    for _ in range(2):
        for s, r in zip(streams, runs[2:]):
            with torch.cuda.stream(s):
                r.launch(6, False)
    for r in runs[1:]:
        got = _result(r)
        assert all(torch.equal(a, b) for a, b in zip(got[:3], want[:3])) and got[3] == want[3]
