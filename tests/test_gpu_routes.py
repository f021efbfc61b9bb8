"""Which kernels a context's calls take: the stage form, whether the loop's stage kernels solve for the
field, and the launches of a loop call, so that the tests of those routes cannot pass on another one."""
import numpy as np
import pytest
import torch

from test_gpu_field_fuse import CASES
from test_gpu_line_kernel import _context

pytestmark = pytest.mark.gpu


def _loop(res, n, precision, split, steps=4):
    from vlasov1d2v_b200 import problem

    p = problem.build(res, n, perturbation="cos", amp=0.1, precision=precision, background_split=split,
                      batch_steps=steps)
    st = p.stepper
    st.run_steps(p.f, p.basis, p.elliptic, p.grids, p.flux, p.refs, 1)
    return p, st, st._run(p.f, p.elliptic, p.grids, p.refs)


def _captured_kernels(run, steps):
    """Kernel nodes of a captured loop call."""
    from cuda.bindings import runtime as rt

    g = torch.cuda.CUDAGraph(keep_graph=True)
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        with torch.cuda.graph(g, stream=s):
            run.ctx.ssp_rk3_steps(run.f, run.sa, run.sb, run.E, run.phi, run.state, steps)
    torch.cuda.current_stream().wait_stream(s)
    raw = rt.cudaGraph_t(init_value=g.raw_cuda_graph())
    err, _, count = rt.cudaGraphGetNodes(raw)
    assert err == rt.cudaError_t.cudaSuccess
    err, nodes, count = rt.cudaGraphGetNodes(raw, count)
    assert err == rt.cudaError_t.cudaSuccess
    kinds = [rt.cudaGraphNodeGetType(n)[1] for n in nodes[:count]]
    del g
    return sum(k == rt.cudaGraphNodeType.cudaGraphNodeTypeKernel for k in kinds)


@pytest.mark.parametrize("res,n,precision,form", [((5, 6, 6), 8, "fp64", "conv"), ((5, 6, 7), 7, "fp32", "conv"),
                                                  ((6, 5, 6), 6, "fp64", "solve"), ((3, 5, 6), 2, "fp32", "conv")])
def test_launches_are_those_of_a_captured_call(cuda, res, n, precision, form, monkeypatch):
    monkeypatch.setenv("VLASOV1D2V_FIELD", form)
    _, _, run = _loop(res, n, precision, False)
    for steps in (1, 3):
        assert _captured_kernels(run, steps) == run.ctx.loop_launches(steps)
    assert run.ctx.loop_launches(0) == 1


# the grids of test_gpu_launch_overlap.py, whose kernels are launched as the one before ends only on this route
OVERLAP = [((1, 1, 1), 6, "fp64", False), ((16, 16, 16), 8, "fp64", False), ((16, 16, 16), 8, "fp32", False),
           ((8, 9, 9), 7, "fp32", False), ((5, 7, 9), 5, "fp64", False), ((16, 20, 20), 6, "fp64", False),
           ((12, 24, 24), 5, "fp32", False), ((4, 40, 40), 9, "fp64", False)]


# (order 10 has no stepper of its own: its context's route alone)
@pytest.mark.parametrize("res,n,precision,split", CASES + OVERLAP + [((3, 4, 4), 10, "fp64", False), ((3, 4, 5), 10, "fp64", False),
                                                           ((3, 4, 4), 10, "fp32", False)])
def test_field_solved_in_the_stages(cuda, res, n, precision, split, monkeypatch):
    """The small grids of the loop tests take the loop with the solve inside (all but FP32 order 2, whose
    kernel has no such form), and none does where separate solves are asked for."""
    from vlasov1d2v_b200 import problem

    for form in ("conv", "solve", "dft"):
        monkeypatch.setenv("VLASOV1D2V_FIELD", form)
        p = problem.build(res, n, perturbation=None, precision=precision, background_split=False)
        ctx = _context(p, precision)
        inside = form == "conv" and not (precision == "fp32" and n == 2)
        assert ctx.loop_launches(5) == (17 if inside else 31), (form, ctx.stage_form)


@pytest.mark.parametrize("res,n,precision,form", [
    ((4, 6, 6), 8, "fp64", "fragment"), ((4, 6, 6), 8, "fp32", "packed"), ((4, 6, 6), 6, "fp64", "generic-tma"),
    ((4, 6, 7), 7, "fp64", "line"), ((4, 6, 6), 9, "fp32", "line"), ((4, 6, 7), 7, "fp32", "line"),
    ((4, 6, 7), 5, "fp32", "line"), ((4, 6, 7), 4, "fp32", "generic-tma"), ((4, 6, 6), 6, "fp32", "generic-tma"),
    ((4, 6, 7), 6, "fp32", "generic-pairs"), ((4, 6, 6), 3, "fp32", "generic-tma"), ((2, 3, 5), 2, "fp32", "generic-pairs"),
    # the grid of the line kernel's comparison with the generic forms
    ((2, 3, 5), 3, "fp64", "line"), ((2, 3, 5), 5, "fp64", "line"), ((2, 3, 5), 7, "fp64", "line"),
    ((2, 3, 5), 9, "fp64", "line"), ((2, 3, 5), 3, "fp32", "line"), ((2, 3, 5), 5, "fp32", "line"),
    ((2, 3, 5), 7, "fp32", "line"), ((2, 3, 5), 9, "fp32", "line"),
    # order 10: by the tiles of a resident CTA (a grid of few whose last line-form turn is nearly empty, too)
    ((8, 17, 19), 10, "fp32", "generic-pairs"), ((16, 16, 16), 10, "fp32", "line"), ((8, 20, 21), 10, "fp32", "line"),
    ((32, 40, 40), 10, "fp32", "generic-tma"), ((32, 40, 41), 10, "fp32", "generic-pairs"),
    ((32, 20, 20), 10, "fp32", "generic-tma"), ((8, 12, 12), 10, "fp32", "line"), ((3, 4, 5), 10, "fp32", "line"),
    # an x slab of 4 GiB or more: past the line form's 32-bit offsets
    ((1, 1300, 1301), 9, "fp32", "pencil"), ((1, 1300, 1300), 9, "fp32", "generic-pairs"),
    ((1, 1300, 1301), 7, "fp64", "generic")])
def test_stage_forms(cuda, res, n, precision, form):
    """The context alone, without a state."""
    from vlasov1d2v_b200.basis import Basis3D
    from vlasov1d2v_b200.context import get_context
    from vlasov1d2v_b200.grid import Grid3D

    grids = Grid3D(basis=Basis3D(np.array([n] * 3)), lows=np.array([-1.0, -8.5, -8.5]),
                   highs=np.array([1.0, 8.5, 8.5]), resolutions=np.array(res))
    assert get_context(grids, precision=precision).stage_form == form


def test_benchmark_counts_its_launches(cuda, monkeypatch):
    """The benchmark reports the launches of the route it timed, not of another one."""
    import bench

    for form, want in (("conv", 8), ("solve", 13)):
        monkeypatch.setenv("VLASOV1D2V_FIELD", form)
        r = bench.measure_precision("fp64", 2, 3, 1, bench._NoDist(), res=(4, 6, 6), order=4, e2e=False)
        assert r["launches"] == want and r["stage_form"] == "generic-tma"
