"""The moment partials of the stage kernels, per x element and node, against the 64-bit moment of the values
that the stage stored.

Tolerance, of the sum of the terms' sizes: FP64 sums of at most nu nv n^2 < 1e4 terms, 1e4 2^-53 = 1e-12;
kernels that sum a tile in FP32 (FP32 orders 2, 3, 5, 6 and 8 with their default kernels): rounded weights
and n terms of 2^-24 each, (n + 1) 6e-8 < 6e-7."""
import numpy as np
import pytest
import torch

from helpers import INNER
from oracle import vlasov_oracle as vo
from test_gpu_line_kernel import _context, _inputs

pytestmark = pytest.mark.gpu

# FP64 sums: every FP64 kernel; in FP32 orders 4 and 10 and the line-form kernel (orders 7, 9, odd rows)
SUM64 = [(10, (32, 20, 20), "fp32"), (10, (2, 3, 4), "fp32"), (4, (2, 3, 5), "fp32"), (4, (3, 5, 16), "fp32"), (4, (2, 4, 33), "fp32"), (7, (2, 3, 5), "fp32"),
         (7, (3, 4, 6), "fp32"), (9, (2, 3, 4), "fp32"), (3, (2, 3, 4), "fp32"), (5, (2, 4, 7), "fp32"),
         (4, (2, 3, 5), "fp64"), (6, (3, 3, 8), "fp64"), (7, (2, 3, 5), "fp64"), (8, (2, 3, 6), "fp64"),
         (9, (2, 3, 4), "fp64")]
SUM32 = [(2, (3, 4, 5), "fp32"), (3, (2, 4, 6), "fp32"), (5, (2, 3, 6), "fp32"), (6, (3, 4, 6), "fp32"),
         (8, (2, 3, 5), "fp32")]


@pytest.mark.parametrize("n,res,precision,tol", [c + (1e-12,) for c in SUM64] + [c + (6e-7,) for c in SUM32])
def test_partials_per_element_and_node(cuda, n, res, precision, tol):
    from vlasov1d2v_b200 import _lib, problem

    p = problem.build(res, n, perturbation=None, precision=precision, background_split=False)
    ctx = _context(p, precision)
    c = vo.make_case(*res, n)
    _, _, _, tf, tfn, tE = _inputs(c.shape, n, res, precision)
    tdt = torch.tensor([0.0071], dtype=torch.float64, device="cuda")
    for stage in (0, 1):
        parts = torch.zeros(ctx.workspace.numel() // 8, dtype=torch.float64, device="cuda")
        out = torch.zeros_like(tf)
        ctx.rk_stage(stage, tf, tfn if stage else None, out, tE, tdt, xhalo=_lib.VL_XHALO_PERIODIC,
                     partials=parts.view(torch.uint8))
        got = parts.cpu().numpy()
        used = int(np.flatnonzero(got)[-1]) + 1   # [nx][CTAs of an element][n]
        assert used % (res[0] * n) == 0
        rho = got[:used].reshape(res[0], -1, n).sum(axis=1)
        f = out.cpu().numpy().astype(np.float64)[INNER]
        want = np.tensordot(f, c.qw, axes=([2, 3, 4, 5], [0, 1, 2, 3]))
        size = np.tensordot(np.abs(f), np.abs(c.qw), axes=([2, 3, 4, 5], [0, 1, 2, 3]))
        assert np.all(np.abs(rho - want) < tol * size), (stage, np.max(np.abs(rho - want) / size))
