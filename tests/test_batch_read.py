"""What a run reads back after a batch (no GPU: the loop's buffers on the host, their copies counted)."""
from types import SimpleNamespace

import numpy as np
import pytest
import torch

from vlasov1d2v_b200 import _lib
from vlasov1d2v_b200.timestep import _Run


@pytest.mark.parametrize("cap,limit,steps", [(1, 1, 1), (32, 3, 3), (32, 32, 17), (40000, 30000, 30000), (5000, 8, 8), (40000, 8, 8),
                                             (200000, 8, 5), (200000, 1, 1), (200000, 1, 0), (200000, None, 7)])
def test_copies_follow_the_steps(cap, limit, steps, monkeypatch):
    run = _Run(SimpleNamespace(nx=2, n=3), torch.zeros(4), cap)
    st = _lib.VlRunState()
    st.steps, st.time, st.status = steps, 0.25, 0
    run.state.copy_(torch.frombuffer(bytearray(bytes(st)), dtype=torch.uint8))
    rows = torch.arange(3.0 * cap, dtype=torch.float64).view(3, cap)
    run.hist.copy_(rows)
    read = []
    cpu = torch.Tensor.cpu
    monkeypatch.setattr(torch.Tensor, "cpu", lambda t: (read.append(t.numel() * t.element_size()), cpu(t))[1])
    got, h = run.read_batch(limit) if limit else run.read_batch()
    assert got.steps == steps and got.time == 0.25
    assert np.array_equal(h[:, :steps], rows[:, :steps].numpy())
    # a call of a few steps does not carry a long ring (or a short one in more than one copy)
    if limit is not None:
        assert sum(read) <= max(48 * limit, 400 << 10) + 256
    assert len(read) <= 2 and (cap > 1000 or len(read) == 1)
