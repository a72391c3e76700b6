"""RK4 adjoint with the recompute's stage derivatives kept against evaluating
them again: the same gradients bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

import goss_b200 as goss

pytestmark = pytest.mark.gpu


# one node, a ragged block, blocks of several warps; segments that end inside the
# trajectory, the last one ragged, and some of them taped
@pytest.mark.parametrize("nodes", [1, 33, 5001])
@pytest.mark.parametrize("intervals, every, tape_segments", [(1, 5, 0), (7, 10, 0), (7, 10, 2)])
def test_kept_stages_do_not_change_the_gradient(nodes, intervals, every, tape_segments, monkeypatch):
    import torch

    from goss_b200 import adjoint

    ode = goss.ParameterizedODE("fitzhughnagumo", field_parameters=["a", "b"])
    rng = np.random.default_rng(nodes)
    fp = torch.tensor(np.array([0.13, 0.013]) * (1 + rng.uniform(-0.05, 0.05, (nodes, 2))), device="cuda")
    y0 = torch.tensor(ode.get_ic()[None, :] * (1 + rng.uniform(-0.05, 0.05, (nodes, 2))) + 0.1, device="cuda")
    segment = every * 2 * ((nodes + 255) // 256 * 256 + 256) * 8
    out = []
    for limit in (adjoint._STAGE_SCRATCH_BYTES, 0):
        monkeypatch.setattr(adjoint, "_STAGE_SCRATCH_BYTES", limit)
        tr = adjoint.RK4Trace(ode, nodes, 0.5, 5, intervals, every, precision="double",
                              tape_bytes=tape_segments * segment)
        assert tr._keep_stages == (limit > 0) and tr.taped_segments == tape_segments
        v = tr.run_forward(fp, y0)
        out.append((v, *tr.run_backward(2 * v)))
    for a, b in zip(*out):
        assert torch.equal(a, b)
    assert torch.isfinite(out[0][1]).all() and (out[0][1] != 0).any()
