"""Device memory of the FP64 RK4 adjoint: the room for kept stage derivatives
is taken only where a segment is recomputed, and the automatic tape counts it."""
from __future__ import annotations

import pytest

import goss_b200 as goss

pytestmark = pytest.mark.gpu

NODES, STEPS, INTERVALS = 100, 5, 6  # six segments of five steps
ROW = (256 + 256) * 8
SEGMENT = STEPS * 2 * ROW


def _trace(**more):
    from goss_b200 import adjoint

    ode = goss.ParameterizedODE("fitzhughnagumo", field_parameters=["a", "b"])
    return adjoint.RK4Trace(ode, NODES, 0.5, STEPS, INTERVALS, STEPS, precision="double", **more)


@pytest.mark.parametrize("taped", [0, 5, 6])
def test_scratch_holds_stages_only_for_recomputed_segments(taped):
    t = _trace(tape_bytes=taped * SEGMENT)
    assert t.taped_segments == taped and t._keep_stages == (taped < INTERVALS)
    assert t._scratch.numel() * 8 == (4 if taped < INTERVALS else 1) * SEGMENT


# the free memory in segments beyond the reserve: one goes to the scratch, and
# three more to the stages where the tape does not hold every segment
@pytest.mark.parametrize("free, taped", [(7, 6), (9, 6), (6.9, 2), (5, 1), (3, 0), (0, 0)])
def test_automatic_tape_leaves_room_for_the_scratch(free, taped, monkeypatch):
    import torch

    reserve = 1 << 20
    monkeypatch.setattr(torch.cuda, "mem_get_info", lambda *_: (int(reserve + free * SEGMENT), 1 << 40))
    t = _trace(tape_bytes="auto", tape_reserve=reserve)
    assert t.taped_segments == taped and t._keep_stages == (taped < INTERVALS)


def test_without_the_memory_for_stages_they_are_evaluated_again(monkeypatch):
    import torch

    empty, asked = torch.empty, []

    def tight(shape, *args, **kwargs):
        if len(shape) == 3 and shape[1] == 8:
            asked.append(shape)
            raise torch.OutOfMemoryError("no room")
        return empty(shape, *args, **kwargs)

    monkeypatch.setattr(torch, "empty", tight)
    t = _trace()
    monkeypatch.undo()
    assert asked and not t._keep_stages
    ode = t.ode
    fp = torch.tensor([[0.13, 0.013]], dtype=torch.float64, device="cuda").repeat(NODES, 1)
    y0 = torch.tensor(ode.get_ic(), device="cuda").repeat(NODES, 1) + 0.1
    u = _trace()
    for x, y in zip((t.run_forward(fp, y0), *t.run_backward(torch.ones(INTERVALS, NODES, device="cuda"))),
                    (u.run_forward(fp, y0), *u.run_backward(torch.ones(INTERVALS, NODES, device="cuda")))):
        assert torch.equal(x, y)
