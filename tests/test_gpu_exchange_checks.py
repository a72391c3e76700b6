"""The field-state exchange kernels on maps that changed after construction, on
empty populations, and on vectors only torch's own operations can take."""
from __future__ import annotations

import numpy as np
import pytest

import goss_b200 as goss
from goss_b200 import _capi

pytestmark = pytest.mark.gpu


def _coupling(nodes=(40, 30), solvers=("RK4", "ThetaSolver"), total=80):
    from goss_b200.coupling import FieldStateCoupling

    rng = np.random.default_rng(5)
    order = rng.permutation(total)
    systems, dofs, at = {}, {}, 0
    for k, (n, name) in enumerate(zip(nodes, solvers)):
        ode = goss.ParameterizedODE("fitzhughnagumo", field_states=["V"])
        solver = goss.solvers.solver_mapper[name](ode)
        solver.internal_time_step = 0.05
        systems[str(k)] = goss.ODESystemSolver(n, solver, ode)
        systems[str(k)].set_states(ode.get_ic()[None, :] * (1 + rng.uniform(-0.2, 0.2, (n, 2))) + 0.1)
        dofs[str(k)] = order[at:at + n]
        at += n
    return FieldStateCoupling(systems, dofs, total)


def _vector(total=80):
    import torch

    return torch.tensor(np.random.default_rng(6).uniform(-90, 20, total), device="cuda")


# the solver that exchanges inside its own launch and the one that does not
@pytest.mark.parametrize("label", ["0", "1"])
@pytest.mark.parametrize("entry", [80, -1, 2**62])
def test_an_entry_outside_the_vector_is_left_out_and_reported(label, entry):
    c, v = _coupling(), _vector()
    before, dofs = v.cpu().numpy(), c.dofs[label].cpu().numpy()
    c.dofs[label][3] = entry
    c.step((0.0, 0.1), v)
    with pytest.raises(ValueError, match="dof map"):
        c.systems[label].synchronize()
    system = c.systems[label]
    assert system.status() & _capi.GOSS_FLAG_BAD_DOF
    status = system.node_status()
    assert status[3] & _capi.GOSS_FLAG_BAD_DOF and not status[np.arange(status.size) != 3].any()
    after = v.cpu().numpy()
    assert after[dofs[3]] == before[dofs[3]]  # its dof no longer has a node
    assert (np.delete(after[dofs], 3) != np.delete(before[dofs], 3)).all()
    assert (system.states[3] != _coupling().systems[label].states[3]).any()  # the node went on by itself


def test_a_map_on_the_host_is_not_read_by_a_kernel():
    c, v = _coupling(), _vector()
    c.dofs["0"] = c.dofs["0"].cpu()
    assert not c._plain(v)
    with pytest.raises(RuntimeError):
        c.step((0.0, 0.1), v)


def test_a_replaced_map_is_followed():
    c, d = _coupling(), _coupling()
    v, w = _vector(), _vector()
    flipped = c.dofs["0"].flip(0).contiguous()
    c.dofs["0"] = flipped
    d.dofs["0"].copy_(flipped)
    c.step((0.0, 0.1), v)
    d.step((0.0, 0.1), w)
    c.synchronize()
    assert (v == w).all()


def test_an_empty_population_takes_no_part():
    c, v = _coupling(nodes=(40, 0)), _vector()
    for k in range(2):
        c.step((0.1 * k, 0.1 * (k + 1)), v)
    c.to_field_states(v)
    c.from_field_states(v)
    c.synchronize()
    np.testing.assert_array_equal(v[c.dofs["0"]].cpu().numpy(), c.systems["0"].field_states[:, 0])


def test_transforms_and_modes_see_the_copies():
    import torch
    from torch.autograd import forward_ad
    from torch.utils._python_dispatch import TorchDispatchMode

    c = _coupling()

    def read(v):
        v = v.clone()
        c.from_field_states(v)
        return v

    one = read(_vector())
    assert torch.equal(torch.func.vmap(read)(_vector().repeat(3, 1)), one.repeat(3, 1))
    seen = []

    class Watch(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            seen.append(str(func))
            return func(*args, **(kwargs or {}))

    v = _vector()
    with Watch():
        c.from_field_states(v)
    assert any("index_copy" in s for s in seen) and torch.equal(v, one)
    with forward_ad.dual_level():
        dual = forward_ad.make_dual(_vector(), torch.ones(80, dtype=torch.float64, device="cuda"))
        assert not c._plain(dual) and c._plain(_vector())
        c.from_field_states(dual)
        owned = torch.cat([c.dofs["0"], c.dofs["1"]])
        tangent = forward_ad.unpack_dual(dual).tangent
        assert not tangent[owned].any() and tangent.sum() == 80 - owned.numel()
    with torch.inference_mode():
        v = _vector()
        c.from_field_states(v)
        assert torch.equal(v, one)
