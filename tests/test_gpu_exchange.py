"""Field-state exchange with a device vector: the kernels against torch's
indexing (taken for vectors the kernels do not take) on every kind of vector."""
from __future__ import annotations

import numpy as np
import pytest

import goss_b200 as goss

pytestmark = pytest.mark.gpu


def _coupling(nodes, fields):
    import torch

    from goss_b200.coupling import FieldStateCoupling

    rng = np.random.default_rng(nodes)
    total = sum(nodes)
    order = rng.permutation(total + 3)  # some dofs belong to no node
    systems, dofs, at = {}, {}, 0
    for k, n in enumerate(nodes):
        ode = goss.ParameterizedODE("fitzhughnagumo", field_parameters=["a", "b"] if k else [], field_states=fields)
        solver = goss.solvers.RK4(ode) if k else goss.solvers.ThetaSolver(ode)
        solver.internal_time_step = 0.05
        systems[str(k)] = goss.ODESystemSolver(n, solver, ode)
        systems[str(k)].set_states(ode.get_ic()[None, :] * (1 + rng.uniform(-0.2, 0.2, (n, 2))) + 0.1)
        dofs[str(k)] = order[at:at + n]
        at += n
    shape = (total + 3,) if len(fields) == 1 else (total + 3, len(fields))
    v = torch.tensor(rng.uniform(-90, 20, shape), device="cuda")
    return FieldStateCoupling(systems, dofs, total + 3), v


@pytest.mark.parametrize("nodes", [(1,), (31, 257), (1000, 70_001)])
@pytest.mark.parametrize("fields", [["V"], ["s"], ["s", "V"]])
def test_kernels_equal_torch_indexing(nodes, fields):
    import torch

    a, va = _coupling(nodes, fields)
    b, vb = _coupling(nodes, fields)
    strided = torch.empty(tuple(2 * n for n in vb.shape), dtype=vb.dtype, device="cuda")
    strided = strided[tuple(slice(None, None, 2) for _ in vb.shape)]
    strided.copy_(vb)  # not contiguous: torch's indexing
    assert a._plain(va) and not b._plain(strided)
    version = va._version
    for k in range(3):
        a.step((0.1 * k, 0.1 * (k + 1)), va)
        b.step((0.1 * k, 0.1 * (k + 1)), strided)
        assert torch.equal(va, strided)
    assert va._version > version
    a.from_field_states(va)
    b.from_field_states(strided)
    va += 1.5
    strided += 1.5
    a.to_field_states(va)
    b.to_field_states(strided)
    a.synchronize()
    b.synchronize()
    for lab in a.systems:
        np.testing.assert_array_equal(a.systems[lab].states, b.systems[lab].states)
    with torch.no_grad():
        leaf = va.clone().requires_grad_(True)
        assert not a._plain(leaf)
        a.from_field_states(leaf)
        assert torch.equal(leaf.detach(), va)
    with pytest.raises(TypeError):
        a.step((0.0, 0.1), va.cpu())
    with pytest.raises(ValueError):
        a.step((0.0, 0.1), va[:-1])
