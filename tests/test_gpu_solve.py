"""solve() in one launch per chunk of output times against the loop of forwards
it stands for, bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

import goss_b200 as goss

pytestmark = pytest.mark.gpu


def _system(model, solver, nodes, fields, precision):
    ode = goss.ParameterizedODE(model, field_states=fields)
    s = goss.solvers.solver_mapper[solver](ode)
    s.internal_time_step = 0.03  # 0.1 is not a multiple: four shorter steps
    system = goss.ODESystemSolver(nodes, s, ode, precision=precision)
    rng = np.random.default_rng(nodes)
    system.set_states(ode.get_ic()[None, :] * (1 + rng.uniform(-0.05, 0.05, (nodes, ode.num_states))))
    return system


# one node and many times (several chunks of the staging buffer), a ragged
# block, more than the staging buffer holds 32 times of
@pytest.mark.parametrize("nodes, times", [(1, 9000), (129, 70), (1000, 40)])
@pytest.mark.parametrize("precision", ["single", "double"])
@pytest.mark.parametrize("tangled", [True, False])
def test_solve_equals_forward_loop(nodes, times, precision, tangled):
    fields = ["s", "V"]
    a, b = (_system("fitzhughnagumo", "RK4", nodes, fields, precision) for _ in range(2))
    a._tangled_storage = b._tangled_storage = tangled
    t = np.concatenate([0.1 * np.arange(times - 1), [0.1 * (times - 2) + 0.05]])
    out = a.solve(t).reshape(times, -1)
    for k in range(1, times):
        b.forward(t[k - 1], t[k] - t[k - 1])
        if times < 100 or k % 100 == 0 or k > times - 3:
            np.testing.assert_array_equal(out[k], b.field_states.reshape(-1), err_msg=str(k))
    np.testing.assert_array_equal(a.states, b.states)


@pytest.mark.parametrize("solver", ["GRL1", "GRL2", "ExplicitEuler"])
@pytest.mark.parametrize("precision", ["single", "double"])
def test_one_cell_solve_equals_forward_loop(solver, precision):
    model = "beeler_reuter_1977"
    a, b = (_system(model, solver, 1, ["V"], precision) for _ in range(2))
    t = np.array([0.0, 0.1, 0.5, 0.5, 1.7])
    out = a.solve(t)
    for k in range(1, t.size):
        b.forward(t[k - 1], t[k] - t[k - 1])
        np.testing.assert_array_equal(out[k], b.field_states)
    np.testing.assert_array_equal(a.states, b.states)
