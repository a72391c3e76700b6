"""FP64 explicit steps with a node's rows split over four warps (the default of
small systems) against a thread per node (any other block size than the
default), at the edges of a warp and of the rule that chooses."""
from __future__ import annotations

import numpy as np
import pytest

import goss_b200 as goss

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,ldt", [("GRL1", 0.01), ("RK4", 0.0005)])
@pytest.mark.parametrize("model", ["tentusscher_panfilov_2006_M_cell", "tentusscher_2004_mcell"])
# one node, ragged warps, the largest split system on 148 SMs and one more
@pytest.mark.parametrize("nodes", [1, 31, 33, 16 * 148, 16 * 148 + 1])
def test_split_rows_equal_thread_per_node(model, name, ldt, nodes):
    states = []
    for block in (0, 64):
        ode = goss.ParameterizedODE(model, field_parameters=["g_Kr", "g_Ks", "g_CaL", "g_to"])
        solver = goss.solvers.solver_mapper[name](ode)
        solver.internal_time_step = ldt
        system = goss.ODESystemSolver(nodes, solver, ode)
        system.set_block_size(block)
        rng = np.random.default_rng(nodes)
        system.set_states(ode.get_ic()[None, :] * (1 + rng.uniform(-0.01, 0.01, (nodes, ode.num_states))))
        fields = system.field_parameters
        system.field_parameters = fields * rng.uniform(0.9, 1.1, fields.shape)
        for k in range(3):
            system.forward(20 * ldt * k, 20 * ldt)
        states.append(system.states)
    # the two associate alike but may contract different products: the bar of
    # the FP64 solvers against the reference, on 60 steps of a cell at rest
    scale = np.maximum(np.abs(states[1]), 0.01 * np.abs(states[1]).max(axis=0))
    assert np.max(np.abs(states[0] - states[1]) / scale) < 1e-10
