"""Counter totals summed on the device against the per-node counters."""
from __future__ import annotations

import numpy as np
import pytest

import goss_b200 as goss

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["ThetaSolver", "ImplicitEuler", "ESDIRK23a"])
@pytest.mark.parametrize("nodes", [1, 31, 256, 257, 200_003])  # one warp, one block, ragged, more than one pass
def test_totals_are_the_sums_of_the_node_counters(name, nodes):
    ode = goss.ParameterizedODE("fitzhughnagumo", field_states=["V"])
    solver = goss.solvers.solver_mapper[name](ode)
    system = goss.ODESystemSolver(nodes, solver, ode)
    rng = np.random.default_rng(3)
    system.set_states(ode.get_ic()[None, :] * (1 + rng.uniform(-0.5, 0.5, (nodes, ode.num_states))))
    for k in range(3):
        if k < 2:
            system.forward(0.5 * k, 0.5)
        else:
            system.solve(np.array([1.0, 1.5, 2.0]))
        jc, rj, ac = system.counters()
        assert ac.sum() > 0 and jc.sum() > 0
        assert solver.num_jac_comp() == jc.sum()
        assert (solver._counters["rejected"], solver._counters["accepted"]) == (rj.sum(), ac.sum())
