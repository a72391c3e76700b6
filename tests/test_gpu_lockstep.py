"""The implicit kernels' default block size (chosen from the number of nodes)
against blocks of 256, bit for bit, where it changes."""
from __future__ import annotations

import numpy as np
import pytest

import goss_b200 as goss

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["ThetaSolver", "ImplicitEuler", "ESDIRK23a"])
# one warp per SM, its limit on 148 SMs and one more, one full wave of 256 and one more, ragged waves
@pytest.mark.parametrize("nodes", [1, 33, 148 * 32, 148 * 32 + 1, 148 * 256, 148 * 256 + 1, 50_021])
def test_default_block_equals_256(name, nodes):
    states = []
    for block in (0, 256):
        ode = goss.ParameterizedODE("fitzhughnagumo", field_parameters=["a", "b"])
        system = goss.ODESystemSolver(nodes, goss.solvers.solver_mapper[name](ode), ode)
        system.set_block_size(block)
        rng = np.random.default_rng(nodes)
        system.set_states(ode.get_ic()[None, :] * (1 + rng.uniform(-0.3, 0.3, (nodes, 2))) + 0.1)
        for k in range(4):
            system.forward(0.5 * k, 0.5)
        states.append((system.states, *system.counters()))
    for a, b in zip(*states):
        np.testing.assert_array_equal(a, b)
