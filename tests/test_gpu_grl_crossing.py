"""FP64 GRL1 where a state's coefficient crosses zero.

Next to the crossing e^{ah} - 1 is a few multiples of 2^-53, and the last bit
of the coefficient a decides the eighth digit of the increment.  The 64 nodes of
``golden/tp06_grl1_crossing.npz`` (ten Tusscher-Panfilov, four fields, 100 steps
of 0.01 ms from t = 10, through the stimulus) are those of 2,097,152 random ones
whose V moved the furthest, 1e-9 to 4e-8 of the states' scale, under a change of
the rounding of the linearised model alone; the states are those of the kernels
with CUDA's division and exponentials (CUDA 12.9).
"""
from __future__ import annotations

from pathlib import Path

import numpy as np
import pytest

import goss_b200 as goss

pytestmark = pytest.mark.gpu

GOLDEN = np.load(Path(__file__).parent / "golden" / "tp06_grl1_crossing.npz")


# a thread per node: both register caps (any other block size than the default
# takes the smaller one; 2,560 nodes in default blocks the larger)
@pytest.mark.parametrize("copies, block", [(1, 64), (40, 0)])
@pytest.mark.parametrize("how", ["forward", "solve"])
def test_increments_at_the_crossing(copies, block, how):
    fields = ["g_Kr", "g_Ks", "g_CaL", "g_to"]
    ode = goss.ParameterizedODE("tentusscher_panfilov_2006_M_cell", field_parameters=fields)
    solver = goss.solvers.GRL1(ode)
    solver.internal_time_step = 0.01
    system = goss.ODESystemSolver(64 * copies, solver, ode)
    system.set_block_size(block)
    system.set_states(np.tile(GOLDEN["y0"], (copies, 1)))
    system.field_parameters = np.tile(GOLDEN["fields"], (copies, 1))
    if how == "forward":
        system.forward(10.0, 1.0)
    else:
        system.solve(np.array([10.0, 11.0]))
    want = np.tile(GOLDEN["states"], (copies, 1))
    # the same operations give the same bits; any other rounding is 1e-8 off
    np.testing.assert_allclose(system.states, want, rtol=1e-12, atol=1e-13)
