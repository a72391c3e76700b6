"""Single-precision states that are not finite, zero or tiny between the forwards
of one launch: the same values as one launch per forward, the node's other
states untouched."""
from __future__ import annotations

import numpy as np
import pytest

import goss_b200 as goss
from goss_b200.codegen.odeparse import parse_ode_text

pytestmark = pytest.mark.gpu

N = 5  # two pairs and an odd state
TEXT = f"states({', '.join(f'x{i}=1.0' for i in range(N))})\n" + "".join(
    f"dx{i}_dt = -0.{i + 1}*x{i}\n" for i in range(N))
VALUES = [np.nan, np.inf, -np.inf, 0.0, 1e-25, 1e-40, 3.3, -85.4321]


def _system(nodes, precision="single"):
    ode = goss.ParameterizedODE(parse_ode_text(TEXT, "nonfinite_states"), field_states=[f"x{i}" for i in range(N)])
    solver = goss.solvers.ExplicitEuler(ode)
    solver.internal_time_step = 0.125
    return goss.ODESystemSolver(nodes, solver, ode, precision=precision)


def test_forwards_of_one_launch_equal_single_forwards():
    rng = np.random.default_rng(1)
    # every value in every place beside ordinary ones, then mixtures
    rows = [np.where(np.arange(N) == i, v, rng.uniform(-100, 100, N)) for v in VALUES for i in range(N)]
    rows += [rng.choice(VALUES, N) for _ in range(200)]
    y0 = np.array(rows)
    a, b = _system(len(rows)), _system(len(rows))
    a.set_states(y0)
    b.set_states(y0)
    t = 0.25 * np.arange(9)
    out = a.solve(t)
    for k in range(1, t.size):
        b.forward(t[k - 1], t[k] - t[k - 1])
        np.testing.assert_array_equal(out[k], b.field_states)
    finite = np.isfinite(y0)
    np.testing.assert_array_equal(np.isfinite(out[-1]), finite)
    assert np.array_equal(np.isnan(out[-1])[np.isnan(y0)], np.ones(np.isnan(y0).sum(), bool))
    # an entry that is not finite leaves the node's others alone
    exact = y0 * (1 - 0.125 * (np.arange(N) + 1) / 10) ** 16
    np.testing.assert_allclose(out[-1][finite], exact[finite], rtol=1e-6, atol=1e-37)
