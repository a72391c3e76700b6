"""``solve`` of a solver class with a ``forward`` of its own goes through it."""
from __future__ import annotations

import numpy as np
import pytest

import goss_b200 as goss

pytestmark = pytest.mark.gpu


def test_solve_calls_a_subclass_forward():
    class Clamped(goss.solvers.RK4):
        calls = 0

        def forward(self, y, t, interval):
            super().forward(y, t, interval)
            Clamped.calls += 1
            y[0] = min(y[0], -50.0)

    ode = goss.ParameterizedODE("fitzhughnagumo")
    plain, clamped = goss.solvers.RK4(ode), Clamped(ode)
    plain.internal_time_step = clamped.internal_time_step = 0.1
    t = np.linspace(0.0, 4.0, 9)
    out = clamped.solve(t)
    assert Clamped.calls == 8 and out[1:, 0].max() == -50.0
    assert plain.solve(t)[1:, 0].max() > -50.0
