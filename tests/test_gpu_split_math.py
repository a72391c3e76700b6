"""FP64 arithmetic of the split model programs: reciprocal, exponentials,
logarithm, square root and the GRL increment, through explicit steps of small
models, against extended precision.

One ExplicitEuler step of length 1 from x = 0 leaves x = f(y), so a model with
``dx_dt = f(y)`` and a constant state y returns the function itself.
"""
from __future__ import annotations

import numpy as np
import pytest

import goss_b200 as goss
from goss_b200.codegen.odeparse import parse_ode_text

pytestmark = pytest.mark.gpu

FUNCTIONS = """
parameters(k=1.0)
states(rcp=0.0, div=0.0, ex=0.0, ex2=0.0, lg=0.0, sq=0.0, y=1.0)
drcp_dt = 1/y
ddiv_dt = Conditional(Gt(y, 0), 3.7/y, -3.7/y)
dex_dt = exp(k*y)
dex2_dt = exp(3*y)
dlg_dt = log(y)
dsq_dt = sqrt(y)
dy_dt = 0*y
"""
NAMES = ["rcp", "div", "ex", "ex2", "lg", "sq"]


def _evaluate(y):
    ode = goss.ParameterizedODE(parse_ode_text(FUNCTIONS, "split_math"))
    solver = goss.solvers.ExplicitEuler(ode)
    solver.internal_time_step = 1.0
    system = goss.ODESystemSolver(y.size, solver, ode)
    y0 = np.zeros((y.size, ode.num_states))
    iy = ode.state_names.index("y")
    y0[:, iy] = y
    system.set_states(y0)
    system.forward(0.0, 1.0)
    s = system.states
    return {k: s[:, ode.state_names.index(k)] for k in NAMES}


def _reference(y):
    v = y.astype(np.longdouble)
    with np.errstate(all="ignore"):
        return dict(rcp=1 / v, div=np.where(y > 0, 1, -1) * (np.longdouble(3.7) / v), ex=np.exp(v), ex2=np.exp(3 * v),
                    lg=np.log(v), sq=np.sqrt(v))


@pytest.mark.parametrize("low, high", [(1e-300, 1e300), (1e-8, 700.0), (0.5, 2.0), (0.7071, 1.4143)])
@pytest.mark.parametrize("sign", [1.0, -1.0])
def test_functions_against_extended_precision(low, high, sign):
    rng = np.random.default_rng(11)
    y = sign * np.exp(rng.uniform(np.log(low), np.log(high), 4096))
    got, ref = _evaluate(y), _reference(y)
    # one rounding for the reciprocal and the quotient, one and the function's
    # own for the others; exp(3 y) also rounds its argument 3 log2(e) y once
    # and the constant 3 log2(e) once: |3 y| ulps of the result
    ulps = dict(rcp=1.0, div=1.0, ex=2.0, ex2=2.0 + 2.0 * np.abs(3 * y), lg=2.0, sq=1.0)
    for k in NAMES:
        r = np.asarray(ref[k], dtype=np.float64)
        # inside the normal range with room for the saturation at its ends
        ok = np.isfinite(r) & (np.abs(r) > 1e-307) & (np.abs(r) < 2e307)
        err = np.abs(got[k][ok].astype(np.longdouble) - ref[k][ok]) / np.spacing(np.abs(r[ok]))
        assert np.all(err <= np.broadcast_to(ulps[k], y.shape)[ok]), (k, float(err.max()))
        assert np.array_equal(np.isnan(got[k]), np.isnan(r)), k


def test_special_operands():
    y = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 1e-310, -1e-310, 5e-324, 710.0, -760.0, 1e30, -1e30, 1e300,
                  -1e300, 1.0])
    got, ref = _evaluate(y), _reference(y)
    for k in NAMES:
        r = np.asarray(ref[k], dtype=np.float64)
        np.testing.assert_allclose(got[k], r, rtol=1e-15, atol=1e-305, err_msg=k)


def test_exponential_increment():
    """x' = a x + 0.3: every branch of the GRL1 increment (polynomial,
    exponential, Euler below delta) in steps from 1e-9 to 60 time constants."""
    ode = goss.ParameterizedODE(parse_ode_text(
        "states(x=1.0, a=-1.0)\ndx_dt = a*x + 0.3\nda_dt = 0*a\n", "split_grl"))
    a = np.concatenate([-np.logspace(-9, np.log10(60.0), 500), np.logspace(-9, 1, 200),
                        [-0.125, np.nextafter(-0.125, 0), 0.125, 0.0, -1e-310, -1e-8, -1.0000001e-8]])
    s = goss.solvers.GRL1(ode)
    s.internal_time_step = 1.0
    system = goss.ODESystemSolver(a.size, s, ode)
    system.set_states(np.stack([np.full(a.size, 2.0), a], axis=1))
    system.forward(0.0, 1.0)
    got = system.states[:, 0]
    al = a.astype(np.longdouble)
    f = al * 2 + np.longdouble(0.3)
    with np.errstate(all="ignore"):
        ref = np.asarray(2 + np.where(al == 0, f, f * np.expm1(al) / np.where(al == 0, 1, al)), float)
    # the increment f (e^a - 1)/a keeps the rounding of e^a, 2^-53 max(1, e^a),
    # divided by a (Euler below 1e-8: relative error a/2); ten roundings of the
    # result beside it
    rounding = np.maximum(1, np.exp(np.minimum(a, 50))) * 2.0 ** -53 / np.maximum(np.abs(a), 1e-300)
    quant = np.abs(np.asarray(f, float)) * np.where(np.abs(a) > 1e-8, rounding, 1e-8)
    tol = 4 * np.minimum(quant, np.abs(ref) + 2) + 2e-15 * (np.abs(ref) + 2)
    assert np.all(np.abs(got - ref) <= tol)


@pytest.mark.parametrize("states", [1, 2, 21, 22])  # no pair, one pair, a full group and an odd state, two groups
@pytest.mark.parametrize("solver", ["GRL1", "GRL2"])
def test_single_precision_increment(states, solver):
    """x_i' = a_i x_i + 0.3 in single precision, a_i from 1e-4 to 40 per step on
    both sides of the polynomial's range, the states side by side in pairs."""
    a = -np.logspace(-4, np.log10(40.0), states) if states > 1 else np.array([-0.2])
    a = np.where(np.arange(states) % 3 == 2, np.minimum(-a, 3.0), a)
    text = f"states({', '.join(f'x{i}=2.0' for i in range(states))})\n"
    text += "".join(f"dx{i}_dt = {float(a[i])!r}*x{i} + 0.3\n" for i in range(states))
    ode = goss.ParameterizedODE(parse_ode_text(text, f"split_single_{states}"))
    s = goss.solvers.solver_mapper[solver](ode)
    s.internal_time_step = 1.0
    system = goss.ODESystemSolver(33, s, ode, precision="single")
    system.forward(0.0, 1.0)
    f = 2 * a + 0.3
    if solver == "GRL2":
        f = a * (2 + f * np.expm1(a / 2) / a) + 0.3
    ref = 2 + f * np.expm1(a) / a
    # right-hand side and product in FP32 (6e-8 each of |a x| + 0.3), phi1 at
    # worst the cancellation of e^x - 1 next to |x| = 1/4 (1.2e-7 / 0.22); GRL2
    # carries the half step's error through a
    scale = (np.abs(a) * np.maximum(2, np.abs(ref)) + 0.3) * np.expm1(a) / a
    tol = 3e-6 * scale * (1 + (np.abs(a) if solver == "GRL2" else 0)) + 1e-12
    got = system.states
    assert np.all(got == got[0])  # every node of a warp and of the ragged block
    assert np.all(np.abs(got[0] - ref) <= tol)
