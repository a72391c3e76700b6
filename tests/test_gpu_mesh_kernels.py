"""FP64 GRL1, GRL2 and RK4 with a thread per node -- the kernels of a mesh --
against the FP64 CPU oracle.

Systems of at most 16 nodes per SM split a node's rows over four warps unless a
block size is set, and a thread per node comes in two register caps chosen by the
number of blocks; every combination is reached here, by the block size or by the
number of nodes.
"""
from __future__ import annotations

import numpy as np
import pytest

import goss_b200 as goss
import pyoracle
from helpers import meta, oracle_model, parity, parity_scaled, perturbed_states, variant_dir

pytestmark = pytest.mark.gpu

TP06, TT04 = "tentusscher_panfilov_2006_M_cell", "tentusscher_2004_mcell"
FIELDS = ("g_Kr", "g_Ks", "g_CaL", "g_to")


def _inputs(model, nodes, seed):
    md = meta(variant_dir(model, FIELDS))
    rng = np.random.default_rng(seed)
    y0 = perturbed_states(oracle_model(model, FIELDS).ic, nodes, rng, 0.05)
    defaults = np.array([md["default_parameters"][i] for i in md["field_parameter_indices"]])
    return y0, defaults[None, :] * np.exp(0.2 * rng.standard_normal((nodes, 4)))


def _system(model, solver, ldt, y0, fp, block):
    ode = goss.ParameterizedODE(model, field_parameters=list(FIELDS), field_states=["V"])
    s = goss.solvers.solver_mapper[solver](ode)
    s.internal_time_step = ldt
    system = goss.ODESystemSolver(y0.shape[0], s, ode)
    system.set_block_size(block)
    system.set_states(y0)
    system.field_parameters = fp
    return system


def _oracle(model, solver, ldt, y0, fp):
    o = pyoracle.OracleSystem(oracle_model(model, FIELDS), solver, y0.shape[0], ldt=ldt)
    o.states[:] = y0
    o.field_params[:] = fp
    return o


# 64: the smaller register cap; 128: the larger one (a system this small)
@pytest.mark.parametrize("block", [64, 128])
@pytest.mark.parametrize("solver, dt, ldt", [("GRL1", 0.5, 0.01), ("GRL2", 0.5, 0.05), ("RK4", 0.5, 0.001)])
@pytest.mark.parametrize("model", [TP06, TT04])
def test_stimulus_and_upstroke(model, solver, dt, ldt, block):
    """20 ms, 37 nodes, the bar of the small systems' test."""
    y0, fp = _inputs(model, 37, 11)
    system, o = _system(model, solver, ldt, y0, fp, block), _oracle(model, solver, ldt, y0, fp)
    for k in range(40):
        system.forward(k * dt, dt)
        assert o.forward(k * dt, dt) == 0
    assert parity(system.states, o.states) <= 1.0


# the smaller cap by the block size; the larger one on more nodes than are split
@pytest.mark.parametrize("nodes, block", [(2048, 64), (2449, 0)])
@pytest.mark.parametrize("solver, bar", [("GRL1", 1e-10), ("GRL2", 1e-9)])
def test_lognormal_fields_100ms(nodes, block, solver, bar):
    """The workload and the bars of the 2,048-node test of small systems."""
    y0, fp = _inputs(TP06, nodes, 1234)
    system, o = _system(TP06, solver, 0.01, y0, fp, block), _oracle(TP06, solver, 0.01, y0, fp)
    for k in range(10):
        system.forward(10.0 * k, 10.0)
        o.forward(10.0 * k, 10.0)
    assert parity(system.states, o.states, rtol=bar) <= 1.0


@pytest.mark.parametrize("solver, ldt, t0", [("GRL1", 0.01, 9.9), ("GRL2", 0.01, 9.9), ("RK4", 0.0005, 10.0)])
@pytest.mark.parametrize("model", [TP06, TT04])
def test_mesh_of_50021_nodes(model, solver, ldt, t0):
    """A ragged mesh whose blocks take the smaller cap, a piece of it that takes
    the larger one, other blocks, and every 997th node by the oracle (GRL2, whose
    increment keeps the exponential form at every coefficient, is no nearer than
    1e-9 to it halfway up an upstroke; the tests above hold it after one)."""
    nodes, piece, steps = 50_021, 20_000, 200
    y0, fp = _inputs(model, nodes, 3)
    states = []
    for n, block in ((nodes, 0), (piece, 0), (nodes, 96)):
        system = _system(model, solver, ldt, y0[:n], fp[:n], block)
        system.forward(t0, steps * ldt)
        states.append(system.states)
    np.testing.assert_array_equal(states[0][:piece], states[1])
    np.testing.assert_array_equal(states[0], states[2])
    if solver == "GRL2":
        return
    some = np.r_[0:nodes:997, nodes - 1]
    o = _oracle(model, solver, ldt, y0[some], fp[some])
    o.forward(t0, steps * ldt)
    # V passes zero on the way up: its error against 1 % of its range
    assert parity_scaled(states[0][some], o.states) <= 1.0


@pytest.mark.parametrize("model", [TP06, TT04])
def test_rk4_does_not_depend_on_the_split(model):
    y0, fp = _inputs(model, 1000, 8)
    states = []
    for block in (0, 64):
        system = _system(model, "RK4", 0.0005, y0, fp, block)
        system.forward(9.95, 0.1)  # into the stimulus
        system.solve(np.array([10.05, 10.1, 10.15]))
        states.append(system.states)
    np.testing.assert_array_equal(*states)


@pytest.mark.parametrize("delta", [0.0, 1e-320])
def test_a_delta_below_the_split_stays_with_a_thread_per_node(delta):
    y0, fp = _inputs(TP06, 33, 8)
    states = []
    for block in (0, 64):
        system = _system(TP06, "GRL1", 0.01, y0, fp, block)
        system.solver.set_parameter("delta", delta)
        system.forward(10.0, 0.5)
        states.append(system.states)
    np.testing.assert_array_equal(*states)
