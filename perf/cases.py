"""Performance cases: the work a user of this framework has it do, through its
public entry points.

A case is a dict of plain values; ``listed()`` gives the fixed ones, ``draw``
more of the same ranges, ``prepare`` what a user's program holds before the
call, ``run`` one pass, ``work`` the bytes and operations a pass cannot do
without, and ``exact`` the result in plain 64-bit torch from the models'
published equations.

Kinds of work:

* ``cell``      one cell, ``solver.solve(times, y0)``
* ``tissue``    ``ODESystemSolver.forward`` of a device-resident population
* ``exchange``  a PDE code's step with host copies: field states in, forward,
                field states out
* ``coupled``   the same step with the PDE vector on the device
* ``batch``     several populations of different models in one captured graph
* ``gradient``  a trace misfit and its adjoint (forward and backward)
* ``implicit``  one interval of an implicit solver

Single-precision mode keeps float64 arrays whose values carry single
precision: its results are taken as float32, as a program stores them.
"""
from __future__ import annotations

import math

import numpy as np
import torch

TP06, TT04, FHN = "tentusscher_panfilov_2006_M_cell", "tentusscher_2004_mcell", "fitzhughnagumo"
FIELDS = {TP06: ["g_Kr", "g_Ks", "g_CaL", "g_to"], TT04: ["g_Kr", "g_Ks", "g_CaL", "g_to"], FHN: ["a", "b"]}
IMPLICIT_FIELDS = ["g_Kr", "g_CaL"]  # the fields of the implicit solvers' variants of TT04
LDT = 0.01  # ms, internal step of the cell models
FINE = 0.0005  # ms, with the solvers that are not exponential (the sodium gates' time constants are below 0.001 ms)


def _ldt(solver):
    return LDT if solver.startswith("GRL") else FINE


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # the smallest call: one two-state cell over ten output intervals (a
        # notebook's first run); latency, launches and host work only
        dict(name="cell_fhn", kind="cell", model=FHN, solver="RK4", ldt=0.1, interval=0.5, intervals=10),
        # one ventricular cell, the way single-cell studies use a solver object
        dict(name="cell_tp06", kind="cell", model=TP06, solver="GRL1", ldt=LDT, interval=1.0, intervals=10),
        # the benchmark's workload: 2^20 nodes, 1000 steps a call, single precision
        dict(name="tissue_single_1m", kind="tissue", model=TP06, solver="GRL1", precision="single", nodes=1 << 20,
             interval=10.0),
        # the default precision on a tissue patch
        dict(name="tissue_double_262k", kind="tissue", model=TP06, solver="GRL1", precision="double", nodes=262_144,
             interval=1.0),
        # an odd mesh driven by a host PDE code, V in and out every 0.5 ms, default precision
        dict(name="exchange_double_50k", kind="exchange", model=TP06, solver="GRL1", precision="double",
             nodes=50_021, interval=0.5),
        # a device PDE code over two populations of an odd mesh, one operator-splitting step of 0.1 ms
        dict(name="coupled_single_100k", kind="coupled", precision="single", nodes=100_003, share=0.72,
             interval=0.1),
        # five populations of three models, 100 one-step forwards in one captured graph
        dict(name="batch_single_492k", kind="batch", precision="single", nodes=492_003, forwards=100),
        # parameter identification: gradient of a V-trace misfit, single precision
        dict(name="gradient_single_65k", kind="gradient", solver="GRL1", precision="single", nodes=65_536,
             intervals=10, tape_gb=6),
        # the same in double precision with RK4 on a small odd patch, recomputing from checkpoints
        dict(name="gradient_double_2k", kind="gradient", solver="RK4", precision="double", nodes=2_001, intervals=2,
             tape_gb=0),
        # implicit solvers on unstimulated cells relaxing from perturbed states (every pass
        # alike): the default theta rule with forward differences on a tissue patch,
        dict(name="theta_262k", kind="implicit", solver="ThetaSolver", jacobian=False, nodes=262_144, min_dt=1e-4),
        # implicit Euler with the generated Jacobian on an odd patch,
        dict(name="implicit_euler_20k", kind="implicit", solver="ImplicitEuler", jacobian=True, nodes=20_011,
             min_dt=1e-4),
        # and the adaptive solver where it accepts its steps
        dict(name="esdirk_65k", kind="implicit", solver="ESDIRK23a", jacobian=True, nodes=65_536, min_dt=1e-4),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["cell", "tissue", "tissue", "tissue", "exchange", "coupled", "batch", "gradient", "implicit",
                       "implicit"])
    precision = rng.choice(["single", "double"])
    single = precision == "single"
    if kind == "cell":
        model = rng.choice([FHN, TP06, TT04])
        if model == FHN:
            return dict(kind=kind, model=model, solver=rng.choice(["RK4", "ExplicitEuler"]), ldt=0.1,
                        interval=rng.randint(1, 20) / 10, intervals=rng.randint(2, 20))
        return dict(kind=kind, model=model, solver=rng.choice(["GRL1", "GRL2"]), ldt=LDT,
                    interval=rng.randint(10, 100) / 100, intervals=rng.randint(2, 10))
    if kind in ("tissue", "exchange"):
        solver = rng.choice(["GRL1", "GRL1", "GRL2", "RK4", "ExplicitEuler"])
        evals = {"GRL1": 1, "GRL2": 2, "RK4": 4, "ExplicitEuler": 1}[solver]
        nodes = _log(rng, 100, 1 << 20)
        steps = min(1000, int((1e9 if single else 1.2e8) / evals / nodes))
        steps = _log(rng, 10, max(10, min(steps, 1000 if single else 200)))
        if nodes * steps * evals > (1e9 if single else 1.2e8):
            nodes = int(1.2e8 / evals / steps)
        return dict(kind=kind, model=rng.choice([TP06, TT04]), solver=solver, precision=precision, nodes=nodes,
                    interval=steps * _ldt(solver))
    if kind == "coupled":
        return dict(kind=kind, precision=precision, nodes=_log(rng, 2_000, 300_000),
                    share=rng.randint(10, 90) / 100, interval=rng.randint(5, 20) / 100)
    if kind == "batch":
        return dict(kind=kind, precision=precision, nodes=_log(rng, 10_000, 490_000 if single else 100_000),
                    forwards=rng.randint(10, 100))
    if kind == "gradient":
        solver = rng.choice(["GRL1", "RK4"])
        return dict(kind=kind, solver=solver, precision=precision,
                    nodes=_log(rng, 500, (65_000 if single else 8_000) // (1 if solver == "GRL1" else 4)),
                    intervals=rng.randint(1, 4), tape_gb=rng.choice([0, 2]))
    solver = rng.choice(["ThetaSolver", "ImplicitEuler", "ESDIRK23a"])
    return dict(kind=kind, solver=solver, jacobian=rng.choice([False, True]),
                nodes=_log(rng, 1_000, 60_000 if solver == "ESDIRK23a" else 262_000), min_dt=1e-4)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _patch(model, nodes, seed, fields, salt=0):
    """States at the initial conditions +-5 % and fields with a spread of 20 %
    (conductances; FitzHugh-Nagumo and the implicit workload: +-5 %)."""
    rng = np.random.default_rng([seed, salt])
    m = MODELS[model]
    y0 = m.ic[None, :] * (1.0 + rng.uniform(-0.05, 0.05, (nodes, m.ic.size)))
    base = np.array([m.params[f] for f in fields])
    if model == FHN or fields == IMPLICIT_FIELDS:
        fp = base * (1.0 + rng.uniform(-0.05, 0.05, (nodes, len(fields))))
    else:
        fp = base * np.exp(0.2 * rng.standard_normal((nodes, len(fields))))
    return y0, fp


def _start(seed):
    """Model time of the first call: around the stimulus (10 to 11 ms), so
    upstrokes are among what the solvers meet."""
    return 9.5 + 0.01 * (seed % 100)


def _populations(case):
    """Populations of a batch: model, nodes."""
    n = case["nodes"]
    parts = [(FHN, 3), (FHN, n // 10), (TT04, int(0.35 * n)), (TP06, int(0.03 * n))]
    return parts + [(TP06, n - sum(k for _, k in parts))]


def _inputs(case, seed):
    kind = case["kind"]
    if kind == "cell":
        y0, _ = _patch(case["model"], 1, seed, FIELDS[case["model"]])
        t = _start(seed) if case["model"] != FHN else 0.0
        return y0[0], t + case["interval"] * np.arange(case["intervals"] + 1)
    if kind in ("tissue", "exchange"):
        y0, fp = _patch(case["model"], case["nodes"], seed, FIELDS[case["model"]])
        v = np.random.default_rng([seed, 7]).uniform(-88.0, -80.0, (case["nodes"], 1))
        return y0, fp, v
    if kind == "coupled":
        n = case["nodes"]
        a = max(1, int(case["share"] * n))
        rng = np.random.default_rng([seed, 8])
        order = rng.permutation(n)
        pops = {lab: (model, *_patch(model, k, seed, FIELDS[model], salt), order[at:at + k])
                for lab, model, k, at, salt in (("M", TP06, a, 0, 1), ("old", TT04, n - a, a, 2)) if k}
        return pops, rng.uniform(-88.0, -80.0, n)
    if kind == "batch":
        return [(model, *_patch(model, k, seed, FIELDS[model], i)) for i, (model, k) in enumerate(_populations(case))]
    if kind == "gradient":
        y0, fp = _patch(TP06, case["nodes"], seed, FIELDS[TP06])
        target = np.random.default_rng([seed, 9]).normal(-80.0, 5.0, (case["intervals"], case["nodes"]))
        return y0, fp, target
    return _patch(TT04, case["nodes"], seed, IMPLICIT_FIELDS)


class _Rows:
    """A device array of a solver, for torch.as_tensor; keeps the solver, which owns the memory."""

    def __init__(self, owner, ptr, shape, ld):
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=shape, typestr="<f8", data=(ptr, False), version=3,
                                             strides=(8 * ld, 8), stream=None)


def _states_view(system):
    ptr, ld = system.device_states()
    return torch.as_tensor(_Rows(system, ptr, (system.ode.num_states, system.num_nodes), ld), device="cuda")


def _system(model, solver, y0, fp, fields, precision="double", ldt=LDT, field_states=(), jacobian=False, **more):
    import goss_b200 as goss

    ode = goss.ParameterizedODE(model, field_parameters=fields, field_states=list(field_states),
                                code_params={"generate_jacobian": True} if jacobian else None)
    if model == TT04 and fields == FIELDS[TT04]:
        ode.set_parameter("stim_amplitude", MODELS[TT04].params["stim_amplitude"])
    s = goss.solvers.solver_mapper[solver](ode)
    if ldt:
        s.internal_time_step = ldt
    for k, v in more.items():
        s.set_parameter(k, v)
    system = goss.ODESystemSolver(y0.shape[0], s, ode, precision=precision)
    system.set_states(y0)
    system.field_parameters = fp
    return system


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def prepare(case, seed):
    import goss_b200 as goss

    kind, st = case["kind"], dict(case=case, t=_start(seed))
    x = _inputs(case, seed)
    if kind == "cell":
        ode = goss.ParameterizedODE(case["model"])
        if case["model"] == TT04:
            ode.set_parameter("stim_amplitude", MODELS[TT04].params["stim_amplitude"])
        st["solver"] = goss.solvers.solver_mapper[case["solver"]](ode)
        st["solver"].internal_time_step = case["ldt"]
        st["y0"], st["times"] = x
    elif kind in ("tissue", "exchange"):
        y0, fp, v = x
        st["system"] = _system(case["model"], case["solver"], y0, fp, FIELDS[case["model"]], case["precision"],
                               _ldt(case["solver"]), ["V"])
        st["states"] = _states_view(st["system"])
        if kind == "exchange":
            host = torch.empty(v.shape, dtype=torch.float64, pin_memory=True)  # page-locked, as a PDE code keeps it
            st["host"], st["v"] = host, host.numpy()
            st["v"][:] = v
    elif kind == "coupled":
        from goss_b200.coupling import FieldStateCoupling

        pops, v = x
        systems = {lab: _system(m, "GRL1", y0, fp, FIELDS[m], case["precision"], field_states=["V"])
                   for lab, (m, y0, fp, _) in pops.items()}
        st["v"], st["views"] = torch.tensor(v, device="cuda"), [_states_view(s) for s in systems.values()]
        st["coupling"] = FieldStateCoupling(systems, {lab: p[3] for lab, p in pops.items()}, case["nodes"])
    elif kind == "batch":
        systems = [_system(m, "RK4" if m == FHN else "GRL1", y0, fp, FIELDS[m], case["precision"])
                   for m, y0, fp in x]
        st["systems"], st["views"] = systems, [_states_view(s) for s in systems]
        st["batch"] = goss.BatchSolver(systems)
        st["batch"].capture(st["t"], LDT, case["forwards"])
    elif kind == "gradient":
        from goss_b200 import adjoint

        y0, fp, target = x
        make = adjoint.GRL1Trace if case["solver"] == "GRL1" else adjoint.RK4Trace
        ode = goss.ParameterizedODE(TP06, field_parameters=FIELDS[TP06])
        st["trace"] = make(ode, case["nodes"], 100 * _ldt(case["solver"]), 100, case["intervals"], 100,
                           precision=case["precision"], t0=st["t"], tape_bytes=case["tape_gb"] << 30)
        st["fields"] = torch.tensor(fp, device="cuda", requires_grad=True)
        st["y0"] = torch.tensor(y0, device="cuda", requires_grad=True)
        st["target"] = torch.tensor(target, device="cuda")
    else:
        y0, fp = x
        st["system"] = _system(TT04, case["solver"], y0, fp, IMPLICIT_FIELDS, ldt=0, jacobian=case["jacobian"],
                               min_dt=case["min_dt"])
        st["states"] = _states_view(st["system"])
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    single = case.get("precision") == "single"
    if kind == "cell":
        return st["solver"].solve(st["times"], st["y0"])
    if kind == "tissue":
        st["system"].forward(st["t"], case["interval"])
        st["t"] += case["interval"]
        return st["states"].float() if single else st["states"]
    if kind == "exchange":
        st["system"].field_states = st["v"]
        st["system"].forward(st["t"], case["interval"])
        st["t"] += case["interval"]
        st["system"].get_field_states(out=st["v"])
        if single:
            return dict(field_states=st["v"].astype(np.float32), states=st["states"].float())
        return dict(field_states=st["v"], states=st["states"])
    if kind == "coupled":
        st["coupling"].step((st["t"], st["t"] + case["interval"]), st["v"])
        st["t"] += case["interval"]
        out = dict(pde=st["v"], states=st["views"])
        return dict(pde=out["pde"].float(), states=[x.float() for x in out["states"]]) if single else out
    if kind == "batch":
        st["batch"].replay()
        return [v.float() if single else v for v in st["views"]]
    if kind == "gradient":
        from goss_b200 import adjoint

        v = adjoint.trace(st["trace"], st["fields"], st["y0"])
        gf, gy = torch.autograd.grad(((v - st["target"]) ** 2).sum(), (st["fields"], st["y0"]))
        out = dict(trace=v.detach(), grad_fields=gf, grad_states=gy)
        return {k: x.float() for k, x in out.items()} if single else out
    st["system"].forward(st["t"], 0.1)
    st["t"] += 0.1
    return st["states"]


# ---------------------------------------------------------------------------
# the least a pass can do
# ---------------------------------------------------------------------------
#: floating-point operations of one evaluation, an exponential or a division
#: counted as one: right-hand side, and right-hand side with linear terms
_OPS = {TP06: (650, 950), TT04: (600, 850), FHN: (25, 40)}


def _step_ops(model, solver):
    rhs, lin = _OPS[model]
    n = MODELS[model].ic.size
    return {"GRL1": lin + 6 * n, "GRL2": 2 * (lin + 6 * n), "RK4": 4 * (rhs + 3 * n),
            "ExplicitEuler": rhs + 2 * n}[solver]


def work(case):
    kind = case["kind"]
    if kind == "cell":
        steps = round(case["interval"] / case["ldt"]) * case["intervals"]
        return dict(bytes=8 * MODELS[case["model"]].ic.size * (case["intervals"] + 2),
                    flops=steps * _step_ops(case["model"], case["solver"]))
    nodes = case["nodes"]
    if kind in ("tissue", "exchange"):
        n = MODELS[case["model"]].ic.size
        return dict(bytes=nodes * 8 * (2 * n + 4 + (2 if kind == "exchange" else 0)),
                    flops=nodes * round(case["interval"] / _ldt(case["solver"])) * _step_ops(case["model"], case["solver"]))
    if kind == "coupled":
        return dict(bytes=nodes * 8 * (2 * 18 + 4 + 2),
                    flops=nodes * round(case["interval"] / LDT) * _step_ops(TP06, "GRL1"))
    if kind == "batch":
        return dict(bytes=sum(k * 8 * (2 * MODELS[m].ic.size + len(FIELDS[m])) for m, k in _populations(case)),
                    flops=case["forwards"] * sum(k * _step_ops(m, "RK4" if m == FHN else "GRL1")
                                                 for m, k in _populations(case)))
    if kind == "gradient":
        # the forward step, and a reverse sweep of twice its operations
        return dict(bytes=nodes * 8 * (2 * 19 + 2 * 4 + 2 * case["intervals"]),
                    flops=3 * nodes * 100 * case["intervals"] * _step_ops(TP06, case["solver"]))
    # three Newton iterations a stage at least, a right-hand side, a Jacobian of twice that and a solve each
    stages = {"ThetaSolver": 1, "ImplicitEuler": 1, "ESDIRK23a": 3 * 5}[case["solver"]]
    return dict(bytes=nodes * 8 * (2 * 17 + 2), flops=nodes * stages * 3 * (3 * _OPS[TT04][0] + 300))


# ---------------------------------------------------------------------------
# the models' published equations in plain 64-bit torch
# ---------------------------------------------------------------------------
def _re(x):
    return x.real if x.is_complex() else x


def _where(c, a, b):
    a, b = (z if torch.is_tensor(z) else torch.full(c.shape, float(z), dtype=torch.float64, device=c.device)
            for z in (a, b))
    if a.is_complex() != b.is_complex():
        a, b = a.to(torch.complex128), b.to(torch.complex128)
    return torch.where(c, a, b)


_e = torch.exp


class _TenTusscher:
    """What the 2004 and the 2006 M-cell models share."""

    def reversals(self, Ca_i, Na_i, K_i):
        p = self.params
        rtf = p["R"] * p["T"] / p["F"]
        return (rtf * torch.log(p["Na_o"] / Na_i), rtf * torch.log(p["K_o"] / K_i),
                rtf * torch.log((p["K_o"] + p["P_kna"] * p["Na_o"]) / (K_i + p["P_kna"] * Na_i)),
                0.5 * rtf * torch.log(p["Ca_o"] / Ca_i))

    def common_gates(self, V):
        """Xr1, Xr2, m, h, j, d: steady state and time constant."""
        low = _re(V) < -40.0
        ah = _where(low, 0.057 * _e(-(V + 80.0) / 6.8), 0.0)
        bh = _where(low, 2.7 * _e(0.079 * V) + 310000.0 * _e(0.3485 * V), 0.77 / (0.13 * (1 + _e(-(V + 10.66) / 11.1))))
        aj = _where(low, (-25428.0 * _e(0.2444 * V) - 6.948e-6 * _e(-0.04391 * V)) * (V + 37.78)
                    / (1 + _e(0.311 * (V + 79.23))), 0.0)
        bj = _where(low, 0.02424 * _e(-0.01052 * V) / (1 + _e(-0.1378 * (V + 40.14))),
                    0.6 * _e(0.057 * V) / (1 + _e(-0.1 * (V + 32.0))))
        h_inf = 1 / (1 + _e((V + 71.55) / 7.43)) ** 2
        return dict(
            Xr1=(1 / (1 + _e((-26.0 - V) / 7.0)),
                 450.0 / (1 + _e((-45.0 - V) / 10.0)) * 6.0 / (1 + _e((V + 30.0) / 11.5))),
            Xr2=(1 / (1 + _e((V + 88.0) / 24.0)),
                 3.0 / (1 + _e((-60.0 - V) / 20.0)) * 1.12 / (1 + _e((V - 60.0) / 20.0))),
            m=(1 / (1 + _e((-56.86 - V) / 9.03)) ** 2,
               1 / (1 + _e((-60.0 - V) / 5.0)) * (0.1 / (1 + _e((V + 35.0) / 5.0)) + 0.1 / (1 + _e((V - 50.0) / 200.0)))),
            h=(h_inf, 1 / (ah + bh)), j=(h_inf, 1 / (aj + bj)),
            s=(1 / (1 + _e((V + 20.0) / 5.0)),
               85.0 * _e(-(V + 45.0) ** 2 / 320.0) + 5.0 / (1 + _e((V - 20.0) / 5.0)) + 3.0),
            r=(1 / (1 + _e((20.0 - V) / 6.0)), 9.5 * _e(-(V + 40.0) ** 2 / 1800.0) + 0.8),
            d_tau=(1.4 / (1 + _e((-35.0 - V) / 13.0)) + 0.25) * 1.4 / (1 + _e((V + 5.0) / 5.0))
            + 1 / (1 + _e((50.0 - V) / 20.0)))

    def membrane(self, g, F, Ca_i, Na_i, V, K_i):
        """Currents of the membrane but I_CaL: K1, Kr, Ks, Na, bNa, bCa, to, NaK, NaCa, pCa, pK."""
        p = {**self.params, **F}
        E_Na, E_K, E_Ks, E_Ca = self.reversals(Ca_i, Na_i, K_i)
        frt = p["F"] / (p["R"] * p["T"])
        a = 0.1 / (1 + _e(0.06 * (V - E_K - 200.0)))
        b = (3.0 * _e(0.0002 * (V - E_K + 100.0)) + _e(0.1 * (V - E_K - 10.0))) / (1 + _e(-0.5 * (V - E_K)))
        root = math.sqrt(p["K_o"] / 5.4)
        e1, e2 = _e(p["gamma"] * V * frt), _e((p["gamma"] - 1.0) * V * frt)
        return dict(
            K1=p["g_K1"] * (a / (a + b)) * root * (V - E_K), Kr=p["g_Kr"] * root * g["Xr1"] * g["Xr2"] * (V - E_K),
            Ks=p["g_Ks"] * g["Xs"] ** 2 * (V - E_Ks), Na=p["g_Na"] * g["m"] ** 3 * g["h"] * g["j"] * (V - E_Na),
            bNa=p["g_bna"] * (V - E_Na), bCa=p["g_bca"] * (V - E_Ca), to=p["g_to"] * g["r"] * g["s"] * (V - E_K),
            NaK=p["P_NaK"] * p["K_o"] / (p["K_o"] + p["K_mk"]) * Na_i / (Na_i + p["K_mNa"])
            / (1 + 0.1245 * _e(-0.1 * V * frt) + 0.0353 * _e(-V * frt)),
            NaCa=p["K_NaCa"] * (e1 * Na_i ** 3 * p["Ca_o"] - e2 * p["Na_o"] ** 3 * Ca_i * p["alpha"])
            / ((p["Km_Nai"] ** 3 + p["Na_o"] ** 3) * (p["Km_Ca"] + p["Ca_o"]) * (1 + p["K_sat"] * e2)),
            pCa=p["g_pCa"] * Ca_i / (Ca_i + p["K_pCa"]), pK=p["g_pK"] * (V - E_K) / (1 + _e((25.0 - V) / 5.98)))

    def stimulus(self, t):
        p = self.params
        if t is None:  # the implicit workload: unstimulated cells
            return 0.0
        phase = t - math.floor(t / p["stim_period"]) * p["stim_period"]
        return -p["stim_amplitude"] if p["stim_start"] <= phase <= p["stim_start"] + p["stim_duration"] else 0.0

    def f(self, y, t, F):
        g = dict(zip(self.gate_names, y))
        return self.gates(y, False) + self.pools(g, y, t, F)

    def linear(self, y, t, F):
        """d f_i / d y_i: -1/tau of the gates, a complex step for the others."""
        n, k = len(y), len(self.gate_names)
        lin = self.gates(y, True)
        eye = torch.eye(n - k, dtype=torch.float64, device=y[0].device)[:, :, None] * 1e-30
        z = list(y[:k]) + [torch.complex(y[k + i].expand(n - k, -1).contiguous(),
                                         eye[:, i].expand(-1, y[0].numel()).contiguous()) for i in range(n - k)]
        f = self.pools(dict(zip(self.gate_names, z)), z, t, F)
        lin += [(f[i].expand(n - k, -1))[i].imag / 1e-30 for i in range(n - k)]
        return self.amend(lin, y)

    def amend(self, lin, y):
        return lin


class _TP06(_TenTusscher):
    gate_names = ["Xr1", "Xr2", "Xs", "m", "h", "j", "d", "f", "f2", "fCass", "s", "r"]
    ic = np.array([0.0165, 0.473, 0.0174, 0.00165, 0.749, 0.6788, 3.288e-05, 0.7026, 0.9526, 0.9942, 0.999998,
                   2.347e-08, 0.000153, 0.8978, 4.272, 0.00042, 10.132, -85.423, 138.52])
    params = dict(
        P_kna=0.03, g_K1=5.405, g_Kr=0.153, g_Ks=0.098, g_Na=14.838, g_bna=0.00029, g_CaL=3.98e-05, g_bca=0.000592,
        g_to=0.294, K_mNa=40.0, K_mk=1.0, P_NaK=2.724, K_NaCa=1000.0, K_sat=0.1, Km_Ca=1.38, Km_Nai=87.5, alpha=2.5,
        gamma=0.35, K_pCa=0.0005, g_pCa=0.1238, g_pK=0.0146, Buf_c=0.2, Buf_sr=10.0, Buf_ss=0.4, Ca_o=2.0, EC=1.5,
        K_buf_c=0.001, K_buf_sr=0.3, K_buf_ss=0.00025, K_up=0.00025, V_leak=0.00036, V_rel=0.102, V_sr=0.001094,
        V_ss=5.468e-05, V_xfer=0.0038, Vmax_up=0.006375, k1_prime=0.15, k2_prime=0.045, k3=0.06, k4=0.005, max_sr=2.5,
        min_sr=1.0, Na_o=140.0, Cm=0.185, F=96485.3415, R=8314.472, T=310.0, V_c=0.016404, stim_amplitude=52.0,
        stim_duration=1.0, stim_period=1000.0, stim_start=10.0, K_o=5.4)

    def gates(self, y, linear):
        V, Ca_ss = y[17], y[15]
        c = self.common_gates(V)
        q = 1 / (1 + (Ca_ss / 0.05) ** 2)
        c.update(
            Xs=(1 / (1 + _e((-5.0 - V) / 14.0)),
                1400.0 / torch.sqrt(1 + _e((5.0 - V) / 6.0)) / (1 + _e((V - 35.0) / 15.0)) + 80.0),
            d=(1 / (1 + _e((-8.0 - V) / 7.5)), c["d_tau"]),
            f=(1 / (1 + _e((V + 20.0) / 7.0)), 1102.5 * _e(-(V + 27.0) ** 2 / 225.0) + 200.0 / (1 + _e((13.0 - V) / 10.0))
               + 180.0 / (1 + _e((V + 30.0) / 10.0)) + 20.0),
            f2=(0.67 / (1 + _e((V + 35.0) / 7.0)) + 0.33, 562.0 * _e(-(V + 27.0) ** 2 / 240.0)
                + 31.0 / (1 + _e((25.0 - V) / 10.0)) + 80.0 / (1 + _e((V + 30.0) / 10.0))),
            fCass=(0.6 * q + 0.4, 80.0 * q + 2.0))
        return [-1 / c[k][1] if linear else (c[k][0] - y[i]) / c[k][1] for i, k in enumerate(self.gate_names)]

    def release(self, R_prime, Ca_SR, Ca_ss):
        p = self.params
        kc = p["max_sr"] - (p["max_sr"] - p["min_sr"]) / (1 + (p["EC"] / Ca_SR) ** 2)
        k1 = p["k1_prime"] / kc
        O = k1 * Ca_ss ** 2 * R_prime / (p["k3"] + k1 * Ca_ss ** 2)
        return O, p["V_rel"] * O * (Ca_SR - Ca_ss), p["k2_prime"] * kc

    def pools(self, g, y, t, F):
        p = {**self.params, **F}
        Ca_i, R_prime, Ca_SR, Ca_ss, Na_i, V, K_i = y[12:]
        I = self.membrane(g, F, Ca_i, Na_i, V, K_i)
        frt = p["F"] / (p["R"] * p["T"])
        w = _where(_re(V - 15.0).abs() < 0.01, 0.01 + 0 * V, V - 15.0)
        ex = _e(2 * w * frt)
        CaL = p["g_CaL"] * g["d"] * g["f"] * g["f2"] * g["fCass"] * 4 * w * p["F"] * frt \
            * (0.25 * Ca_ss * ex - p["Ca_o"]) / (ex - 1)
        up, leak = p["Vmax_up"] / (1 + p["K_up"] ** 2 / Ca_i ** 2), p["V_leak"] * (Ca_SR - Ca_i)
        _, rel, k2 = self.release(R_prime, Ca_SR, Ca_ss)
        xfer = p["V_xfer"] * (Ca_ss - Ca_i)
        cap, stim = p["Cm"] / (p["V_c"] * p["F"]), self.stimulus(t)
        bc = 1 / (1 + p["Buf_c"] * p["K_buf_c"] / (Ca_i + p["K_buf_c"]) ** 2)
        bsr = 1 / (1 + p["Buf_sr"] * p["K_buf_sr"] / (Ca_SR + p["K_buf_sr"]) ** 2)
        bss = 1 / (1 + p["Buf_ss"] * p["K_buf_ss"] / (Ca_ss + p["K_buf_ss"]) ** 2)
        return [
            bc * ((leak - up) * p["V_sr"] / p["V_c"] + xfer - (I["bCa"] + I["pCa"] - 2 * I["NaCa"]) * cap / 2),
            -k2 * Ca_ss * R_prime + p["k4"] * (1 - R_prime),
            bsr * (up - rel - leak),
            bss * (-CaL * p["Cm"] / (2 * p["V_ss"] * p["F"]) + rel * p["V_sr"] / p["V_ss"]
                   - xfer * p["V_c"] / p["V_ss"]),
            -(I["Na"] + I["bNa"] + 3 * I["NaK"] + 3 * I["NaCa"]) * cap,
            -(I["K1"] + I["to"] + I["Kr"] + I["Ks"] + CaL + I["NaK"] + I["Na"] + I["bNa"] + I["NaCa"] + I["bCa"]
              + I["pK"] + I["pCa"] + stim),
            -(I["K1"] + I["to"] + I["Kr"] + I["Ks"] - 2 * I["NaK"] + I["pK"] + stim) * cap]

    def amend(self, lin, y):
        # the model generator's linearisation counts the release's dependence
        # on Ca_ss through the open probability twice
        p = self.params
        R_prime, Ca_SR, Ca_ss = y[13], y[14], y[15]
        kc = p["max_sr"] - (p["max_sr"] - p["min_sr"]) / (1 + (p["EC"] / Ca_SR) ** 2)
        k1 = p["k1_prime"] / kc
        dO = 2 * k1 * Ca_ss * R_prime * p["k3"] / (p["k3"] + k1 * Ca_ss ** 2) ** 2
        bss = 1 / (1 + p["Buf_ss"] * p["K_buf_ss"] / (Ca_ss + p["K_buf_ss"]) ** 2)
        lin[15] = lin[15] + bss * p["V_sr"] / p["V_ss"] * p["V_rel"] * (Ca_SR - Ca_ss) * dO
        return lin


class _TT04(_TenTusscher):
    gate_names = ["Xr1", "Xr2", "Xs", "m", "h", "j", "d", "f", "fCa", "s", "r", "g"]
    ic = np.array([0.0, 1.0, 0.0, 0.0, 0.75, 0.75, 0.0, 1.0, 1.0, 1.0, 0.0, 1.0, 0.0002, 0.2, 11.6, -86.2, 138.3])
    # stimulated as the 2006 model is (the model file's default amplitude is 0, kept for the implicit workload)
    params = dict(
        P_kna=0.03, g_K1=5.405, g_Kr=0.096, g_Ks=0.062, g_Na=14.838, g_bna=0.00029, g_CaL=0.000175, g_bca=0.000592,
        g_to=0.294, K_mNa=40.0, K_mk=1.0, P_NaK=1.362, K_NaCa=1000.0, K_sat=0.1, Km_Ca=1.38, Km_Nai=87.5, alpha=2.5,
        gamma=0.35, K_pCa=0.0005, g_pCa=0.825, g_pK=0.0146, Buf_c=0.15, Buf_sr=10.0, Ca_o=2.0, K_buf_c=0.001,
        K_buf_sr=0.3, K_up=0.00025, V_leak=8e-05, V_sr=0.001094, Vmax_up=0.000425, a_rel=0.016464, b_rel=0.25,
        c_rel=0.008232, tau_g=2.0, Na_o=140.0, Cm=0.185, F=96485.3415, R=8314.472, T=310.0, V_c=0.016404,
        stim_amplitude=52.0, stim_duration=1.0, stim_period=1000.0, stim_start=10.0, K_o=5.4)

    def gates(self, y, linear):
        V, Ca_i = y[15], y[12]
        c = self.common_gates(V)
        fCa_inf = (1 / (1 + (Ca_i / 0.000325) ** 8) + 0.1 / (1 + _e((Ca_i - 0.0005) / 0.0001))
                   + 0.2 / (1 + _e((Ca_i - 0.00075) / 0.0008)) + 0.23) / 1.46
        g_inf = _where(_re(Ca_i) < 0.00035, 1 / (1 + (Ca_i / 0.00035) ** 6), 1 / (1 + (Ca_i / 0.00035) ** 16))
        c.update(
            Xs=(1 / (1 + _e((-5.0 - V) / 14.0)),
                1100.0 / torch.sqrt(1 + _e((-10.0 - V) / 6.0)) / (1 + _e((V - 60.0) / 20.0))),
            d=(1 / (1 + _e((-5.0 - V) / 7.5)), c["d_tau"]),
            f=(1 / (1 + _e((V + 20.0) / 7.0)),
               1125.0 * _e(-(V + 27.0) ** 2 / 240.0) + 80.0 + 165.0 / (1 + _e((25.0 - V) / 10.0))),
            fCa=(fCa_inf, 2.0), g=(g_inf, self.params["tau_g"]))
        out = []
        for i, k in enumerate(self.gate_names):
            inf, tau = c[k]
            v = (-1 / tau if torch.is_tensor(tau) else torch.full_like(_re(y[i]), -1 / tau)) if linear \
                else (inf - y[i]) / tau
            if k in ("fCa", "g"):  # these two only fall while the membrane is depolarised
                v = 2 * v if linear else v  # the generator's rule counts this chain twice
                v = _where((_re(V) > -60.0) & (_re(inf) > _re(y[i])), 0.0, v)
            out.append(v)
        return out

    def pools(self, g, y, t, F):
        p = {**self.params, **F}
        Ca_i, Ca_SR, Na_i, V, K_i = y[12:]
        I = self.membrane(g, F, Ca_i, Na_i, V, K_i)
        frt = p["F"] / (p["R"] * p["T"])
        ex = _e(2 * V * frt)
        CaL = p["g_CaL"] * g["d"] * g["f"] * g["fCa"] * 4 * V * p["F"] * frt \
            * (Ca_i * ex - 0.341 * p["Ca_o"]) / (ex - 1)
        up, leak = p["Vmax_up"] / (1 + p["K_up"] ** 2 / Ca_i ** 2), p["V_leak"] * (Ca_SR - Ca_i)
        rel = (p["a_rel"] * Ca_SR ** 2 / (p["b_rel"] ** 2 + Ca_SR ** 2) + p["c_rel"]) * g["d"] * g["g"]
        cap, stim = p["Cm"] / (p["V_c"] * p["F"]), self.stimulus(t)
        bc = 1 / (1 + p["Buf_c"] * p["K_buf_c"] / (Ca_i + p["K_buf_c"]) ** 2)
        bsr = 1 / (1 + p["Buf_sr"] * p["K_buf_sr"] / (Ca_SR + p["K_buf_sr"]) ** 2)
        return [
            bc * (leak - up + rel - (CaL + I["bCa"] + I["pCa"] - 2 * I["NaCa"]) * cap / 2),
            bsr * p["V_c"] / p["V_sr"] * (up - rel - leak),
            -(I["Na"] + I["bNa"] + 3 * I["NaK"] + 3 * I["NaCa"]) * cap,
            -(I["K1"] + I["to"] + I["Kr"] + I["Ks"] + CaL + I["NaK"] + I["Na"] + I["bNa"] + I["NaCa"] + I["bCa"]
              + I["pK"] + I["pCa"] + stim),
            -(I["K1"] + I["to"] + I["Kr"] + I["Ks"] - 2 * I["NaK"] + I["pK"] + stim) * cap]


class _FHN:
    ic = np.array([-85.0, 0.0])
    params = dict(V_peak=40.0, V_rest=-85.0, a=0.13, b=0.013, c_1=0.26, c_2=0.1, c_3=1.0, stim_amplitude=50.0,
                  stim_duration=1.0, stim_start=1.0)

    def f(self, y, t, F):
        p = {**self.params, **F}
        V, s = y
        amp = p["V_peak"] - p["V_rest"]
        th = p["V_rest"] + p["a"] * amp
        current = -p["c_2"] * s * (V - p["V_rest"]) / amp \
            + p["c_1"] * (V - p["V_rest"]) * (V - th) * (p["V_peak"] - V) / amp ** 2
        on = 1 - 1 / (1 + math.exp(min(5 * (t - p["stim_start"]), 700.0)))
        stim = p["stim_amplitude"] * on / (1 + math.exp(min(5 * (t - p["stim_start"] - p["stim_duration"]), 700.0)))
        return [current + stim, p["b"] * (V - p["V_rest"] - p["c_3"] * s)]


MODELS = {TP06: _TP06(), TT04: _TT04(), FHN: _FHN()}


def _advance(model, solver, y, fp, fields, t, interval, ldt):
    """``forward(t, interval)`` of an explicit solver: lists of tensors, one per state."""
    m = MODELS[model]
    F = {k: fp[:, i] for i, k in enumerate(fields)}
    steps = math.ceil(interval / ldt - 1e-12)
    h = interval / steps

    def grl(at, half):
        f, a = m.f(at, t, F), m.linear(at, t, F)
        return [x + torch.where(c == 0, half * b, b / c * torch.expm1(c * half)) for x, b, c in zip(y, f, a)]

    for _ in range(steps):
        if solver == "GRL1":
            y = grl(y, h)
        elif solver == "GRL2":
            half = grl(y, 0.5 * h)
            y = grl(half, h)
        elif solver == "ExplicitEuler":
            y = [x + h * k for x, k in zip(y, m.f(y, t, F))]
        else:
            k1 = m.f(y, t, F)
            k2 = m.f([x + 0.5 * h * k for x, k in zip(y, k1)], t + 0.5 * h, F)
            k3 = m.f([x + 0.5 * h * k for x, k in zip(y, k2)], t + 0.5 * h, F)
            k4 = m.f([x + h * k for x, k in zip(y, k3)], t + h, F)
            y = [x + h / 6 * (a + 2 * b + 2 * c + d) for x, a, b, c, d in zip(y, k1, k2, k3, k4)]
        t += h
    return y


def _implicit(y0, fp, h, theta):
    """One step of the theta rule on unstimulated TT04 by Newton's method with a complex-step Jacobian."""
    m = MODELS[TT04]
    F = {k: fp[:, i] for i, k in enumerate(IMPLICIT_FIELDS)}
    n = len(y0)
    eye = torch.eye(n, dtype=torch.float64, device=fp.device)
    explicit = [(1 - theta) * f for f in m.f(y0, None, F)]
    z = torch.zeros((fp.shape[0], n), dtype=torch.float64, device=fp.device)
    for _ in range(10):
        y = [y0[i] + z[:, i] for i in range(n)]
        f = m.f(y, None, F)
        r = torch.stack([h * (explicit[i] + theta * f[i]) for i in range(n)], 1) - z
        jac = torch.empty((fp.shape[0], n, n), dtype=torch.float64, device=fp.device)
        for j in range(n):
            c = [torch.complex(x, torch.full_like(x, 1e-30 if k == j else 0.0)) for k, x in enumerate(y)]
            for i, q in enumerate(m.f(c, None, F)):
                jac[:, i, j] = q.imag / 1e-30 if q.is_complex() else 0.0
        z = z + torch.linalg.solve(eye - h * theta * jac, r.unsqueeze(-1)).squeeze(-1)
    return torch.stack([y0[i] + z[:, i] for i in range(n)])


def exact(case, seed):
    kind, t = case["kind"], _start(seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    x = _inputs(case, seed)
    cols = lambda a: list(torch.tensor(a, device=dev).t().contiguous())  # noqa: E731
    ten = lambda a: torch.tensor(a, device=dev)  # noqa: E731
    if kind == "cell":
        y0, times = x
        y, out = cols(y0[None, :]), [torch.tensor(y0)]
        fields = FIELDS[case["model"]]
        fp = ten(np.array([[MODELS[case["model"]].params[f] for f in fields]]))
        for a, b in zip(times[:-1], times[1:]):
            y = _advance(case["model"], case["solver"], y, fp, fields, a, b - a, case["ldt"])
            out.append(torch.cat(y).cpu())
        return torch.stack(out)
    if kind in ("tissue", "exchange"):
        y0, fp, v = x
        ldt = _ldt(case["solver"])
        cost = case["nodes"] * case["interval"] / ldt * {"GRL2": 2, "RK4": 2}.get(case["solver"], 1)
        if cost > 1.5e8:
            return None  # minutes in plain torch
        y, iv = cols(y0), 17 if case["model"] == TP06 else 15
        if kind == "exchange":
            y[iv] = ten(v[:, 0])
        y = _advance(case["model"], case["solver"], y, ten(fp), FIELDS[case["model"]], t, case["interval"], ldt)
        y = torch.stack(y)
        return dict(field_states=y[iv][:, None].cpu(), states=y) if kind == "exchange" else y
    if kind == "coupled":
        pops, v = x
        v = ten(v)
        out, states = v.clone(), []
        for model, y0, fp, dofs in pops.values():
            y, iv, at = cols(y0), 17 if model == TP06 else 15, ten(dofs)
            y[iv] = v[at]
            y = _advance(model, "GRL1", y, ten(fp), FIELDS[model], t, (t + case["interval"]) - t, LDT)
            out[at] = y[iv]
            states.append(torch.stack(y))
        return dict(pde=out, states=states)
    if kind == "batch":
        out = []
        for model, y0, fp in x:
            y = cols(y0)
            for k in range(case["forwards"]):
                y = _advance(model, "RK4" if model == FHN else "GRL1", y, ten(fp), FIELDS[model], t + k * LDT, LDT, LDT)
            out.append(torch.stack(y))
        return out
    if kind == "gradient":
        y0, fp, target = x
        with_grad = case["solver"] == "RK4" and case["nodes"] * case["intervals"] <= 5_000
        if not with_grad and case["solver"] == "RK4":
            return None
        fields, start = ten(fp).requires_grad_(with_grad), ten(y0).requires_grad_(with_grad)
        y, rows = [start[:, i] for i in range(19)], []
        ldt = _ldt(case["solver"])
        for j in range(case["intervals"]):
            y = _advance(TP06, case["solver"], y, fields, FIELDS[TP06], t + j * 100 * ldt, 100 * ldt, ldt)
            rows.append(y[17])
        trace = torch.stack(rows)
        if not with_grad:  # a second derivative of the linear terms has no plain form here
            return dict(trace=trace, grad_fields=None, grad_states=None)
        gf, gy = torch.autograd.grad(((trace - ten(target)) ** 2).sum(), (fields, start))
        return dict(trace=trace.detach(), grad_fields=gf, grad_states=gy)
    if case["solver"] == "ESDIRK23a":
        return None  # the adaptive controller's accepted solution is not the equations' own
    y0, fp = x
    return _implicit(cols(y0), ten(fp), 0.1, 0.5 if case["solver"] == "ThetaSolver" else 1.0)
