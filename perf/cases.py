"""The work that programs have this framework do, as cases to time and compare.

A case is one call pattern of the public entry points on one mechanism: the
drop-in ``Algorithm.solve`` on one group of cells, the device-resident
``Batch`` (each step loop), the copy-overlapped ``solve_host_intervals``,
several mechanisms in one ``MultiBatch``, the constrained RODAS3 system, and a
recorded forward run with its adjoint. Mechanisms are the repository's
synthetic generators' (sizes from 20 species / 40 reactions to 210 / 500) and
the 209-species TS1 tables of its fixtures. A case's mechanism belongs to the
case; its cells (state, temperatures, rate constants) come from the seed.

Fields of a case: ``call`` (the entry point), ``family`` (synthetic, ts1,
dae), ``n``, ``R``, ``mechanism`` (the generator's seed), ``cells``,
``group``, ``loop`` (algorithm, restarting, backward-euler), ``tableau``,
``dt``, ``rtol``, ``spin`` (intervals integrated while preparing: 0 starts a
run cold, at 1e-6 of the interval; 2 continues one whose step is settled) and
``intervals`` of one pass.
"""
import dataclasses
import math

import numpy as np
import torch

from fastode_gb300 import ROS3, RODAS3, Algorithm, BackwardEuler, ChemSystem, Counts, Memory, RestartingLoop
from fastode_gb300 import synthetic
from fastode_gb300.adjoint import adjoint, forward_record
from fastode_gb300.batch import Batch, HostState, solve_host_intervals
from fastode_gb300.multi import MultiBatch, Part
from fastode_gb300.plan import analyze


def _case(name, call, family, n, R, mechanism, cells, spin, intervals, group=32, loop="algorithm", tableau="ros3",
          dt=30.0, rtol=1e-3):
    return dict(name=name, call=call, family=family, n=n, R=R, mechanism=mechanism, cells=cells, group=group,
                loop=loop, tableau=tableau, dt=dt, rtol=rtol, spin=spin, intervals=intervals)


def listed():
    return [
        # the reference's own call on one group of cells, host arrays in and
        # out: the smallest mechanism on a settled step (latency only) ...
        _case("solve_20x40_group", "solve", "synthetic", 20, 40, 1, 32, 2, 1),
        # ... and the full-size mechanism's first call of a run
        _case("solve_210x500_group", "solve", "synthetic", 210, 500, 2, 32, 0, 1),
        # a whole small run: 64 cells x 20 intervals, one launch each
        _case("batch_20x40_64", "batch", "synthetic", 20, 40, 1, 64, 0, 20),
        # the archived TS1 scenario's size: 64 cells, the first intervals
        _case("batch_ts1_64", "batch", "ts1", 209, 547, 0, 64, 0, 8),
        # TS1 on a regional domain, the last group short of cells
        _case("batch_ts1_8200", "batch", "ts1", 209, 547, 0, 8200, 2, 2),
        # the baseline backward Euler on groups that leave lanes idle
        _case("euler_120x260_1000", "batch", "synthetic", 120, 260, 13, 1000, 2, 1, group=24, loop="backward-euler",
              dt=60.0),
        # the cold first interval of a medium run: about twenty attempts
        _case("batch_210x500_16384_cold", "batch", "synthetic", 210, 500, 2, 16384, 0, 1),
        # the headline workload: 65,536 cells, a settled interval
        _case("batch_210x500_65536", "batch", "synthetic", 210, 500, 2, 65536, 2, 1),
        # a host model's loop: host arrays, copies overlapped with the solves
        _case("host_120x260_8192", "host", "synthetic", 120, 260, 13, 8192, 2, 3),
        # three mechanisms in one persistent launch, half the cells in darkness
        _case("multi_196608", "multi", "synthetic", 210, 500, 3, 196608, 2, 1, dt=60.0),
        # RODAS3 with ten quasi-steady species, projection every interval
        _case("dae_160x340_16384", "batch", "dae", 160, 340, 5, 16384, 2, 1, tableau="rodas3", dt=60.0, rtol=1e-4),
        # forward recording and its discrete adjoint (gradients with respect
        # to the initial state and every rate constant)
        _case("adjoint_210x500_4096", "adjoint", "synthetic", 210, 500, 2, 4096, 0, 1),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    call = rng.choice(["solve", "batch", "batch", "batch", "batch", "host", "multi", "adjoint"])
    family = rng.choice(["synthetic", "synthetic", "ts1", "dae"]) if call == "batch" else "synthetic"
    spin = 0 if call == "adjoint" else rng.choice([0, 2])
    n = log(20, 210)
    R = int(n * rng.uniform(1.9, 2.4))
    mechanism = rng.randint(1, 40)
    loop, tableau, group, dt, rtol = "algorithm", "ros3", rng.choice([32, 32, 32, 24, 17]), rng.choice([30.0, 60.0]), 1e-3
    if call in ("multi", "adjoint"):
        group = 32
    if family == "ts1":
        n, R, mechanism = 209, 547, 0
    elif family == "dae":
        n = max(n, 40)
        R, tableau, rtol = 2 * n + 20, "rodas3", 1e-4
    elif call == "batch":
        loop = rng.choice(["algorithm", "algorithm", "restarting", "backward-euler"])
        tableau = rng.choice(["ros3", "rodas3"])
    # the largest run's cells shrink with the work of a cell
    most = int({"solve": 32, "batch": 49152, "host": 16384, "multi": 131072, "adjoint": 4096}[call])
    if call == "batch" and (spin == 0 or loop != "algorithm"):
        most = 8192
    cells = rng.randint(1, group) if call == "solve" else log(40, most)
    return {k: v for k, v in _case("", call, family, n, R, mechanism, cells, spin, rng.choice([1, 2, 3]) if spin else 1,
                                   group, loop, tableau, dt, rtol).items() if k != "name"}


# ---- mechanisms ---------------------------------------------------------------------

class _Tables:
    """The TS1 mechanism from the tables of the repository's fixture."""

    def __init__(self, f):
        self.n, self.R, self.P = int(f["m_n"]), int(f["m_R"]), int(f["m_P"])
        self.react = np.asarray(f["m_react"], dtype=np.int64)
        self.S = np.zeros((self.n, self.R))
        self.S[f["m_S_rows"], f["m_S_cols"]] = f["m_S_vals"]
        self.pattern = type("Pattern", (), {})()
        self.pattern.rows = np.asarray(f["m_rows"], dtype=np.int64)
        self.pattern.cols = np.asarray(f["m_cols"], dtype=np.int64)
        self._map = (np.asarray(f["m_gt_indptr"], np.int32), np.asarray(f["m_gt_indices"], np.int32),
                     np.asarray(f["m_gt_data"], np.float64))

    def jac_csr(self):
        return tuple(a.copy() for a in self._map)


_mechanisms = {}


def _mechanism(case):
    """What a program builds once: the mechanism with its rate parameters."""
    key = (case["call"] == "multi", case["family"], case["n"], case["R"], case["mechanism"])
    if key not in _mechanisms:
        if case["family"] == "ts1":
            f = dict(np.load("tests/golden/ts1_tier1_30s.npz"))
            got = dict(mech=_Tables(f), fixture=f, mass=None)
        elif case["family"] == "dae":
            w = synthetic.dae_constrained(32, 1, case["mechanism"], n_diff=case["n"] - 10, n_alg=10,
                                          n_reactions=case["R"] - 10)
            got = dict(mech=w.sm.mech, sm=w.sm, mass=w.mass)
        elif case["call"] == "multi":
            n, R, s = case["n"], case["R"], case["mechanism"]
            sizes = ((max(20, n * 2 // 7), max(20, R * 2 // 25)), (n * 4 // 7, R * 13 // 25), (n, R))
            got = dict(parts=[synthetic.synthetic_mechanism(a, b, s + 10 * i, third_body_fraction=0.1)
                              for i, (a, b) in enumerate(sizes)])
        else:
            sm = synthetic.synthetic_mechanism(case["n"], case["R"], case["mechanism"],
                                               third_body_fraction=0.0 if case["n"] == 20 else 0.1)
            got = dict(mech=sm.mech, sm=sm, mass=None)
        _mechanisms[key] = got
    return _mechanisms[key]


# ---- inputs, on the GPU from the seed ---------------------------------------------------

DAY = 86400.0


def _uniform(g, lo, hi, *shape):
    return lo + (hi - lo) * torch.rand(*shape, generator=g, dtype=torch.float64, device="cuda")


def _cells(sm, cells, seed, phases):
    """Initial states (cells, n), rate constants (cells, R) in the light of
    t = 0 and the solar phases, distributed as the repository's workloads."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed * 7919 + 13)
    T = _uniform(g, 200.0, 310.0, cells, 1)
    M = 100.0 * _uniform(g, 10.0, 1000.0, cells, 1) / (synthetic.R_GAS * T)
    phase = _uniform(g, -phases, phases, cells)
    Y = 10.0 ** _uniform(g, -15.0, -3.0, cells, sm.n)
    A, E, power = (torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in (sm.A, sm.E, sm.mech.third_body_power))
    k = A * torch.exp(-E / T) * torch.where(power > 0, M, torch.ones_like(M))
    return Y, k, phase


def _light(sm, k, phase, t):
    """Rate constants of an interval that starts at t: photolysis follows the
    diurnal cosine."""
    photo = torch.from_numpy(np.nonzero(sm.photolytic)[0]).cuda()
    f = torch.cos(phase + 2.0 * math.pi * t / DAY).clamp_min(0.0)
    k = k.clone()
    k[:, photo] = torch.from_numpy(sm.J[sm.photolytic]).cuda() * f[:, None]
    return k


def _inputs(case, seed):
    """(Y0 (cells, n), [k (cells, R) of each interval, spin included], atol)."""
    m = _mechanism(case)
    cells, count = case["cells"], case["spin"] + case["intervals"]
    if case["family"] == "ts1":
        f = m["fixture"]
        g = torch.Generator(device="cuda")
        g.manual_seed(seed * 7919 + 29)
        at = torch.randint(len(f["Y0"]), (cells,), generator=g, device="cuda")

        def rows(a, spread):
            a = torch.from_numpy(np.ascontiguousarray(a)).cuda()[at]
            return a * torch.exp(spread * torch.randn(a.shape, generator=g, dtype=torch.float64, device="cuda"))

        Y, k, base = rows(f["Y0"], 0.3), rows(f["k_static"], 0.05), rows(f["base"], 0.1)
        photo, scaling = torch.from_numpy(f["photo"]).cuda(), torch.from_numpy(f["scaling"]).cuda()
        ks = []
        for i in range(count):
            ki = k.clone()
            ki[:, photo] = base * float(f["f"][i]) * scaling
            ks.append(ki)
        return Y, ks, torch.from_numpy(np.asarray(f["atol"], dtype=np.float64)).cuda()
    sm = m["sm"]
    Y, k, phase = _cells(sm, cells, seed, 1.2)
    ks = [_light(sm, k, phase, i * case["dt"]) for i in range(count)]
    return Y, ks, torch.full((sm.n,), case["rtol"] * 1e-14, dtype=torch.float64, device="cuda")


def _solver(case):
    tableau = RODAS3 if case["tableau"] == "rodas3" else ROS3
    if case["loop"] == "backward-euler":
        return BackwardEuler()
    return RestartingLoop(tableau) if case["loop"] == "restarting" else Algorithm(tableau)


# ---- the calls --------------------------------------------------------------------------

def prepare(case, seed):
    m = _mechanism(case)
    return {"solve": _prepare_solve, "batch": _prepare_batch, "host": _prepare_host, "multi": _prepare_multi,
            "adjoint": _prepare_adjoint}[case["call"]](case, seed, m)


def run(state):
    return state["run"](state)


def _prepare_solve(case, seed, m):
    Y, ks, atol = _inputs(case, seed)
    Y, ks, atol = Y.cpu().numpy(), [k.cpu().numpy() for k in ks], atol.cpu().numpy()
    solver, memory = _solver(case), Memory()
    for k in ks[:case["spin"]]:
        Y, _ = solver.solve(ChemSystem(m["mech"], k), Y, case["dt"], atol, case["rtol"], Counts(), memory)
    systems = [ChemSystem(m["mech"], k) for k in ks[case["spin"]:]]
    return dict(run=_run_solve, case=case, solver=solver, Y=Y, atol=atol, systems=systems,
                memory=(memory.h_next, memory.err_prev, memory.h_prev))


def _run_solve(s):
    """The reference's loop over intervals for one group of cells."""
    Y, memory, counts = s["Y"], Memory(*s["memory"]), Counts()
    for system in s["systems"]:
        Y, status = s["solver"].solve(system, Y, s["case"]["dt"], s["atol"], s["case"]["rtol"], counts, memory)
    return {"Y": Y, "memory": np.array([memory.h_next, memory.err_prev, memory.h_prev]),
            "counts": np.array(dataclasses.astuple(counts), dtype=np.int64), "converged": status == "converged"}


def _prepare_batch(case, seed, m):
    Y, ks, atol = _inputs(case, seed)
    batch = Batch(m["mech"], Y, group_size=case["group"], algorithm=_solver(case), mass=m["mass"])
    ks = [k.t().contiguous() for k in ks]
    for k in ks[:case["spin"]]:
        batch.step(k, case["dt"], atol, case["rtol"])
    return dict(run=_run_batch, case=case, batch=batch, ks=ks[case["spin"]:], atol=atol, Y=batch.Y.clone(),
                memory=batch.memory.clone())


def _run_batch(s):
    """Continue (or begin) the run from the state it was left in."""
    b, case = s["batch"], s["case"]
    b.Y.copy_(s["Y"])
    b.memory.copy_(s["memory"])
    b.counts.zero_()
    for k in s["ks"]:
        b.step(k, case["dt"], s["atol"], case["rtol"])
    return {"Y": b.Y, "memory": b.memory, "counts": b.counts, "status": b.status}


def _prepare_host(case, seed, m):
    Y, ks, atol = _inputs(case, seed)
    state = HostState(m["mech"], case["cells"], m["mech"].n, m["mech"].R, case["group"], _solver(case), m["mass"], 0,
                      torch.device("cuda", torch.cuda.current_device()))
    Y, ks, atol = Y.cpu().pin_memory(), [k.cpu().pin_memory() for k in ks], atol.cpu().numpy()
    if case["spin"]:
        Y, _, _ = solve_host_intervals(m["mech"], Y, ks[:case["spin"]], case["dt"], atol, case["rtol"], state=state)
        Y = Y.clone().pin_memory()
    return dict(run=_run_host, case=case, mech=m["mech"], state=state, Y=Y, ks=ks[case["spin"]:], atol=atol,
                memory=state.memory.clone())


def _run_host(s):
    """Host arrays through several intervals, every interval's state read back."""
    case, st, seen = s["case"], s["state"], []
    st.memory.copy_(s["memory"])
    st.counts.zero_()
    solve_host_intervals(s["mech"], s["Y"], s["ks"], case["dt"], s["atol"], case["rtol"], state=st,
                         on_result=lambda i, Y, status: seen.append(Y.clone()))
    return {"Y": seen, "memory": st.memory, "counts": st.counts, "status": st.status_out}


def _multi_inputs(case, seed):
    out = []
    groups = case["cells"] // case["group"]
    for i, sm in enumerate(_mechanism(case)["parts"]):
        g = max(1, groups // 3 + (1 if i < groups % 3 else 0))
        out.append((sm, *_cells(sm, g * case["group"], seed * 3 + i, math.pi)))
    return out


def _prepare_multi(case, seed, m):
    parts = []
    for sm, Y, k, phase in _multi_inputs(case, seed):
        rxn = np.nonzero(sm.photolytic)[0]
        parts.append(Part(sm.mech, Y, k, np.full(sm.n, case["rtol"] * 1e-14), case["rtol"], case["dt"],
                          group_size=case["group"], algorithm=_solver(case),
                          photolysis=(rxn, sm.J[rxn], phase.cpu().numpy())))
    mb = MultiBatch(parts)
    mb.capture()
    mb.reset()
    mb.run(case["spin"])
    return dict(run=_run_multi, case=case, mb=mb, t=mb.t.clone(), kept=[(p.Y.clone(), p.memory.clone()) for p in parts])


def _run_multi(s):
    """Continue (or begin) the run of all mechanisms, a graph per interval."""
    mb = s["mb"]
    for p, (Y, memory) in zip(mb.parts, s["kept"]):
        p.Y.copy_(Y)
        p.memory.copy_(memory)
        p.counts.zero_()
    mb.t.copy_(s["t"])
    mb.run(s["case"]["intervals"])
    return [{"Y": p.Y, "memory": p.memory, "counts": p.counts, "status": p.status} for p in mb.parts]


def _prepare_adjoint(case, seed, m):
    Y, ks, atol = _inputs(case, seed)
    g = torch.Generator(device="cuda")
    g.manual_seed(seed * 7919 + 31)
    return dict(run=_run_adjoint, case=case, mech=m["mech"], Y=Y, ks=[k.t().contiguous() for k in ks], atol=atol,
                weights=torch.randn(m["mech"].n, case["cells"], generator=g, dtype=torch.float64, device="cuda"))


def _run_adjoint(s):
    """The forward run, recorded, and the gradient of sum(weights * log Y)."""
    case = s["case"]
    traj = forward_record(s["mech"], s["Y"], lambda i: s["ks"][i], case["dt"], s["atol"], case["rtol"],
                          case["intervals"], group_size=case["group"], algorithm=_solver(case))
    Y = traj.batch.Y
    lam, log_k = adjoint(traj, s["weights"] / Y.clamp_min(1e-14))
    return {"Y": Y, "dY0": lam * s["Y"].t(), "dlogk": log_k, "counts": traj.batch.counts}


# ---- the work of a pass -----------------------------------------------------------------

_analyses = {}


def _mechanism_work(mech, mass, S):
    """(flops of an attempt of one cell, its n, its R) under a sparse
    elimination order, multiply-adds as two."""
    key = id(mech)
    if key not in _analyses:
        a = analyze(mech, mass=mass)
        rates = 2 * a["R"] * a["P"]
        _analyses[key] = (mech, 2 * a["lu_fma"] + 2 * S * a["solve_fma"] + 2 * a["jac_terms"] + (S - 1) * (rates + 2 * a["stoich_nnz"]))
    return _analyses[key][1], mech.n, mech.R


def work(case):
    m = _mechanism(case)
    stages = {"backward-euler": 1}.get(case["loop"], 4 if case["tableau"] == "rodas3" else 3)
    # attempts of a group: a cold interval grows its step from 1e-6 of the
    # interval in about twenty, a settled one takes one to three
    per = 1.2 if case["loop"] == "algorithm" and case["family"] != "dae" else 3.0
    cold = case["spin"] == 0 or case["loop"] == "restarting"
    attempts = 20.0 + per * (case["intervals"] - 1) if cold else per * case["intervals"]
    if case["call"] == "multi":
        groups = case["cells"] // case["group"]
        of = [(_mechanism_work(sm.mech, None, stages), (groups // 3) * case["group"]) for sm in m["parts"]]
    else:
        of = [(_mechanism_work(m["mech"], m["mass"], stages), case["cells"])]
    flops = sum(c * f for (f, n, R), c in of) * attempts
    nbytes = sum(c * 8.0 * (2 * n + R * case["intervals"]) for (f, n, R), c in of)
    if case["call"] == "adjoint":
        flops, nbytes = 4.0 * flops, 2.0 * nbytes + sum(c * 8.0 * (2 * n + R) for (f, n, R), c in of)
    return {"bytes": nbytes, "flops": flops}


# ---- the same in 64 bits with dense torch ------------------------------------------------

class _Dense:
    """Mass-action forcing and dense Jacobian of cells (..., n)."""

    def __init__(self, mech, mass):
        self.n, self.R, self.P = int(mech.n), int(mech.R), int(mech.P)
        self.react = torch.from_numpy(np.asarray(mech.react)).cuda()
        S = np.asarray(mech.S, dtype=np.float64)
        self.S = torch.from_numpy(S).cuda()
        self.mass = torch.ones(self.n, dtype=torch.float64, device="cuda") if mass is None else \
            torch.from_numpy(np.asarray(mass, dtype=np.float64)).cuda()
        sp, rx = np.nonzero(S)
        self.at, self.of, self.coef = [], [], []
        for p in range(self.P):
            col = np.asarray(mech.react)[rx, p]
            ok = col < self.n
            self.at.append(torch.from_numpy(sp[ok] * self.n + col[ok]).cuda())
            self.of.append(torch.from_numpy(rx[ok]).cuda())
            self.coef.append(torch.from_numpy(S[sp[ok], rx[ok]]).cuda())

    def factors(self, Y):
        one = torch.ones_like(Y[:, :1])
        return torch.cat([Y, one], dim=1)[:, self.react]                    # (cells, R, P)

    def F(self, Y, k):
        return (k * self.factors(Y).prod(dim=2)) @ self.S.T

    def J(self, Y, k):
        x = self.factors(Y)
        out = torch.zeros(Y.shape[0], self.n * self.n, dtype=torch.float64, device="cuda")
        for p in range(self.P):
            d = k
            for q in range(self.P):
                if q != p:
                    d = d * x[:, :, q]
            out = out.index_add(1, self.at[p], d[:, self.of[p]] * self.coef[p])
        return out.view(-1, self.n, self.n)

    def step(self, Y, k, H, tab):
        """One Rosenbrock step of sizes H (cells,): (Y_new, E)."""
        A = torch.diag(self.mass) / (H * tab.gamma)[:, None, None] - self.J(Y, k)
        lu, piv = torch.linalg.lu_factor(A)
        K, force = [], None
        for r in range(len(tab.m)):
            if r == 0 or tab.new_forcing[r]:
                at = Y
                for s in range(r):
                    if tab.a[r, s] != 0.0:
                        at = at + float(tab.a[r, s]) * K[s]
                force = self.F(at, k)
            b = force
            for s in range(r):
                if tab.c[r, s] != 0.0:
                    b = b + (float(tab.c[r, s]) / H)[:, None] * self.mass * K[s]
            K.append(torch.linalg.lu_solve(lu, piv, b[:, :, None])[:, :, 0])
        y, e = Y, torch.zeros_like(Y)
        for r in range(len(tab.m)):
            y = y + float(tab.m[r]) * K[r]
            e = e + float(tab.e[r]) * K[r]
        return y, e

    def project(self, Y, k, atol, rtol, group):
        """Damped Newton on the algebraic rows, group by group."""
        alg = self.mass == 0.0
        index = torch.nonzero(alg)[:, 0]
        G = int(group.max()) + 1

        def most(v):
            return torch.zeros(G, dtype=torch.float64, device="cuda").scatter_reduce(0, group, v.amax(dim=1), "amax")

        def weighted(z, d):
            return most(d.abs() / (atol[index] + rtol * torch.maximum(z.abs(), (z + d).abs())))

        def residual(Y):
            return self.F(Y, k)[:, index]

        todo = torch.ones(G, dtype=torch.bool, device="cuda")
        for _ in range(11):
            A = -self.J(Y, k)[:, index][:, :, index]
            lu, piv = torch.linalg.lu_factor(A)
            d = torch.linalg.lu_solve(lu, piv, residual(Y)[:, :, None])[:, :, 0]
            q = weighted(Y[:, index], d)
            todo = todo & (q > 0.1)
            if not bool(todo.any()):
                break
            step = torch.ones(G, dtype=torch.float64, device="cuda")
            seek, new = todo.clone(), Y.clone()
            for _ in range(25):
                cand = Y.clone()
                cand[:, index] = Y[:, index] + step[group][:, None] * d
                trial = torch.linalg.lu_solve(lu, piv, residual(cand)[:, :, None])[:, :, 0]
                qt = weighted(cand[:, index], trial)
                good = seek & ((qt <= 0.1) | (qt < (1.0 - 1e-4 * step) * q))
                new = torch.where(good[group][:, None], cand, new)
                seek = seek & ~good
                if not bool(seek.any()):
                    break
                step = torch.where(seek, step * 0.5, step)
            Y = new
        return Y


def _quantize(h, dt):
    return dt if h >= dt else dt / max(math.ceil(dt / h - 1e-9), 1)


def _interval(sys, tab, Y, k, dt, atol, rtol, group, sizes, mem, restarting, mass_rows):
    """One interval of every group: each with its own step, all in step rounds.
    Returns (Y, [accepted steps of each group])."""
    G = len(sizes)
    if mass_rows is not None:
        Y = sys.project(Y, k, atol, rtol, group)
    t, H, last_rej, more_rej, accepted, counts = [0.0] * G, [], [False] * G, [False] * G, [[] for _ in range(G)], [0] * G
    for g in range(G):
        h = 1e-6 * dt if restarting or mem[g][0] <= 0.0 else mem[g][0]
        h = min(max(1e-15 * dt, h), dt)
        H.append(h if restarting else _quantize(h, dt))
    live = list(range(G))
    where = [torch.nonzero(group == g)[:, 0] for g in range(G)]
    proposed = list(H)
    while live:
        h_used, short = [], []
        for g in live:
            h, left = H[g], dt - t[g]
            if restarting:
                h_used.append(min(h, left))
                short.append(False)
                continue
            last = left <= h * (1.0 + 1e-8)
            short.append(last and left < h * (1.0 - 1e-8))
            h_used.append(left if last else h)
        rows = torch.cat([where[g] for g in live])
        hs = torch.cat([torch.full((sizes[g],), h, dtype=torch.float64, device="cuda") for g, h in zip(live, h_used)])
        y, e = sys.step(Y[rows], k[rows], hs, tab)
        if restarting and mass_rows is not None:
            e = torch.where(sys.mass == 0.0, y - Y[rows], e)
        w = e / (atol + rtol * torch.maximum(Y[rows].abs(), y.abs()))
        total = torch.zeros(G, dtype=torch.float64, device="cuda").index_add(0, group[rows], (w * w).sum(dim=1)).tolist()
        good, at = [], 0
        for g, h, sh in zip(live, h_used, short):
            err = max(math.sqrt(total[g] / (sizes[g] * sys.n)), 1e-10)
            counts[g] += 1
            ok = err < 1.0
            good += [ok] * sizes[g]
            if restarting:
                fac = min(6.0, max(0.2, 0.9 / err ** (1.0 / 3.0)))
            elif ok:
                fac = 0.9 / err ** (1.0 / 3.0)
                if mem[g][1] > 0.0 and mem[g][2] > 0.0:
                    fac = 0.9 * (err * mem[g][1]) ** (-1.0 / 12.0) * (h / mem[g][2]) ** -0.25
                fac = min(6.0, max(0.2, fac))
            else:
                fac = max(0.2, 0.9 / err ** (1.0 / 3.0))
            if ok:
                accepted[g].append(h)
                done = sh or (not restarting and h == dt - t[g])
                t[g] = dt if done else t[g] + h
                if sh:
                    proposed[g] = H[g]
                else:
                    new = h * fac
                    if last_rej[g]:
                        new = min(new, h)
                    new = max(1e-15 * dt, min(new, dt))
                    H[g] = proposed[g] = new if restarting else _quantize(new, dt)
                    mem[g][1], mem[g][2] = err, h
                last_rej[g] = more_rej[g] = False
            else:
                new = h * 0.1 if more_rej[g] else h * fac
                more_rej[g], last_rej[g] = last_rej[g], True
                H[g] = new if restarting else _quantize(new, dt)
        good = torch.tensor(good, device="cuda")
        Y = Y.index_copy(0, rows, torch.where(good[:, None], y, Y[rows]))
        live = [g for g in live if t[g] - dt + 2.220446049250313e-16 <= 0.0 and counts[g] < 1000]
    for g in range(G):
        mem[g][0] = proposed[g]
    return torch.where(sys.mass == 1.0, Y.clamp_min(0.0), Y), accepted


def _euler(sys, Y, k, dt, atol, rtol, where):
    """Backward Euler with full Newton iterations, group by group."""
    out = Y.clone()
    for rows in where:
        kg, Yn, H, t, wins, cuts = k[rows], Y[rows], dt, 0.0, 0, 0
        it = Yn
        while t < dt:
            ok = False
            for i in range(11):
                A = torch.diag(sys.mass) / H - sys.J(it, kg)
                d = torch.linalg.solve(A, (sys.F(it, kg) - (it - Yn) / H)[:, :, None])[:, :, 0]
                it = (it + d).clamp_min(0.0)
                if i and bool((d.abs() <= torch.maximum(atol, rtol * it.abs()).clamp_min(1e-40)).all()):
                    ok = True
                    break
            if ok:
                t, Yn, wins = t + H, it, wins + 1
                if wins >= 2:
                    wins, H = 0, 2.0 * H
            elif cuts >= 5:
                break
            else:
                it, wins, H, cuts = Yn, 0, H * (0.5, 0.5, 0.5, 0.5, 0.1)[cuts], cuts + 1
            H = min(H, dt - t)
        out[rows] = it
    return out


def exact(case, seed):
    """What ``run`` returns, from dense torch in 64 bits: the integrated state,
    and the gradients of a recorded run."""
    m = _mechanism(case)
    if case["call"] == "multi":
        return None                      # its mechanisms' sizes are those of the batch cases
    n, C = m["mech"].n, case["cells"]
    rounds = (12 if case["loop"] == "backward-euler" else 0) + (25 if case["spin"] == 0 else 35)
    if case["loop"] == "restarting":
        rounds = 25 * (case["spin"] + case["intervals"])
    if case["call"] == "adjoint":
        rounds *= 4
    # batched dense factorizations at some 0.1 TFLOP/s, and their latencies
    if rounds * C * 0.7 * n ** 3 > 4.0e12 or rounds * n * math.ceil(C / case["group"]) > 2.5e6:
        return None
    sys = _Dense(m["mech"], m["mass"])
    Y, ks, atol = _inputs(case, seed)
    dt, rtol = case["dt"], case["rtol"]
    group = torch.arange(C, device="cuda") // case["group"]
    sizes = torch.bincount(group).tolist()
    where = [torch.nonzero(group == g)[:, 0] for g in range(len(sizes))]
    tab = RODAS3 if case["tableau"] == "rodas3" else ROS3
    mem = [[0.0, 0.0, 0.0] for _ in sizes]
    seen, taken = [], []
    for i, k in enumerate(ks):
        start = Y
        if case["loop"] == "backward-euler":
            Y, steps = _euler(sys, Y, k, dt, atol, rtol, where), None
        else:
            Y, steps = _interval(sys, tab, Y, k, dt, atol, rtol, group, sizes, mem, case["loop"] == "restarting",
                                 m["mass"])
        taken.append((start, k, steps))
        if i >= case["spin"]:
            seen.append(Y)
    if case["call"] == "solve":
        return {"Y": Y, "memory": None, "counts": None, "converged": None}
    if case["call"] == "host":
        return {"Y": seen, "memory": None, "counts": None, "status": None}
    if case["call"] == "batch":
        return {"Y": Y.t().contiguous(), "memory": None, "counts": None, "status": None}
    s = _prepare_adjoint(case, seed, m)
    lam = (s["weights"] / Y.t().clamp_min(1e-14)).t().contiguous()
    dk = torch.zeros_like(ks[0])
    for start, k, steps in reversed(taken):
        depth = max(len(v) for v in steps)
        H = torch.tensor([v + [0.0] * (depth - len(v)) for v in steps], dtype=torch.float64, device="cuda")[group]
        ys = [start]
        for d in range(depth):
            on = H[:, d] > 0.0
            y, _ = sys.step(ys[-1], k, torch.where(on, H[:, d], torch.ones_like(H[:, d])), tab)
            ys.append(torch.where(on[:, None], y, ys[-1]))
        lam = torch.where(ys[-1] > 0.0, lam, torch.zeros_like(lam))
        for d in reversed(range(depth)):
            on = H[:, d] > 0.0
            y0 = ys[d].detach().requires_grad_(True)
            theta = torch.zeros_like(k).requires_grad_(True)
            y, _ = sys.step(y0, k * torch.exp(theta), torch.where(on, H[:, d], torch.ones_like(H[:, d])), tab)
            torch.where(on[:, None], y, y0).backward(lam)
            lam = y0.grad
            dk += theta.grad
    return {"Y": Y.t().contiguous(), "dY0": (lam * s["Y"]).t().contiguous(), "dlogk": dk.t().contiguous(), "counts": None}
