"""Teams of warps per group: the launch chooses 16, 8, 4, 2 or 1 warps by the
number of groups, and results must not depend on it; and the drop-in call's
kept buffers, which calls of other shapes and on other threads must not share.
"""
import threading

import numpy as np
import pytest

from golden_cases import load, mechanism_of, table_mechanism

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case,groups", [("ros3_20x40", (2, 200, 400, 800, 1600)), ("rodas3_chapman_qssa", (1, 170, 320, 640, 1280)),
                                         ("ros3_210x500_subset", (8, 168, 312))])
@pytest.mark.parametrize("lockstep", [True, False])
def test_results_do_not_depend_on_the_team(cuda, case, groups, lockstep):
    """The same cells repeated until the launch takes the next smaller team:
    every copy of a group gets the bits of the smallest launch."""
    from fastode_gb300 import RODAS3, ROS3, Algorithm
    from fastode_gb300.batch import Batch
    torch = cuda
    f = load(case)
    dae = case.startswith("rodas3")
    mech = table_mechanism(f) if dae else mechanism_of(f)
    C0 = f["Y0"].shape[0]
    k0 = f["k"] if dae else f["k"][0] if "k" in f else f["k0"]
    k0 = np.broadcast_to(k0, (C0, mech.R))
    size = 32 if C0 >= 32 else C0
    want = None
    for g in groups:
        copies = -(-g * size // C0)
        b = Batch(mech, np.tile(f["Y0"], (copies, 1)), group_size=size, mass=f["mass"] if dae else None,
                  algorithm=Algorithm(RODAS3 if dae else ROS3, lockstep=lockstep))
        atol = torch.from_numpy(np.ascontiguousarray(np.broadcast_to(f["atol"], (mech.n,)))).cuda()
        k = torch.from_numpy(np.ascontiguousarray(np.tile(k0, (copies, 1)).T)).cuda()
        for _ in range(2):
            b.step(k, float(f["dt"]), atol, float(f["rtol"]))
        torch.cuda.synchronize()
        got = (b.Y.view(mech.n, copies, C0), b.memory.view(copies, -1, 3), b.counts.view(copies, -1, 13))
        if want is None:
            want = [v.clone() for v in (got[0][:, 0], got[1][0], got[2][0])]
        assert torch.equal(got[0], want[0][:, None].expand_as(got[0])), g
        assert torch.equal(got[1], want[1][None].expand_as(got[1])), g
        assert torch.equal(got[2], want[2][None].expand_as(got[2])), g


@pytest.mark.parametrize("case,intervals", [("ros3_20x40", 3), ("rodas3_dae_160x340", 2)])
def test_adjoint_with_and_without_kept_steps(cuda, case, intervals, monkeypatch):
    """The reverse sweep on the replay's kept steps gives the bits of the one
    that computes every step again."""
    from fastode_gb300 import RODAS3, ROS3, Algorithm, adjoint as A
    torch = cuda
    f = load(case)
    dae = "mass" in f
    mech = mechanism_of(f)
    ks = [torch.from_numpy(np.ascontiguousarray(f["k"][i].T)).cuda() for i in range(intervals)]
    traj = A.forward_record(mech, f["Y0"], lambda i: ks[i], float(f["dt"]), f["atol"], float(f["rtol"]), intervals,
                            algorithm=Algorithm(RODAS3 if dae else ROS3), mass=f["mass"] if dae else None)
    lam = torch.from_numpy(np.random.default_rng(3).standard_normal(traj.batch.Y.shape)).cuda() / traj.batch.Y.clamp_min(1e-14)
    sizes, plain = [], A._workspace

    def spy(t, keep=False):
        ws = plain(t, keep)
        sizes.append(ws.numel())
        return ws

    monkeypatch.setattr(A, "_workspace", spy)
    kept = A.adjoint(traj, lam)
    monkeypatch.setattr(A, "_workspace", lambda t, keep=False: spy(t, False))
    again = A.adjoint(traj, lam)
    assert sizes[0] > sizes[1]
    for x, y in zip(kept, again):
        assert torch.equal(x, y)


def test_dropin_calls_share_no_buffers(cuda):
    """Drop-in calls of several shapes in turn, and from four threads on their
    own streams, against the same calls one at a time."""
    from fastode_gb300 import Algorithm, ChemSystem, Counts, Memory
    torch = cuda
    f = load("ros3_20x40")
    mech = mechanism_of(f)

    def call(lo, hi, single_k=False):
        k = f["k"][0][lo:lo + 1] if single_k else f["k"][0][lo:hi]
        mem, counts = Memory(), Counts()
        Y = f["Y0"][lo:hi]
        for _ in range(3):
            Y, status = Algorithm().solve(ChemSystem(mech, k), Y, float(f["dt"]), f["atol"], float(f["rtol"]), counts, mem)
        return Y, (mem.h_next, mem.err_prev, mem.h_prev), counts, status

    jobs = [(0, 32), (32, 64), (0, 7), (5, 37), (40, 41), (0, 32, True), (8, 24, True)]
    want = [call(*j) for j in jobs]
    got = [[None] * len(jobs) for _ in range(4)]

    def work(t):
        with torch.cuda.stream(torch.cuda.Stream()):
            for q in range(len(jobs)):
                i = (q + t) % len(jobs)
                got[t][i] = call(*jobs[i])

    threads = [threading.Thread(target=work, args=(t,)) for t in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for t in range(4):
        for w, g in zip(want, got[t]):
            np.testing.assert_array_equal(w[0], g[0])
            assert w[1:] == g[1:]


def test_few_reactions_and_many_species(cuda):
    """Four reactions with hundreds of products: enough work for a cluster, but
    fewer rates than a cluster's blocks exchange values. Two groups and 400
    (one-block teams) of the same cells give the same bits."""
    from fastode_gb300 import BackwardEuler, Mechanism
    from fastode_gb300.batch import Batch
    from fastode_gb300.plan import analyze
    torch = cuda
    n, rng = 600, np.random.default_rng(11)
    names = [f"S{i}" for i in range(n)]
    mech = Mechanism(names, [([names[2 * j], names[2 * j + 1]], [(s, 0.01 * (1 + i % 7)) for i, s in enumerate(names[8:])])
                             for j in range(4)])
    a = analyze(mech)
    assert a["lu_fma"] + 3 * a["solve_fma"] + a["jac_terms"] + 2 * a["stoich_nnz"] > 10000
    Y0, k0 = 10.0 ** rng.uniform(-9, -3, (64, n)), 10.0 ** rng.uniform(0, 3, (64, 4))
    got = []
    for copies in (1, 200):
        b = Batch(mech, np.tile(Y0, (copies, 1)), group_size=32, algorithm=BackwardEuler())
        atol = torch.full((n,), 1e-17, dtype=torch.float64, device="cuda")
        k = torch.from_numpy(np.ascontiguousarray(np.tile(k0, (copies, 1)).T)).cuda()
        for _ in range(2):
            b.step(k, 30.0, atol, 1e-3)
        got.append((b.Y.view(n, copies, 64).clone(), b.counts.view(copies, 2, 13).clone()))
    assert torch.equal(got[1][0], got[0][0].expand_as(got[1][0]))
    assert torch.equal(got[1][1], got[0][1].expand_as(got[1][1]))


@pytest.mark.parametrize("slots", [0, 700])
def test_rounds_with_groups_that_end_early(cuda, slots):
    """Groups that fail in the middle of a round (a NaN rate constant), cold
    and settled ones, one block per group (more than are resident, so that
    blocks join rounds under way) and a queue: the bits of a run without
    rounds."""
    from fastode_gb300 import Algorithm, synthetic as syn
    from fastode_gb300.batch import Batch
    torch = cuda
    groups = 2600
    sm = syn.synthetic_mechanism(48, 100, 3)
    wl = syn.Workload("ros3-48x100", sm, syn.synthetic_cells(sm, 32 * groups, 5), 30.0, 2, 1.0e-3, 32, False)
    at = torch.from_numpy(wl.atol).cuda()
    k = [torch.from_numpy(np.ascontiguousarray(wl.k_at(i).T)).cuda() for i in range(2)]
    k[1] = k[1].clone()
    k[1][:, ::32 * 7] = float("nan")      # every seventh group fails at its first attempt
    out = []
    for lockstep in (True, False):
        b = Batch(wl.sm.mech, wl.cells.Y0, group_size=32, slots=slots, algorithm=Algorithm(lockstep=lockstep))
        b.step(k[0], wl.dt, at, wl.rtol)
        b.memory[::3] = 0.0               # every third group starts cold again
        b.step(k[1], wl.dt, at, wl.rtol)
        torch.cuda.synchronize()
        out.append((b.state(), b.counts.cpu().numpy(), b.memory.cpu().numpy(), b.status.cpu().numpy()))
    assert len(set(out[0][3])) == 2
    for x, y in zip(*out):
        np.testing.assert_array_equal(x, y)
