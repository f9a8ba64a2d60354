"""The dense square of several blocks (120/260: six, 210/500: twelve) on every
size of team, down to the one-warp elimination and solves that large launches
run (dense_lu_warp, square_triangle in rosenbrock.cuh)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# groups per SM that take clusters (two groups in all) and teams of 16, 8, 4, 2
# and 1 warps (16 warps per SM)
PER_SM = (0, 1, 2, 4, 8, 9)


def pairs_of_groups(torch, per_sm):
    return max(1, per_sm * torch.cuda.get_device_properties(0).multi_processor_count // 2)


def workload(n, R, intervals, cells=64):
    from fastode_gb300 import synthetic as syn
    sm = syn.synthetic_mechanism(n, R, 2, third_body_fraction=0.1)
    cells = syn.synthetic_cells(sm, cells, 17, T_range=(200.0, 310.0), p_range_hpa=(10.0, 1000.0), phase_range=(-1.2, 1.2))
    return syn.Workload(f"ros3-{n}x{R}", sm, cells, 30.0, intervals, 1.0e-3, 32, True)


@pytest.mark.parametrize("n,R,sizes", [(120, 260, PER_SM), (210, 500, (0, 4, 8, 9))])
def test_every_team_gives_the_plain_bits(cuda, n, R, sizes):
    """Two groups' states, Counts and memory with the plain row loops, and
    every copy of them in launches of all team sizes."""
    from fastode_gb300 import Algorithm
    from fastode_gb300.batch import Batch
    torch = cuda
    wl = workload(n, R, 2)
    at = torch.from_numpy(wl.atol).cuda()
    ks = [np.ascontiguousarray(wl.k_at(i).T) for i in range(2)]

    def run(copies, kernel):
        b = Batch(wl.sm.mech, np.tile(wl.cells.Y0, (copies, 1)), algorithm=Algorithm(kernel=kernel))
        for k in ks:
            b.step(torch.from_numpy(np.tile(k, (1, copies))).cuda(), wl.dt, at, wl.rtol)
        torch.cuda.synchronize()
        return (b.Y.view(n, copies, 64).transpose(0, 1), b.memory.view(copies, 2, 3), b.counts.view(copies, 2, 13),
                b.status.view(copies, 2))

    want = [v[:1].clone() for v in run(1, "plain")]
    assert not np.any(want[3].cpu().numpy())
    for per_sm in sizes:
        for got, w in zip(run(pairs_of_groups(torch, per_sm), "generated"), want):
            assert torch.equal(got, w.expand_as(got)), per_sm


def test_adjoint_of_one_warp_teams(cuda, monkeypatch):
    """The transposed solves and the reverse sweep of one warp per group
    against teams of sixteen: every copy of two groups has the same gradients."""
    from fastode_gb300 import adjoint as A
    torch = cuda
    wl = workload(120, 260, 1)
    plain = A._workspace
    monkeypatch.setattr(A, "_workspace", lambda t, keep=False: plain(t, False))
    rng = np.random.default_rng(9)
    lam = rng.standard_normal((wl.sm.n, 64))
    want = None
    for copies in (1, pairs_of_groups(torch, 9)):
        k = torch.from_numpy(np.tile(np.ascontiguousarray(wl.k_at(0).T), (1, copies))).cuda()
        traj = A.forward_record(wl.sm.mech, np.tile(wl.cells.Y0, (copies, 1)), lambda i: k, wl.dt, wl.atol, wl.rtol, 1)
        got = A.adjoint(traj, torch.from_numpy(np.tile(lam, (1, copies))).cuda())
        got = [v.view(-1, copies, 64) for v in got]
        want = got if want is None else want
        for x, y in zip(got, want):
            assert torch.isfinite(x).all() and torch.equal(x, y[:, :1].expand_as(x))
