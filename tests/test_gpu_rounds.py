"""Lockstep rounds (rosenbrock.cuh), which run from one and a half blocks per
SM and with 5,000 operations an attempt or more: that they run where a test
means them to is read from the rounds' words in the workspace."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# the workspace's header: the queue counter, then a state of 32 bytes for each
# of 256 SMs, whose first word holds the meetings above bit 16
HEADER, ROUNDS = 256, 8192


def clear_rounds(b):
    b.ws[:HEADER + ROUNDS].zero_()


def meetings(torch, b):
    """The meetings per SM since the last launch began."""
    words = b.ws[HEADER:HEADER + ROUNDS].view(torch.int32).view(-1, 8)[:, 0]
    return (words.cpu().numpy().view(np.uint32) >> 16).astype(np.int64)


def sm_count(torch):
    return torch.cuda.get_device_properties(0).multi_processor_count


def test_a_failed_attempt_ends_its_round(cuda):
    """Groups whose first attempt fails (a NaN rate constant) leave both of
    the round's meetings behind them, as any attempt does, so that the blocks'
    later groups meet the others before the solves and not after them: every SM
    that held a block has held whole rounds, two meetings each."""
    from fastode_gb300 import Algorithm, synthetic as syn
    from fastode_gb300.batch import Batch
    torch = cuda
    groups = 2 * sm_count(torch)
    sm = syn.synthetic_mechanism(48, 100, 3)
    b = Batch(sm.mech, syn.synthetic_cells(sm, 32 * groups, 5).Y0, algorithm=Algorithm())
    k = torch.full((sm.R, 32 * groups), float("nan"), dtype=torch.float64, device="cuda")
    at = torch.full((sm.n,), 1e-17, dtype=torch.float64, device="cuda")
    clear_rounds(b)
    b.step(k, 30.0, at, 1e-3)
    torch.cuda.synchronize()
    assert set(b.statuses()) == {"nan or inf"}
    held = meetings(torch, b)
    assert np.any(held) and np.all(held % 2 == 0)


def equal(a, b):
    for x, y in zip(a, b):
        np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("per_sm", [0, 1.6, 9])
def test_rounds_of_several_mechanisms(cuda, per_sm):
    """120/260 with mechanisms whose attempts are a fifth and a fiftieth of its
    work, every ninth group failing at its first attempt, on blocks that pull
    groups of all three, captured and replayed: the bits of the launch without
    rounds. Six blocks per SM, one for each group (0: teams of 2), and 1.6 and
    9 blocks per SM (teams of 8, one warp) that take the groups in turn."""
    from fastode_gb300 import Algorithm, synthetic as syn
    from fastode_gb300.multi import MultiBatch, Part
    torch = cuda
    slots = int(per_sm * sm_count(torch))
    groups = max(6 * sm_count(torch), 2 * slots)
    wls = syn.batched_uneven(n_cells=32 * groups, intervals=3, sizes=((20, 40), (60, 120), (120, 260)))
    runs = []
    for lockstep in (True, False):
        parts = []
        for wl in wls:
            photo = np.nonzero(wl.sm.photolytic)[0]
            parts.append(Part(wl.sm.mech, wl.cells.Y0, wl.k_at(0), wl.atol, wl.rtol, wl.dt,
                              algorithm=Algorithm(lockstep=lockstep), photolysis=(photo, wl.sm.J[photo], wl.cells.phase)))
            thermal = np.nonzero(~wl.sm.photolytic)[0][0]
            parts[-1].k[int(thermal), ::32 * 9] = float("nan")
        mb = MultiBatch(parts, slots=slots)
        clear_rounds(mb)
        mb.run(3, graph=True)
        torch.cuda.synchronize()
        assert np.any(meetings(torch, mb)) == lockstep
        runs.append([v for p in mb.parts for v in (p.state(), p.counts.cpu().numpy(), p.memory.cpu().numpy(),
                                                   p.status.cpu().numpy())])
        del mb, parts
    assert all(set(s) == {0, 3} for s in runs[0][3::4])
    equal(*runs)


@pytest.mark.parametrize("per_sm", [2, 9])
def test_rounds_of_a_constrained_mechanism(cuda, per_sm):
    """RODAS3 160/340, whose groups project onto their constraints while the
    others of their SM are in a round (and every seventh, with a NaN rate
    constant, does not get past that): the bits of the launch without rounds,
    on teams of 8 and of one warp."""
    from fastode_gb300 import RODAS3, Algorithm, synthetic as syn
    from fastode_gb300.batch import Batch
    torch = cuda
    groups = per_sm * sm_count(torch)
    wl = syn.dae_constrained(n_cells=32 * groups, intervals=2)
    at = torch.from_numpy(wl.atol).cuda()
    ks = [torch.from_numpy(np.ascontiguousarray(wl.k_at(i).T)).cuda() for i in range(2)]
    ks[1][:, ::32 * 7] = float("nan")
    runs = []
    for lockstep in (True, False):
        b = Batch(wl.sm.mech, wl.cells.Y0, mass=wl.mass, algorithm=Algorithm(RODAS3, lockstep=lockstep))
        clear_rounds(b)
        for k in ks:
            b.step(k, wl.dt, at, wl.rtol)
        torch.cuda.synchronize()
        assert np.any(meetings(torch, b)) == lockstep
        runs.append([b.state(), b.counts.cpu().numpy(), b.memory.cpu().numpy(), b.status.cpu().numpy()])
        del b
    assert set(runs[0][3]) == {0, 4}
    equal(*runs)
