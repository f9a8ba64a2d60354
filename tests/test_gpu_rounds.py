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
