"""The adjoint under a memory cap that its small workspace fits."""
import numpy as np
import pytest

from golden_cases import load, mechanism_of

pytestmark = pytest.mark.gpu


def test_adjoint_under_a_memory_cap(cuda):
    """With torch's share of the device capped below the workspace that keeps
    the replayed steps, the adjoint runs in the small one: the same bits."""
    from fastode_gb300 import adjoint as A
    torch = cuda
    f = load("ros3_20x40")
    mech = mechanism_of(f)
    copies = 32
    Y0 = np.tile(f["Y0"], (copies, 1))
    k = torch.from_numpy(np.ascontiguousarray(np.tile(f["k"][0], (copies, 1)).T)).cuda()
    traj = A.forward_record(mech, Y0, lambda i: k, float(f["dt"]), f["atol"], float(f["rtol"]), 1)
    lam = torch.ones_like(traj.batch.Y)
    want = A.adjoint(traj, lam)
    small, large = A._workspace(traj).numel(), A._workspace(traj, keep=True).numel()
    spare = 64 << 20      # the other tensors of the call, in blocks of up to 20 MB
    assert large > small + spare
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    cap = torch.cuda.memory_reserved() + small + spare
    try:
        torch.cuda.set_per_process_memory_fraction(cap / total)
        got = A.adjoint(traj, lam)
        torch.cuda.synchronize()
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    for x, y in zip(want, got):
        assert torch.equal(x, y)
