"""How many of a drop-in call's buffers stay with a plan (solvers._Staging), on
the host: sets are made without their device buffers."""
import threading
from types import SimpleNamespace

from fastode_gb300.solvers import _Staging


def staging(plan, cells, bytes_):
    """A set as a call holds it: an idle one of its shape, else a new one."""
    with plan.staging_lock:
        for i, st in enumerate(plan.staging):
            if st.key == (cells, 1):
                return plan.staging.pop(i)
    st = _Staging.__new__(_Staging)
    st.key = (cells, 1)
    st.ws = SimpleNamespace(numel=lambda: bytes_)
    return st


def idle(calls):
    """The workspace bytes that stay after the calls (cells, bytes), in turn."""
    plan = SimpleNamespace(staging=[], staging_lock=threading.Lock())
    for cells, bytes_ in calls:
        staging(plan, cells, bytes_).give(plan)
    return [st.ws.numel() for st in plan.staging]


def test_one_large_workspace_stays_with_a_plan():
    """Groups of many cells of a large mechanism: their workspaces are tens of
    megabytes, of which one stays, as many as before the buffers were kept."""
    big = 33 << 20
    assert idle([(c, big) for c in (256, 255, 254, 253, 252)]) == [big]
    assert idle([(256, big), (32, 4 << 20), (255, big)]) == [4 << 20, big]


def test_small_sets_stay():
    assert idle([(c, 1 << 20) for c in range(1, 9)]) == [1 << 20] * _Staging.KEEP
    assert idle([(32, 4 << 20)] * 5) == [4 << 20]
