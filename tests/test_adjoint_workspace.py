"""The adjoint's choice of workspace (adjoint.py), on the host: the sizes come
from a stand-in library, device memory from stand-ins of torch's queries."""
from types import SimpleNamespace

import pytest

PLAIN, KEPT = 1 << 20, 1 << 24


class Lib:
    """fo_adjoint_workspace_bytes and fo_adjoint_kept_bytes of a fixed size."""

    def fo_adjoint_workspace_bytes(self, handle, ngroups, cells, steps, out):
        out._obj.value = PLAIN
        return 0

    def fo_adjoint_kept_bytes(self, handle, ngroups, cells, steps, out):
        out._obj.value = KEPT
        return 0


@pytest.fixture
def ask(monkeypatch):
    """ask(free, limit): the size of the workspace with `free` bytes of device
    memory when torch refuses to allocate more than `limit` at once."""
    import torch
    from fastode_gb300 import _abi, adjoint as A

    def run(free, limit, variant="generated", keep=True):
        def empty(n, **kw):
            if n > limit:
                raise torch.cuda.OutOfMemoryError("out of memory")
            return SimpleNamespace(numel=lambda: n)

        monkeypatch.setattr(_abi, "lib", lambda: Lib())
        monkeypatch.setattr(torch.cuda, "mem_get_info", lambda dev=None: (free, 1 << 40))
        monkeypatch.setattr(torch.cuda, "memory_reserved", lambda dev=None: 0)
        monkeypatch.setattr(torch.cuda, "memory_allocated", lambda dev=None: 0)
        monkeypatch.setattr(torch, "empty", empty)
        batch = SimpleNamespace(plan=SimpleNamespace(handle=None), ngroups=1, max_cells=32,
                                Y=SimpleNamespace(device="cuda:0"),
                                opts=SimpleNamespace(variant=_abi.VARIANTS[variant]))
        ws = A._workspace(SimpleNamespace(batch=batch, max_steps=4), keep=keep)
        return ws.numel()

    return run


def test_kept_steps_where_memory_allows(ask):
    assert ask(8 * KEPT, KEPT) == KEPT
    assert ask(8 * KEPT - 1, KEPT) == PLAIN
    assert ask(8 * KEPT, KEPT, keep=False) == PLAIN


def test_small_workspace_when_the_large_one_is_refused(ask):
    """Free memory says nothing of a cap on the process or of a cache in
    fragments: a refused allocation must not fail a call that the small
    workspace serves."""
    assert ask(8 * KEPT, KEPT - 1) == PLAIN


@pytest.mark.parametrize("variant", ["compact", "pipelined", "plain"])
def test_only_the_generated_adjoint_keeps_steps(ask, variant):
    """The table-driven kernels compute every step again whatever the
    workspace, so they get the small one."""
    assert ask(8 * KEPT, KEPT, variant) == PLAIN
