"""The CPU side of bench.py where the reference is not installed."""
import json
import multiprocessing as mp
import sys

import pytest

from oracle import pool


def test_pool_without_the_reference_ends():
    """A worker on the oracle's restatement steps and stops by itself."""
    if pool.reference_installed():
        pytest.skip("the reference is installed")
    with pool.GroupPool(mp.get_context("spawn"), 1, 64) as p:
        assert p.kind == "port"
        assert p.step() == ["converged"]


def test_reference_arm_without_the_reference(monkeypatch, tmp_path, capsys):
    """One line that says that the reference's own code cannot be timed."""
    import bench
    monkeypatch.setattr(pool, "REFERENCE", tmp_path)
    monkeypatch.setattr(sys, "argv", ["bench.py", "--impl", "reference", "--steps", "1", "--cells", "64",
                                      "--cpu-workers", "1"])
    bench.main()
    out = json.loads(capsys.readouterr().out)
    assert out["impl"] == "reference" and out["unavailable"]
