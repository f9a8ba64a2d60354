"""The generated phases' schedule on teams of warps, emulated on the host
(tests/cpp/team_emulator.cpp): no two warps of a team touch the same item
between two barriers when one of them writes it, no access leaves the scratch,
and evaluations, factors and solutions are those of plain loops bit for bit
for teams of 1 to 128 warps."""
import shutil
import subprocess
import sys
from pathlib import Path

import pytest

from golden_cases import load, mechanism_of, table_mechanism

ROOT = Path(__file__).resolve().parents[1]
sys.path.insert(0, str(ROOT / "tests"))


@pytest.fixture(scope="module")
def team_emulator(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    cuda = next((p for p in ("/usr/local/cuda/include",) if Path(p).exists()), None)
    if cuda is None:
        pytest.skip("no CUDA headers")
    out = tmp_path_factory.mktemp("emu") / "team_emulator"
    csrc = ROOT / "fast-ode-atmospheric-chem_gb300" / "csrc"
    subprocess.run([cxx, "-std=c++17", "-O2", "-ffp-contract=off", f"-I{csrc}", f"-I{ROOT / 'include'}", f"-I{cuda}",
                    str(ROOT / "tests" / "cpp" / "team_emulator.cpp"),
                    *(str(csrc / s) for s in ("symbolic.cpp", "layout.cpp", "codegen.cpp")), "-o", str(out)],
                   check=True)
    return out


# (mechanism, algebraic species, register tile): no square, one block, several;
# rows and tiles that do not divide; one species
@pytest.mark.parametrize("which,algebraic,tile", [
    ("ros3_20x40", 0, 6), ("ros3_20x40", 3, 4), ("ros3_210x500", 0, 6), ("ts1", 0, 6), ("dae", 10, 6), ("60x40", 0, 6),
    ("120x260", 0, 8), ("120x260", 7, 5), ("1x1", 0, 6), ("2x2", 1, 6), ("3x4", 0, 1), ("7x20", 0, 6), ("33x90", 2, 16)])
def test_generated_phases_on_teams(team_emulator, tmp_path, which, algebraic, tile):
    from fastode_gb300 import synthetic as syn
    from test_host import _write_descriptor
    if which.startswith("ros3"):
        mech = mechanism_of(load(which))
    elif which == "ts1":
        mech = table_mechanism(load("ts1_tier1_30s"))
    elif which == "dae":
        mech = syn.dae_constrained(n_cells=32, intervals=1).sm.mech
    else:
        n, r = (int(v) for v in which.split("x"))
        mech = syn.synthetic_mechanism(n, r, seed=3).mech
    desc = tmp_path / "mech.bin"
    _write_descriptor(desc, mech)
    r = subprocess.run([str(team_emulator), str(desc), str(algebraic), str(tile)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    print(r.stdout)
