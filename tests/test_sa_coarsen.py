"""Level steps of the smoothed aggregation on stretched grids and spread coefficients (CPU): every step must halve
the rows at least, or be refused at the first sign, on one of the first two levels (the plain aggregation then serves)."""
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    exe = tmp_path_factory.mktemp("sa") / "sa_coarsen_check"
    src = [ROOT / "tests/native/sa_coarsen_check.cpp", ROOT / "anabasis_b200/csrc/sa_setup.cpp"]
    subprocess.run(["g++", "-O2", "-std=c++17", "-fopenmp", "-I/usr/local/cuda/include", *map(str, src), "-o", str(exe)],
                   check=True, capture_output=True)
    return exe


# (cells a side, spacings, spread, level that is refused)
CASES = [(24, (1, 1, 1), 1, None), (48, (1, 1, 1), 1, None), (48, (6, 1, 1), 1, None), (48, (1, 1, 6), 1, None),
         (48, (10, 1, 1), 1, None), (32, (10, 1, 1), 1, None), (48, (5, 5, 1), 1, None), (48, (30, 30, 1), 1, 1),
         (48, (1, 30, 30), 1, 1), (32, (30, 30, 1), 1, 1), (48, (10, 10, 1), 1, None), (32, (10, 10, 1), 1, None),
         (24, (1, 1, 1), 1e5, None), (48, (1, 1, 1), 1e3, None), (48, (1, 1, 1), 1e4, None), (48, (1, 1, 1), 1e5, None),
         (32, (1, 1, 1), 1e6, None), (64, (10, 10, 1), 1, 0)]


@pytest.mark.parametrize("n,h,spread,refused", CASES)
def test_steps(checker, n, h, spread, refused):
    r = subprocess.run([str(checker), str(n), *map(str, h), str(spread)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
    assert r.stdout.startswith("levels" if refused is None else f"refused at {refused}"), r.stdout
