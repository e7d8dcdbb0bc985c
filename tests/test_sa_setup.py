"""Patterns of the smoothed-aggregation set-up on the host against their definitions (CPU)."""
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    exe = tmp_path_factory.mktemp("sa") / "sa_setup_check"
    src = [ROOT / "tests/native/sa_setup_check.cpp", ROOT / "anabasis_b200/csrc/sa_setup.cpp"]
    subprocess.run(["g++", "-O1", "-std=c++17", "-fopenmp", "-I/usr/local/cuda/include", *map(str, src), "-o", str(exe)],
                   check=True, capture_output=True)
    return exe


@pytest.mark.parametrize("grid", [(1, 1, 1), (2, 1, 1), (4, 3, 1), (23, 11, 9), (40, 30, 17)])
@pytest.mark.parametrize("theta", [0.02, 0.1])
def test_patterns(checker, grid, theta):
    r = subprocess.run([str(checker), *map(str, grid), str(theta)], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout
