"""Device arena on the host (no GPU): tests/native/dev_arena_check.cpp runs csrc/dev_arena.hpp on a stand-in for
the CUDA runtime whose copies from pageable memory return before their data has landed."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]


def test_arena(tmp_path):
    exe = tmp_path / "dev_arena_check"
    subprocess.run(["g++", "-O1", "-std=c++17", "-I/usr/local/cuda/include", "-o", str(exe),
                    str(ROOT / "tests/native/dev_arena_check.cpp")], check=True, capture_output=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout
