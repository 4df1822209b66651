"""The plan of the decode kernels, shares or equal pieces: tests/host_plan/piece_check.cpp is compiled with the library's own
host_logic.cpp and checks random steps and which plan timed steps get."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


def test_pieces_of_random_and_timed_steps(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no C++ compiler")
    exe, csrc = tmp_path / "piece_check", ROOT / "psi-dec_b200" / "csrc"
    done = subprocess.run([gxx, "-std=c++17", "-O2", "-Wall", "-Wextra", "-Werror", f"-I{ROOT / 'include'}", f"-I{csrc}",
                           str(ROOT / "tests" / "host_plan" / "piece_check.cpp"), str(csrc / "host_logic.cpp"), "-o", str(exe)],
                          capture_output=True, text=True)
    assert done.returncode == 0, done.stderr
    done = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert done.returncode == 0 and "pieces ok" in done.stdout, done.stdout + done.stderr
