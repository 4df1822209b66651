"""Which cut units are merged in the launch: tests/host_plan/merge_check.cpp is compiled with the library's own host_logic.cpp."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


def test_merges_of_random_steps(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no C++ compiler")
    exe, csrc = tmp_path / "merge_check", ROOT / "psi-dec_b200" / "csrc"
    done = subprocess.run([gxx, "-std=c++17", "-O2", "-Wall", "-Wextra", "-Werror", f"-I{ROOT / 'include'}", f"-I{csrc}",
                           str(ROOT / "tests" / "host_plan" / "merge_check.cpp"), str(csrc / "host_logic.cpp"), "-o", str(exe)],
                          capture_output=True, text=True)
    assert done.returncode == 0, done.stderr
    done = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert done.returncode == 0 and "merges ok" in done.stdout, done.stdout + done.stderr
