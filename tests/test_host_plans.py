"""The planners behind psi_gqa_prepare, called directly: tests/host_plan/plan_check.cpp is compiled with the library's own
host_logic.cpp and checks random steps (every unit covered once, partial slots, counters, balance, the replay capacity, the
merge of rows at one position) and which kernel timed steps are dealt to."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


def test_plans_of_random_steps(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no C++ compiler")
    exe, csrc = tmp_path / "plan_check", ROOT / "psi-dec_b200" / "csrc"
    done = subprocess.run([gxx, "-std=c++17", "-O2", "-Wall", "-Wextra", "-Werror", f"-I{ROOT / 'include'}", f"-I{csrc}",
                           str(ROOT / "tests" / "host_plan" / "plan_check.cpp"), str(csrc / "host_logic.cpp"), "-o", str(exe)],
                          capture_output=True, text=True)
    assert done.returncode == 0, done.stderr
    done = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert done.returncode == 0 and "plans ok" in done.stdout, done.stdout + done.stderr
