"""The process's shared copy team on CPU (no GPU): builds and runs tests/native/host_team_shared_check.cpp
against fherma-polynomial-cuda_b200/csrc/host_io.h (who shares a team, when it ends, and jobs posted
from several threads at once)."""
import os
import subprocess

from conftest import REPO


def test_plans_share_one_copy_team(tmp_path):
    out = tmp_path / "host_team_shared_check"
    source = os.path.join(REPO, "tests", "native", "host_team_shared_check.cpp")
    subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", source, "-o", str(out)], check=True)
    done = subprocess.run([str(out)], capture_output=True, text=True, timeout=120)
    assert done.returncode == 0 and "ok" in done.stdout, done.stderr + done.stdout
