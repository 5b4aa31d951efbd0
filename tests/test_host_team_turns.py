"""Long copies on the shared copy team on CPU (no GPU): builds tests/native/host_team_turns_check.cpp
against fherma-polynomial-cuda_b200/csrc/host_io.h and runs it (a short job beside a long copy of another
thread, and the pieces of several callers' pack jobs)."""
import os
import subprocess

from conftest import REPO


def test_short_job_beside_a_long_copy(tmp_path):
    binary = tmp_path / "host_team_turns_check"
    source = os.path.join(REPO, "tests", "native", "host_team_turns_check.cpp")
    subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", source, "-o", str(binary)], check=True)
    done = subprocess.run([str(binary)], capture_output=True, text=True, timeout=120)
    assert done.returncode == 0, done.stderr[-2000:] + done.stdout
    assert "0 failures" in done.stdout
