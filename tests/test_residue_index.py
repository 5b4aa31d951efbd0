"""Residue addresses past 4 GB on CPU (no GPU): builds tests/native/residue_index_check.cpp against
fherma-polynomial-cuda_b200/csrc/residue_index.h and host_plan.cpp and runs it at the widest accepted points."""
import os
import subprocess

from conftest import PACKAGE_DIR, REPO


def test_residue_index_past_four_gigabytes(tmp_path):
    binary = tmp_path / "residue_index_check"
    sources = [os.path.join(REPO, "tests", "native", "residue_index_check.cpp"),
               os.path.join(PACKAGE_DIR, "csrc", "host_plan.cpp")]
    subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", *sources, "-o", str(binary)], check=True)
    done = subprocess.run([str(binary)], capture_output=True, text=True, timeout=600)
    assert done.returncode == 0, done.stderr[-2000:] + done.stdout
    assert "0 failures" in done.stdout
