"""The lowest eigenpair of the Lanczos matrix (mcpi_b200/csrc/tridiag.cpp,
tests/cpp/tridiag_check.cpp): against the whole eigenproblem, in the host
memory that its rotations take, and a status where there is none. No GPU needed."""
import os
import subprocess

from conftest import ROOT


def test_lowest_eigenpair_and_its_memory(tmp_path):
    exe = tmp_path / "tridiag_check"
    subprocess.run(["g++", "-O2", "-std=c++17", os.path.join(ROOT, "tests", "cpp", "tridiag_check.cpp"),
                    "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
