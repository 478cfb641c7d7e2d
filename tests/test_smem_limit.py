"""The dynamic shared-memory limit of a kernel, raised by several host threads at once (csrc/raise_limit.hpp)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_limit_and_record_change_together(tmp_path):
    exe = str(tmp_path / "test_limit")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-pthread", "-o", exe, os.path.join(ROOT, "tests", "cpp", "test_limit.cpp"),
                           "-I", os.path.join(ROOT, "paralleltnnlayers_b200", "csrc")])
    run = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert run.returncode == 0, run.stdout
