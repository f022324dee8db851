"""The slot lookup of the plan builders (tests/cpp/slot_index_check.cpp)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_slot_index(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no host C++ compiler")
    csrc = os.path.join(ROOT, "dnnf90_b200", "csrc")
    exe = str(tmp_path / "slot_index_check")
    subprocess.run([gxx, "-O2", "-std=c++17", "-I", csrc,
                    os.path.join(ROOT, "tests", "cpp", "slot_index_check.cpp"),
                    os.path.join(csrc, "tables.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
