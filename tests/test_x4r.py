"""The table-driven packed executor of the STOKE chains against the per-opcode
one, for every instruction and for sequences (tests/x4r_check.cpp)."""
import os
import subprocess

from conftest import PKG_DIR, ROOT


def test_table_driven_exec_matches(tmp_path):
    exe = str(tmp_path / "x4r_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(PKG_DIR, "csrc"), "-o", exe,
                    os.path.join(ROOT, "tests", "x4r_check.cpp")], check=True)
    run = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert run.returncode == 0, run.stdout
