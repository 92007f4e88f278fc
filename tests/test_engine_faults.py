"""The engine's host side when a CUDA call fails, and the order of its work on
its streams, against a runtime on the host (tests/engine_faults.cpp)."""
import os
import shutil
import subprocess

import pytest

from conftest import PKG_DIR, ROOT

CUDA_HOME = os.environ.get("CUDA_HOME") or os.path.dirname(os.path.dirname(shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"))


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    obj = os.path.join(PKG_DIR, "lib", "engine.o")
    subprocess.run(["make", "-s", "-C", PKG_DIR, "lib/engine.o"], check=True)
    exe = str(tmp_path_factory.mktemp("faults") / "engine_faults")
    tests = os.path.join(ROOT, "tests")
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", os.path.join(ROOT, "include"), "-I", os.path.join(CUDA_HOME, "include"),
                    "-o", exe, os.path.join(tests, "engine_faults.cpp"), os.path.join(tests, "fake_cuda.cpp"), obj,
                    "-ldl", "-lpthread"], check=True)
    return exe


@pytest.mark.parametrize("what", ["tables", "errors", "order", "masks"])
def test_engine_faults(program, what):
    run = subprocess.run([program, what], capture_output=True, text=True, timeout=600)
    assert run.returncode == 0, run.stdout
