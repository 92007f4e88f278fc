"""Every epilogue of the tcgen05 GEMM at ragged shapes (tests/gemm_modes.cu):
the network itself runs them with rows padded to 128 only."""
import os
import shutil
import subprocess

import pytest

from conftest import PKG_DIR, ROOT

pytestmark = pytest.mark.gpu


def test_every_epilogue_at_ragged_shapes(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = str(tmp_path / "gemm_modes")
    subprocess.run([nvcc, "-O2", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "--expt-relaxed-constexpr",
                    "-I", os.path.join(PKG_DIR, "csrc"), "-o", exe, os.path.join(ROOT, "tests", "gemm_modes.cu")], check=True)
    run = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert run.returncode == 0, run.stdout
