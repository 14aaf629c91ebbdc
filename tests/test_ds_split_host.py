"""The bit forms of the double <-> double-single conversions equal the plain
FP64 ones wherever they claim to (host compilation, no GPU)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "3d-bi-anisotropic-phc_gb300", "csrc")


def test_bit_conversions_equal_the_plain_ones(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    exe = str(tmp_path / "split_check")
    subprocess.run([nvcc, "-std=c++17", "-O1", "-x", "cu", "-I", CSRC, os.path.join(HERE, "ds_split_host_check.cu"),
                    "-o", exe], check=True, capture_output=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
