"""The 113-bit integer arithmetic of the double-double integrand behind the
split assembly (cdet_widefloat.cuh), checked on the host against binary128:
products, base - l r, inverses, the stored format and its ordering."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "cdet-renyi-entanglement-hpc_gb300", "csrc")


def test_wide_arithmetic(tmp_path):
    nvcc = shutil.which("nvcc") or ("/usr/local/cuda/bin/nvcc" if os.path.exists("/usr/local/cuda/bin/nvcc")
                                    else None)
    if nvcc is None:
        pytest.skip("nvcc not found")
    exe = tmp_path / "widefloat_check"
    subprocess.run([nvcc, "-std=c++17", "-O1", "--extended-lambda", f"-I{CSRC}",
                    os.path.join(HERE, "cpp", "widefloat_check.cu"), "-o", str(exe)], check=True, capture_output=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
    assert " 0 violations" in out.stdout
