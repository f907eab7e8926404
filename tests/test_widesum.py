"""The fixed-point sums of the 113-bit connected recursion (WideSum,
cdet_widefloat.cuh), checked on the host against binary128 on graded subset
values: a mask's bits do not depend on how large other masks are."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "cdet-renyi-entanglement-hpc_gb300", "csrc")


def test_wide_sums(tmp_path):
    nvcc = shutil.which("nvcc") or ("/usr/local/cuda/bin/nvcc" if os.path.exists("/usr/local/cuda/bin/nvcc")
                                    else None)
    if nvcc is None:
        pytest.skip("nvcc not found")
    exe = tmp_path / "widesum_check"
    subprocess.run([nvcc, "-std=c++17", "-O1", f"-I{CSRC}", os.path.join(HERE, "cpp", "widesum_check.cu"),
                    "-o", str(exe)], check=True, capture_output=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
    assert " 0 violations" in out.stdout
