"""The FP64 reciprocal on the integer pipes, checked on the host.

tests/cpp/softrcp_check.cu compares the reciprocal that the principal minors
take (cdet_softmul.cuh) with the host's IEEE quotient.
"""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "cdet-renyi-entanglement-hpc_gb300", "csrc")


def test_soft_reciprocal_is_the_ieee_quotient(tmp_path):
    nvcc = shutil.which("nvcc") or ("/usr/local/cuda/bin/nvcc" if os.path.exists("/usr/local/cuda/bin/nvcc")
                                    else None)
    if nvcc is None:
        pytest.skip("nvcc not found")
    exe = tmp_path / "softrcp_check"
    subprocess.run([nvcc, "-std=c++17", "-O1", f"-I{CSRC}", os.path.join(HERE, "cpp", "softrcp_check.cu"), "-o",
                    str(exe)], check=True, capture_output=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
    assert " 0 wrong, 0 not reported" in out.stdout
