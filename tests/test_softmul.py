"""The FP64 product on the integer pipes, checked on the host.

tests/cpp/softmul_check.cu includes cdet_softmul.cuh (the product the FP64
Green assembly takes) and compares it with the host's IEEE product: random
factors, ties, carries, the ends of the exponent ranges and the values that
must be reported.
"""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "cdet-renyi-entanglement-hpc_gb300", "csrc")


def test_soft_product_is_the_ieee_product(tmp_path):
    nvcc = shutil.which("nvcc") or ("/usr/local/cuda/bin/nvcc" if os.path.exists("/usr/local/cuda/bin/nvcc")
                                    else None)
    if nvcc is None:
        pytest.skip("nvcc not found")
    exe = tmp_path / "softmul_check"
    subprocess.run([nvcc, "-std=c++17", "-O1", f"-I{CSRC}", os.path.join(HERE, "cpp", "softmul_check.cu"), "-o",
                    str(exe)], check=True, capture_output=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
    assert " 0 wrong, 0 out of range" in out.stdout
