"""No launch indexes the LU-fallback scratch past the regions it has: the launch
shapes of the staged minors, the queue kernel and the double-double kernels,
checked on the host (tests/cpp/launch_check.cu, linked to the library)."""
import os
import shutil
import subprocess

import pytest

from cdet_gb300 import build as cuda_build

HERE = os.path.dirname(os.path.abspath(__file__))


def test_launches_stay_inside_the_scratch(tmp_path):
    nvcc = shutil.which("nvcc") or ("/usr/local/cuda/bin/nvcc" if os.path.exists("/usr/local/cuda/bin/nvcc")
                                    else None)
    if nvcc is None:
        pytest.skip("nvcc not found")
    lib = cuda_build.build()
    exe = tmp_path / "launch_check"
    subprocess.run([nvcc, "-std=c++17", "-O1", f"-I{cuda_build.CSRC}", os.path.join(HERE, "cpp", "launch_check.cu"),
                    lib, "-Xlinker", f"-rpath={os.path.dirname(lib)}", "-o", str(exe)], check=True, capture_output=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
    assert " 0 violations" in out.stdout
