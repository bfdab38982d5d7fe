"""The host side of the C ABI without a GPU: each library source on a CUDA
runtime in host memory (fake_cuda.h), where a check sees the device state a
call leaves and gives the answer of any launch."""
import os
import subprocess

import pytest

from sampo_gb300 import build

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.parametrize("name", ["batch"])
def test_host_side(tmp_path, name):
    try:
        nvcc = build.nvcc()
    except RuntimeError:
        pytest.skip("nvcc not available")
    exe = str(tmp_path / "check")
    subprocess.run([nvcc, *build.ARCH, "-O1", "-std=c++17", "--fmad=false", "-Xcompiler", "-ffp-contract=off",
                    os.path.join(HERE, f"host_{name}_check.cu"), "-o", exe], check=True, capture_output=True, text=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stdout + out.stderr
