"""The host side of the C ABI without a GPU: each library source on a CUDA
runtime in host memory (fake_cuda.h), where a check sees the device state a
call leaves and gives the answer of any launch."""
import os
import subprocess

import pytest

from sampo_gb300 import build

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.parametrize("name", ["api", "batch", "noalloc"])
def test_host_side(tmp_path, name):
    try:
        nvcc = build.nvcc()
    except RuntimeError:
        pytest.skip("nvcc not available")
    exe = str(tmp_path / "check")
    subprocess.run([nvcc, *build.ARCH, "-O1", "-std=c++17", "--fmad=false", "-Xcompiler", "-ffp-contract=off",
                    os.path.join(HERE, f"host_{name}_check.cu"), "-o", exe], check=True, capture_output=True, text=True)
    out = subprocess.run([exe], cwd=tmp_path, capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stdout + out.stderr


@pytest.mark.gpu
def test_days_behind_a_launch_that_gave_up(gpu_ready, tmp_path):
    exe = str(tmp_path / "check")
    objs = [os.path.join(build.OUT, o + ".o") for o in
            ("sampo_kernels.cu", "sampo_host.cpp", "sampo_species.cu", "sampo_jit_sources.cpp")]
    subprocess.run([build.nvcc(), *build.NVFLAGS, os.path.join(HERE, "device_rows_check.cu"), *objs, "-o", exe, "-ldl", "-lpthread"],
                   check=True, capture_output=True, text=True)
    out = subprocess.run([exe, str(tmp_path / "a.ck")], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stdout + out.stderr
