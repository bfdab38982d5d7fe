"""The kill threshold and the whole-hour days of sampo_model.cuh, compiled from
the header: on the host, and on the device for every whole age of a narrow
pool and a third of all mortalities."""
import os
import subprocess

import pytest

from sampo_gb300 import build

HERE = os.path.dirname(os.path.abspath(__file__))


def _check(tmp_path, where):
    try:
        nvcc = build.nvcc()
    except RuntimeError:
        pytest.skip("nvcc not available")
    exe = str(tmp_path / "check")
    subprocess.run([nvcc, *build.NVFLAGS, os.path.join(HERE, "model_check.cu"), "-o", exe], check=True, capture_output=True, text=True)
    out = subprocess.run([exe, where], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and out.stdout == "thresholds 0 days 0\n", out.stdout + out.stderr


def test_kill_threshold_on_the_host(tmp_path):
    _check(tmp_path, "host")


@pytest.mark.gpu
def test_kill_threshold_and_days_on_the_device(gpu_ready, tmp_path):
    _check(tmp_path, "device")
