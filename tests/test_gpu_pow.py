"""The fixed-point power on the device (tests/pow_device.cu, compiled here for
sm_103a) gives the host build's bits, whose error test_pow.py bounds, on the
operands that the fixed-point path takes."""

import subprocess
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

HERE = Path(__file__).resolve().parent


def test_device_power_is_the_hosts(tmp_path, cuda_device):
    from meshcfd_gb300.build import nvcc

    try:
        compiler = nvcc()
    except RuntimeError:
        pytest.skip("needs nvcc")
    exe = tmp_path / "pow_device"
    subprocess.run([compiler, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "-Xcompiler",
                    "-ffp-contract=off", "-o", str(exe), str(HERE / "pow_device.cu")], check=True)
    for seed in ("1", "2"):
        out = subprocess.run([str(exe), "1000000", seed], capture_output=True, text=True, timeout=120)
        assert out.returncode == 0, out.stdout + out.stderr
