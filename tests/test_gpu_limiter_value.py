"""The reverse mode's limiter function (tests/limiter_check.cu, compiled here):
the forward limiter's correctly rounded quotient bit for bit; its slope within
12 relative roundings (three products, two sums and the reciprocal twice)."""

import subprocess
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

HERE = Path(__file__).resolve().parent


def test_reverse_limiter_is_the_forward_quotient(tmp_path, cuda_device):
    from meshcfd_gb300.build import nvcc

    try:
        compiler = nvcc()
    except RuntimeError:
        pytest.skip("needs nvcc")
    exe = tmp_path / "limiter_check"
    subprocess.run([compiler, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "-fmad=false",
                    "-o", str(exe), str(HERE / "limiter_check.cu")], check=True)
    out = subprocess.run([str(exe), "300000"], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stdout + out.stderr
    got = dict(p.split("=") for p in out.stdout.split() if "=" in p)
    assert float(got["slope"]) <= 12.0, out.stdout
