"""The fixed-point power (meshcfd_gb300/csrc/mcfd_pow.cuh, shared with the
device code) on the host against the C library's long double power: within
0.51 units in the last place for |y| <= 8 and 0.56 for |y| <= 64 (the bounds
its error analysis states), and pow's own values for every operand and result
it does not take."""

import shutil
import subprocess
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
@pytest.mark.parametrize("seed", (1, 2))
def test_fixed_point_power_error(tmp_path, seed):
    exe = tmp_path / "pow_check"
    subprocess.run(["g++", "-O2", "-ffp-contract=off", "-std=c++17", "-o", str(exe), str(HERE / "pow_check.cpp")],
                   check=True)
    out = subprocess.run([str(exe), "1000000", str(seed)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout + out.stderr
    got = dict(p.split("=") for p in out.stdout.split() if "=" in p)
    assert float(got["worst8"]) < 0.51 and float(got["worst64"]) < 0.56, out.stdout
