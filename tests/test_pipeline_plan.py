"""The pipelined band LU-SGS sweep's plan
(meshcfd_gb300/csrc/mcfd_pipeline_plan.h, plain C++ shared with the library):
executed on the host as k_lusgs_pipeline executes it, with the bands
interleaved at random, it reproduces the natural-order substitution bit for
bit, forward and backward, on structured, long-range-coupled and randomly
numbered grids, with roomy and tight rings, without a deadlock, and writes
every slot once.  The device sweep's bits: tests/test_gpu_pipeline_sweep.py."""

import shutil
import subprocess
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_pipeline_plan_executes_to_the_substitution(tmp_path):
    exe = tmp_path / "pipeline_plan_check"
    subprocess.run(["g++", "-O2", "-ffp-contract=off", "-std=c++17", "-o", str(exe),
                    str(HERE / "pipeline_plan_check.cpp")], check=True)
    for seed in (1, 2, 3):
        out = subprocess.run([str(exe), str(seed)], capture_output=True, text=True)
        assert out.returncode == 0, out.stdout + out.stderr
        assert "failures=0" in out.stdout
        assert int(out.stdout.split("planned=")[1].split()[0]) > 700, out.stdout
