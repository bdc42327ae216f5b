"""The pipelined LU-SGS sweep's bounded waits (tests/pipeline_wait.cu, compiled
here with the product's source): a strip of the most steps a plan may have, in
which every band waits for all bands before it, finishes within its limit with
the bits of the substitution; limits of a few polls end the kernels with the
time-out status and leave the plan as it was."""

import subprocess
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

HERE = Path(__file__).resolve().parent


@pytest.mark.parametrize("polls", (None, 0, 1, 40, 4000))
def test_waits_cover_the_longest_plan_and_run_out_cleanly(tmp_path, cuda_device, polls):
    from meshcfd_gb300.build import nvcc

    try:
        compiler = nvcc()
    except RuntimeError:
        pytest.skip("needs nvcc")
    exe = tmp_path / "pipeline_wait"
    limit = [] if polls is None else [f"-DMCFD_PIPELINE_SPINS={polls}"]
    subprocess.run([compiler, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "-fmad=false",
                    "-Xcompiler", "-ffp-contract=off", *limit, "-o", str(exe), str(HERE / "pipeline_wait.cu")],
                   check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=240)
    print(out.stdout)
    if out.returncode == 77:
        pytest.skip("the device runs no cluster of the sweep's blocks")
    assert out.returncode == 0, out.stdout + out.stderr
    got = dict(p.split("=") for p in out.stdout.split() if "=" in p)
    assert int(got["cases"]) == 12
    assert int(got["timeouts"]) == 0 if polls is None else polls > 0 or int(got["timeouts"]) == 12, out.stdout
