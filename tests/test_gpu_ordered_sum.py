"""The residual sum of squares' final sum (block sums added in block order by
integer prefix sums, mcfd_reduce.cuh) against the sequential loop it stands
for, bit for bit: the kernel's own partial sums are restated with NumPy and
added one after the other.  Inputs cross binades, tie, vanish against the
sum, and hold zeros, subnormal squares, infinities and NaN."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BLOCKS, THREADS = 608, 256


def sequential(R):
    """Grid-stride thread sums (one term a thread here), shuffle trees per
    warp, warps in order, then blocks in order."""
    out = []
    with np.errstate(over="ignore", invalid="ignore"):
        for k in range(4):
            x = np.zeros(BLOCKS * THREADS)
            x[: len(R)] = 0.0 + R[:, k] * R[:, k]
            v = x.reshape(BLOCKS, THREADS // 32, 32)
            for off in (16, 8, 4, 2, 1):
                v = v[:, :, :off] + v[:, :, off:2 * off]
            v = v[:, :, 0]
            s = v[:, 0].copy()
            for w in range(1, v.shape[1]):
                s = s + v[:, w]
            out.append(np.add.accumulate(np.concatenate(([0.0], s)))[-1])
    return np.array(out)


def fields(kind, n):
    rng = np.random.default_rng(n)
    if kind == "uniform":
        return rng.uniform(-1.0, 1.0, (n, 4))
    if kind == "wide":  # sixty decades: most terms vanish against the sum, some start it over
        return rng.standard_normal((n, 4)) * 10.0 ** rng.uniform(-30, 30, (n, 4))
    if kind == "ties":  # powers of two: block sums land halfway between neighbours
        return 2.0 ** rng.integers(-27, 1, (n, 4)).astype(float)
    if kind == "growing":
        return np.linspace(0.0, 1.0, n)[:, None] ** 8 * np.ones(4)
    if kind == "tiny":
        return rng.standard_normal((n, 4)) * 1e-160
    R = rng.standard_normal((n, 4))
    R[:, 0] = 0.0
    R[n // 2, 1] = np.inf
    R[n // 3, 2] = np.nan
    R[n // 2, 3] = 1e160
    return R


@pytest.mark.parametrize("n", (1, 255, 257, 8200, 40000, 155648))
@pytest.mark.parametrize("kind", ("uniform", "wide", "ties", "growing", "tiny", "special"))
def test_final_sum_has_the_sequential_bits(cuda_device, kind, n):
    import torch
    from meshcfd_gb300 import _lib

    lib = _lib.native()
    R = np.ascontiguousarray(fields(kind, n))
    Rd = torch.as_tensor(R, device=cuda_device)
    got = torch.empty(4, dtype=torch.float64, device=cuda_device)
    assert lib.mcfd_residual_sumsq_noalloc(Rd.data_ptr(), n, got.data_ptr(),
                                           torch.cuda.current_stream().cuda_stream) == 0
    np.testing.assert_array_equal(got.cpu().numpy(), sequential(R))
