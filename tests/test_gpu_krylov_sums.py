"""GMRES's sums at the edges of their grids: one block of the vector, one
entry row more, the last size with one entry a thread of the Gram-Schmidt
grid and the first with more (304 blocks of 256 threads on 152 SMs), against
SciPy's GMRES over the device's own operator and preconditioner.

With the exact Jacobian both are linear to rounding, so the two runs differ by
rounding times the condition of the Hessenberg matrix; 1e-9 of the solution
leaves six decades over the unit roundoff for it."""

import ctypes as C

import numpy as np
import pytest

from test_gpu_implicit import _prepare_on

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx, ny", ((8, 8), (13, 5), (152, 128), (153, 129)))
def test_gmres_follows_scipy_over_the_device_operator(cuda_device, nx, ny):
    import torch
    from scipy.sparse.linalg import LinearOperator, gmres
    from meshcfd_gb300.geometry import build_geometry
    from meshcfd_gb300.meshes import bump_case

    case, P = bump_case(nx, ny)
    P = P * (1.0 + 0.02 * np.random.default_rng(5).standard_normal(P.shape))
    dg, U0, dt, _ = _prepare_on(build_geometry(case.mesh, case), case.numerics, P, cuda_device)
    assert dg.lib.mcfd_implicit_set_jacobian(dg.handle, 1) == 0
    stream = torch.cuda.current_stream().cuda_stream

    def apply(call):
        def mv(x):
            v = torch.as_tensor(np.ascontiguousarray(x).reshape(U0.shape), device=cuda_device)
            out = torch.empty_like(v)
            assert call(dg.handle, v.data_ptr(), out.data_ptr(), stream) == 0
            return out.cpu().numpy().ravel()
        return LinearOperator((U0.size, U0.size), matvec=mv, dtype=float)

    b = np.random.default_rng(nx).standard_normal(U0.shape)
    bd = torch.as_tensor(b, device=cuda_device)
    x = torch.empty_like(bd)
    iters = C.c_int32(0)
    rc = dg.lib.mcfd_gmres(dg.handle, bd.data_ptr(), x.data_ptr(), 1e-6, 120, 30, C.byref(iters), stream)
    A, M = apply(dg.lib.mcfd_implicit_matvec), apply(dg.lib.mcfd_lusgs_apply)
    ref, used, info = np.zeros(U0.size), 0, 1
    while used < 120 and info:  # cycle by cycle, converged or not
        steps = []
        ref, info = gmres(A, b.ravel(), x0=ref, M=M, restart=30, maxiter=1, rtol=1e-6, atol=0.0,
                          callback=steps.append, callback_type="pr_norm")
        used += len(steps)
    assert rc == (6 if info else 0) and iters.value == used
    assert np.abs(x.cpu().numpy().ravel() - ref).max() <= 1e-9 * np.abs(ref).max()
